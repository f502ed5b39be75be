"""Setup that an object needs before its first cycle is ordered on the object's
own stream, which does not wait for the default stream: with work queued there,
a closure is set and the cycles follow at once."""
import os

import pytest
import torch

from conftest import PKG
import pennant_b200 as pb

pytestmark = pytest.mark.gpu

STATE = ("px", "pu", "zr", "ze")


def learned_run(closure, queued):
    d = pb.Deck(text=("cstop 400\ntstop 1.0\nmeshtype rect\nmeshparams 180 180 1.0 1.0\nuinitradial -1.0\nbcx 0.0\nbcy 0.0\n"
                      "ssmin 0.1\nq1 0.1\nq2 1.0\ndtinit 1.0e-4\ndtmax 1.0e-4\nprecision learned\n"))
    h = pb.Hydro(pb.Mesh(deck=d), d.params())
    h.synchronize()
    if queued:
        torch.cuda._sleep(8_000_000)   # about 4 ms: ends during the run
    h.set_closure(closure)
    h.run()
    torch.cuda.synchronize()
    return {k: h.download(k).tobytes() for k in STATE}, h.closure_counts()


def test_closure_set_behind_work_on_the_default_stream():
    closure = pb.Closure(path=os.path.join(PKG, "closure", "qcs_mlp.bin"))
    torch.zeros(1, device="cuda")
    want = learned_run(closure, False)
    for _ in range(60):
        assert learned_run(closure, True) == want
