"""The forms of the mixed and learned pass A (one warp walking 32-zone tiles,
one thread a zone) give the same bits on both sides of the sizes where the
launch goes from one to the other (37888 zones, and 75776 for mixed rect
meshes): a mesh against its own pieces, whose sizes and numbering take another
form."""
import os

import pytest

from conftest import PKG
import pennant_b200 as pb

pytestmark = pytest.mark.gpu

STATE = ("px", "pu", "zr", "ze", "zp", "zetot", "zvol", "zwrate")
CLOSURE = os.path.join(PKG, "closure", "qcs_mlp.bin")


def deck_text(mesh, nx, ny, precision):
    size = f"{nx} {ny}" if mesh == "pie" else f"{nx} {ny} 1.0 {ny / nx!r}"
    return (f"cstop 6\ntstop 1.0\nmeshtype {mesh}\nmeshparams {size}\nuinitradial -1.0\nbcx 0.0\nbcy 0.0\n"
            f"subregion 0.0 0.4 0.0 0.3\nrinitsub 2.0\neinitsub 0.5\neinit 0.01\nssmin 0.1\nq1 0.1\nq2 1.0\n"
            f"dtinit {0.02 / max(nx, ny)!r}\nprecision {precision}\n")


@pytest.mark.parametrize("precision", ["mixed", "learned"])
@pytest.mark.parametrize("mesh,nx,ny,npieces", [
    ("rect", 256, 148, 2),   # 37888: the walk / pieces of 18944: the walk without the rect numbering
    ("rect", 211, 190, 2),   # 40090: mixed, a thread a zone / 20045: the walk
    ("rect", 296, 256, 2),   # 75776: mixed, a thread a zone / 37888: the walk
    ("rect", 281, 270, 2),   # 75870: the walk / 37935: a thread a zone
    ("pie", 200, 190, 2),    # 38000: a thread a zone / 19000: the walk, one with triangles
])
def test_a_mesh_is_its_pieces(mesh, nx, ny, npieces, precision):
    d = pb.Deck(text=deck_text(mesh, nx, ny, precision))
    m = pb.Mesh(deck=d)
    h = pb.Hydro(m, d.params())
    p = pb.Pieces(m, d.params(), npieces)
    if precision == "learned":
        c = pb.Closure(path=CLOSURE)
        h.set_closure(c)
        p.set_closure(c)
    a, b = h.run(), p.run()
    assert a["cycle"] == b["cycle"] == 6 and a["dtnew"] == b["dtnew"]
    for k in STATE:
        assert h.download(k).tobytes() == p.download(k).tobytes(), k
    if precision == "learned":   # every corner of every cycle is counted in one class
        n = h.closure_counts()
        assert n["mlp"] > 0
        assert sum(n[k] for k in ("zero", "dead", "mlp", "fallback", "ood", "acute")) == 6 * m.nums
