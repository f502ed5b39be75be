"""Points of many corners (the origin of a pie mesh): the warp that gathers
them adds in the serial order, at counts around its 32-corner steps and around
where it takes over from the single thread (9 corners)."""
import numpy as np
import pytest

from oracle import Oracle
import pennant_b200 as pb

pytestmark = pytest.mark.gpu

COUNTS = (7, 8, 9, 10, 31, 32, 33, 64, 65, 97)
STATE = ("px", "pu", "zr", "ze", "zp", "zetot", "zvol", "zwrate")


def deck_text(nx: int) -> str:
    return (f"cstop 8\ntstop 0.6\nmeshtype pie\nmeshparams {nx} 6\nuinitradial -1.0\nbcx 0.0\nbcy 0.0\n"
            "ssmin 0.1\nq1 0.1\nq2 1.0\ndtinit 0.001\n")


def hydro(nx: int, precision: str):
    d = pb.Deck(text=deck_text(nx)).set("precision", precision)
    return pb.Hydro(pb.Mesh(deck=d), d.params())


@pytest.mark.parametrize("nx", COUNTS)
def test_origin_of_a_pie_bitwise(nx):
    o = Oracle(text=deck_text(nx))
    h = hydro(nx, "fp64")
    for c in range(8):
        assert o.cycle() == 0
        h.cycle()
        for k in STATE:
            assert o.field(k).tobytes() == h.download(k).tobytes(), (nx, c, k)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batched_pies_match_single_runs(precision):
    decks = [pb.Deck(text=deck_text(nx)).set("precision", precision) for nx in COUNTS]
    b = pb.Batch([pb.Mesh(deck=d) for d in decks], [d.params() for d in decks])
    assert b.run() == 0
    for i, nx in enumerate(COUNTS):
        h = hydro(nx, precision)
        h.run()
        for k in STATE:
            assert b.download(i, k).tobytes() == h.download(k).tobytes(), (nx, k)


@pytest.mark.parametrize("nx", (33, 97))
def test_mixed_origin_against_the_oracle(nx):
    o = Oracle(text=deck_text(nx))
    h = hydro(nx, "mixed")
    h.run()
    for _ in range(8):
        assert o.cycle() == 0
    # FP32 corner masses and forces: 2^-24 a value, 8 cycles
    for k in ("px", "pu", "zr"):
        a, g = o.field(k), h.download(k)
        assert np.linalg.norm(a - g) <= 1e-6 * np.linalg.norm(a), k
