"""Meshes of which a part leaves the range of the straight-line quotients: a
subregion of density 1e40, whose square is too large a divisor, with its edge
through warps' 32-zone tiles and through groups of eight four-lane zones, and
triangles of the pies on both sides of it.  The zones of the subregion are
formed again with the operators, their neighbours are not; state, scalars and
counts of inverted sides are the oracle's, bit for bit."""
import pytest

from oracle import Oracle
import pennant_b200 as pb

STATE = ("px", "pu", "zr", "ze", "zp", "zetot", "zvol", "zwrate")

# below and above 16384 zones (pass A's four lanes a zone) and 40000 (pass C's)
DENSE = {("rect", 33, 20): "0.0 0.37 0.0 0.25", ("rect", 211, 190): "0.0 0.37 0.0 0.41",
         ("pie", 12, 9): "0.0 0.6 0.0 0.05", ("pie", 129, 130): "0.0 0.6 0.0 0.0035"}
MESHES = pytest.mark.parametrize("mesh", DENSE, ids=lambda m: f"{m[0]}-{m[1]}-{m[2]}")


def deck_text(mesh, dtinit=None):
    kind, nx, ny = mesh
    size = f"{nx} {ny}" if kind == "pie" else f"{nx} {ny} 1.0 {ny / nx!r}"
    return (f"cstop 4\ntstop 1.0e60\nmeshtype {kind}\nmeshparams {size}\nuinitradial -1.0\nbcx 0.0\nbcy 0.0\n"
            f"subregion {DENSE[mesh]}\nrinitsub 1.0e40\neinitsub 0.01\neinit 0.01\nssmin 0.1\nq1 0.1\nq2 1.0\n"
            f"dtinit {dtinit or 0.01 / max(nx, ny)!r}\n")


def hydro(text):
    d = pb.Deck(text=text)
    return pb.Hydro(pb.Mesh(deck=d), d.params())


def is_dense(o):
    return o.field("zr") > 2.0 ** 100


@MESHES
def test_the_edge_cuts_tiles(mesh):
    o = Oracle(text=deck_text(mesh))
    dense = is_dense(o)
    for n in (8, 32):
        tiles = dense[:dense.size // n * n].reshape(-1, n)
        assert (tiles.any(1) & ~tiles.all(1)).any()
    tri = o.field("znump") == 3
    assert mesh[0] == "rect" or ((dense & tri).any() and (~dense & tri).any())


@pytest.mark.gpu
@MESHES
def test_cycles(mesh):
    o = Oracle(text=deck_text(mesh))
    h = hydro(deck_text(mesh))
    for c in range(4):
        assert o.cycle() == 0
        s = h.cycle()
        for k in ("time", "dt", "dtrec", "dtnew", "dvovmax"):
            assert s[k] == o.scalar(k), (c, k)
        for k in STATE:
            assert o.field(k).tobytes() == h.download(k).tobytes(), (c, k)


@pytest.mark.gpu
@MESHES
def test_inverted_sides_of_both_parts_are_counted_once(mesh):
    text = deck_text(mesh, dtinit=0.8)
    o = Oracle(text=text)
    dense = is_dense(o)
    assert o.cycle() != 0
    bad = dense[o.field("mapsz")][o.field("svolp") <= 0.0]
    assert bad.any() and not bad.all()
    h = hydro(text)
    with pytest.raises(pb.PntError) as e:
        h.cycle()
    assert e.value.status == pb.PNT_ERR_BADSIDES
    assert h.scalars()["nbad"] == o.num("nbad") == bad.size


@pytest.mark.gpu
def test_pieces():
    mesh = ("rect", 211, 190)   # 20045 zones a piece: quads without the rectangle's numbering
    o = Oracle(text=deck_text(mesh))
    d = pb.Deck(text=deck_text(mesh))
    p = pb.Pieces(pb.Mesh(deck=d), d.params(), 2)
    for _ in range(4):
        assert o.cycle() == 0
        p.cycle()
    for k in STATE:
        assert o.field(k).tobytes() == p.download(k).tobytes(), k


@pytest.mark.gpu
@pytest.mark.parametrize("kinds", [("rect",), ("rect", "pie")])
def test_batches_match_single_runs(kinds):
    texts = [deck_text(m) for m in DENSE if m[0] in kinds]
    decks = [pb.Deck(text=t) for t in texts]
    b = pb.Batch([pb.Mesh(deck=d) for d in decks], [d.params() for d in decks])
    assert b.run() == 0
    for i, t in enumerate(texts):
        h = hydro(t)
        s = h.run()
        assert all(b.scalars(i)[k] == s[k] for k in ("time", "dt", "dtnew")), i
        for k in STATE:
            assert b.download(i, k).tobytes() == h.download(k).tobytes(), (i, k)
