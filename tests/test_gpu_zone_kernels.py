"""The zone passes at the sizes and operands where their forms change, bit for
bit against the oracle: one zone, rows shorter and longer than a warp's 32
zones, the last mesh of four lanes a zone and the first past it (16384 zones
in pass A, 40000 in pass C), boundary planes inside the mesh, and meshes so
large or small in their unit of length that every zone leaves the range of the
straight-line quotients and is formed again with the operators."""
import pytest

from oracle import Oracle
import pennant_b200 as pb

pytestmark = pytest.mark.gpu

STATE = ("px", "pu", "zr", "ze", "zp", "zetot", "zvol", "zwrate")


def deck_text(nx, ny, scale=1.0, q1=0.1, planes="bcx 0.0\nbcy 0.0", mesh="rect"):
    size = f"{nx} {ny}" if mesh == "pie" else f"{nx} {ny} {scale!r} {scale * ny / nx!r}"
    return (f"cstop 4\ntstop 1.0e60\nmeshtype {mesh}\nmeshparams {size}\nuinitradial -1.0\n{planes}\n"
            f"einit 0.01\nssmin 0.1\nq1 {q1}\nq2 1.0\ndtinit {0.01 * scale / max(nx, ny)!r}\n")


def check(text):
    o = Oracle(text=text)
    d = pb.Deck(text=text)
    h = pb.Hydro(pb.Mesh(deck=d), d.params())
    for c in range(4):
        assert o.cycle() == 0
        s = h.cycle()
        for k in ("time", "dt", "dtrec", "dtnew", "dvovmax"):
            assert s[k] == o.scalar(k), (c, k)
        for k in STATE:
            assert o.field(k).tobytes() == h.download(k).tobytes(), (c, k)


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 40), (31, 1), (5, 7), (33, 3), (128, 128), (127, 130), (200, 200),
                                   (211, 190), (650, 64)])
def test_rect_sizes(nx, ny):
    check(deck_text(nx, ny))


@pytest.mark.parametrize("nx,ny", [(1, 2), (128, 128), (129, 128), (200, 200), (201, 200)])
def test_pie_sizes(nx, ny):
    check(deck_text(nx, ny, mesh="pie"))


@pytest.mark.parametrize("nx,ny", [(9, 7), (211, 190)])
@pytest.mark.parametrize("scale", [1.0e25, 1.0e-24])
def test_operands_out_of_the_straight_line_range(nx, ny, scale):
    check(deck_text(nx, ny, scale=scale))


@pytest.mark.parametrize("nx,ny", [(9, 7), (211, 190)])
def test_no_linear_viscosity_and_planes_inside_the_mesh(nx, ny):
    check(deck_text(nx, ny, q1=0.0, planes=f"bcx 0.0 {1.0 / nx * (nx // 2)!r}\nbcy 0.0 {1.0 / nx * (ny // 3)!r}"))


@pytest.mark.parametrize("nbcx,nbcy", [(0, 0), (2, 2), (4, 0), (3, 2), (9, 7)])
def test_few_and_many_planes(nbcx, nbcy):
    # 40090 zones: pass C's row tiles, whose words hold the masks of four planes
    nx, ny = 211, 190
    planes = "".join(f"{name} {' '.join(repr(1.0 / nx * (n * k // 10)) for k in range(count))}\n"
                     for name, n, count in (("bcx", nx, nbcx), ("bcy", ny, nbcy)) if count)
    check(deck_text(nx, ny, planes=planes.strip()))


def test_batch_of_them_matches_single_runs():
    texts = [deck_text(9, 7), deck_text(9, 7, scale=1.0e25), deck_text(1, 1), deck_text(211, 190, scale=1.0e-24),
             deck_text(12, 9, mesh="pie"), deck_text(130, 127)]
    for group in (texts, [t for t in texts if "pie" not in t]):
        decks = [pb.Deck(text=t) for t in group]
        b = pb.Batch([pb.Mesh(deck=d) for d in decks], [d.params() for d in decks])
        assert b.run() == 0
        for i, d in enumerate(decks):
            h = pb.Hydro(pb.Mesh(deck=d), d.params())
            h.run()
            for k in STATE:
                assert b.download(i, k).tobytes() == h.download(k).tobytes(), (i, k)
