"""FP64 states that have blown up: infinities, NaN and numbers whose products
overflow give what the operators give in serial code, the Courant dt of zero
among them.  One cycle against the oracle, in which a NaN stands for any NaN
(their signs and payloads are the processors' own)."""
import ctypes as C

import numpy as np
import pytest

from oracle import Oracle, lib
import pennant_b200 as pb

pytestmark = pytest.mark.gpu

STATE = ("px", "pu", "zr", "ze", "zp", "zetot", "zvol", "zwrate")
MESHES = [("rect", 33, 20), ("rect", 211, 190), ("pie", 12, 9), ("pie", 129, 130)]


def deck_text(mesh, lx=1.0, dtinit=None):
    kind, nx, ny = mesh
    size = f"{nx} {ny}" if kind == "pie" else f"{nx} {ny} {lx!r} {lx * ny / nx!r}"
    return (f"cstop 4\ntstop 1.0e60\nmeshtype {kind}\nmeshparams {size}\nuinitradial -1.0\nbcx 0.0\nbcy 0.0\n"
            f"einit 0.01\nssmin 0.1\nq1 0.1\nq2 1.0\ndtinit {dtinit or 0.01 / max(nx, ny)!r}\n")


def poke(o, name, values):
    C.memmove(lib().orc_field(o.h, name.encode()), np.ascontiguousarray(values).ctypes.data, values.nbytes)


def check_one_cycle(text, change):
    """change(o): {field: values} of the state to start from."""
    o = Oracle(text=text)
    d = pb.Deck(text=text)
    h = pb.Hydro(pb.Mesh(deck=d), d.params())
    for k, v in change(o).items():
        poke(o, k, v)
        h.upload(k, v)
    assert o.cycle() == 0
    s = h.cycle()
    for k in ("dtnew", "dvovmax"):
        assert s[k] == o.scalar(k), k
    for k in STATE:
        np.testing.assert_array_equal(h.download(k), o.field(k), err_msg=k)
    return s


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e250])
@pytest.mark.parametrize("mesh", MESHES, ids=lambda m: f"{m[0]}-{m[1]}-{m[2]}")
def test_one_zone_s_energy(mesh, value):
    def change(o):
        ze = o.field("ze")
        ze[o.numz // 3] = value
        ze[0] = value
        return {"ze": ze}
    # a step so short that the finite one does not invert its neighbours at once
    s = check_one_cycle(deck_text(mesh, dtinit=1e-200 if value == 1e250 else None), change)
    if value == np.inf:
        assert s["dtnew"] == 0.0


@pytest.mark.parametrize("mesh", MESHES, ids=lambda m: f"{m[0]}-{m[1]}-{m[2]}")
def test_a_zone_whose_dt_is_no_number(mesh):
    # without linear viscosity an infinite sound speed gives 0 x inf; the
    # smallest dt of the mesh is left to zones next to that one
    def change(o):
        z = np.arange(o.numz)
        return {"ze": np.where(z == 32, np.inf, np.where(z // 32 == 1, 50.0, 0.01))}
    s = check_one_cycle(deck_text(mesh, dtinit=1e-9).replace("q1 0.1", "q1 0.0"), change)
    assert 0.0 < s["dtnew"] < 1e90


def test_energy_whose_square_term_overflows():
    # (gamma - 1)^2 rho^2 e overflows for finite e and pressure
    text = deck_text(("rect", 33, 20), dtinit=1e-200) + "rinit 1.0e3\n"

    def change(o):
        ze = o.field("ze")
        ze[100] = 1e305
        return {"ze": ze}
    s = check_one_cycle(text, change)
    assert s["dtnew"] == 0.0


@pytest.mark.parametrize("n", [8, 136])
def test_edge_velocity_that_overflows_without_divergence(n):
    # u = A (x, -y) on squares of side h: no divergence, exactly, and A h^2 / 4
    # is finite, but the edges' (du . dx) = A h^2 is not
    h = 2.0 ** 33
    text = deck_text(("rect", n, n), lx=n * h, dtinit=1e-307)

    def change(o):
        return {"pu": o.field("px") * np.array([1.0, -1.0]) * 2.0 ** (1024 - 66)}
    s = check_one_cycle(text, change)
    assert s["dtnew"] == 0.0


@pytest.mark.parametrize("n", [8, 136])
def test_divergence_that_is_no_number(n):
    # u = A (-y, x): the edges' (du . dx) are zeros, and the divergence is
    # the difference of two products A h^2 / 4 that overflow
    h = 2.0 ** 33
    text = deck_text(("rect", n, n), lx=n * h, dtinit=1e-307)

    def change(o):
        return {"pu": o.field("px")[:, ::-1] * np.array([-1.0, 1.0]) * 2.0 ** (1024 - 64)}
    check_one_cycle(text, change)
