"""GPU parity of the NPB MG path (npb-gpu_b200/csrc/mg.cu) through the C ABI.

The kernels form every sum in the reference's order without fused
multiply-adds, so each operator's output grid -- interior and ghost layer --
must equal the oracle's (oracle/mg_oracle.c, pinned to the reference's
verification norms) bit for bit, and so must the whole benchmark's u and r
after the V-cycles.  Only the residual norm's sum runs in another order:
relative 1e-13 against the oracle, and 1e-14 against the sum of the grid's
squares rounded once where the oracle's own serial sum is further off.  Every class S-C must verify against the
reference's norms at the reference's own epsilon, 1e-8 (mg.cu:528-543).
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = [4, 6, 10, 34, 66, 130]


def rand_grid(rng, m):
    return rng.standard_normal(m ** 3)


@pytest.mark.parametrize("m", SIDES)
def test_resid_bitwise(cgb, oracle, m):
    rng = np.random.default_rng(m)
    u, v = rand_grid(rng, m), rand_grid(rng, m)
    assert np.array_equal(cgb.mg_apply(0, m, u, v), oracle.mg_resid(m, u, v))


@pytest.mark.parametrize("m", SIDES)
@pytest.mark.parametrize("smoother", [0, 1])
def test_psinv_bitwise(cgb, oracle, m, smoother):
    rng = np.random.default_rng(100 + m)
    r, u = rand_grid(rng, m), rand_grid(rng, m)
    got = cgb.mg_apply(1, m, r, out=u, smoother=smoother)
    assert np.array_equal(got, oracle.mg_psinv(m, r, u, smoother))


@pytest.mark.parametrize("m", [6, 10, 34, 66, 130])
def test_rprj3_bitwise(cgb, oracle, m):
    rng = np.random.default_rng(200 + m)
    r = rand_grid(rng, m)
    assert np.array_equal(cgb.mg_apply(2, m, r), oracle.mg_rprj3(m, r))


@pytest.mark.parametrize("mj", [4, 6, 18, 34, 66])
def test_interp_bitwise(cgb, oracle, mj):
    rng = np.random.default_rng(300 + mj)
    z = rand_grid(rng, mj)
    mk = 2 * mj - 2
    u = rand_grid(rng, mk)
    assert np.array_equal(cgb.mg_apply(3, mj, z, out=u), oracle.mg_interp(mj, z, u))
    # assigning: the reference's zero3 then interp
    assert np.array_equal(cgb.mg_apply(4, mj, z, out=u), oracle.mg_interp(mj, z, np.zeros(mk ** 3)))


@pytest.mark.parametrize("lt", [2, 5, 7, 8])
def test_zran3_matches_oracle(cgb, oracle, lt):
    m = (1 << lt) + 2
    v, plus, minus = oracle.mg_zran3(m)
    with cgb.Mg(lt, 0) as g:
        gp, gm = g.points()
        assert np.array_equal(gp, plus) and np.array_equal(gm, minus)
        assert np.array_equal(g.grid("v"), v)


@pytest.mark.parametrize("cls", ["S", "W"])
def test_benchmark_grids_bitwise(cgb, oracle, cls):
    c = cgb.MG_CLASSES[cls]
    want = oracle.mg_run(c["lt"], c["nit"], c["smoother"], grids=True)
    with cgb.Mg.for_class(cls) as g:
        got = g.run(c["nit"])
        assert np.array_equal(g.grid("u"), want["u"])
        assert np.array_equal(g.grid("r"), want["r"])
    assert abs(got["rnm2"] - want["rnm2"]) <= 1e-13 * want["rnm2"]
    assert got["rnmu"] == want["rnmu"]


@pytest.mark.parametrize("lt,nit,smoother", [(2, 1, 0), (3, 2, 1), (4, 3, 0), (5, 2, 1),  # k_coarse alone
                                             (6, 1, 0), (6, 2, 1),  # marches whose wraps meet: 64 < 2 x 60 columns
                                             (7, 3, 1), (8, 1, 0)])  # several tiles a side, ragged at the end
def test_fused_cycles_bitwise(cgb, oracle, lt, nit, smoother):
    """The fused marches and the coarse-level cluster form every point's sums
    in the oracle's order: u and r with their ghosts are bit-identical after
    an odd and an even number of cycles (k_up alternates between two u)."""
    want = oracle.mg_run(lt, nit, smoother, grids=True)
    with cgb.Mg(lt, smoother) as g:
        got = g.run(nit)
        assert np.array_equal(g.grid("u"), want["u"])
        assert np.array_equal(g.grid("r"), want["r"])
    assert got["rnmu"] == want["rnmu"]
    # The kernel adds the rounded squares at most 77 deep (lt = 8: 56 rows a
    # block, a tree of 256 threads, five blocks a thread, the tree again), each
    # addition within 2^-53 of a sum of positive terms; the root halves that:
    # 4.3e-15 with the quotient and the root themselves.
    r = want["r"].reshape(3 * ((1 << lt) + 2,))[1:-1, 1:-1, 1:-1]
    exact = math.sqrt(math.fsum((r * r).ravel()) / 8.0**lt)
    assert abs(got["rnm2"] - exact) <= 1e-14 * exact


@pytest.mark.parametrize("cls", ["S", "W", "A", "B", pytest.param("C", marks=pytest.mark.slow)])
def test_class_verifies(cgb, cls):
    c = cgb.MG_CLASSES[cls]
    with cgb.Mg.for_class(cls) as g:
        out = g.run(c["nit"])
    assert abs(out["rnm2"] - c["rnm2"]) / c["rnm2"] <= cgb.MG_VERIFY_EPSILON
    assert out["device_ms"] > 0


def test_runs_repeat_and_recapture(cgb, oracle):
    with cgb.Mg.for_class("S") as g:
        a = g.run(4)
        b = g.run(2)   # another iteration count: a new graph
        c = g.run(4)
    assert a["rnm2"] == c["rnm2"] and a["rnmu"] == c["rnmu"]
    want = oracle.mg_run(5, 2, 0)
    assert abs(b["rnm2"] - want["rnm2"]) <= 1e-13 * want["rnm2"]


def test_grids_held_and_their_places(cgb, oracle):
    """A benchmark object holds three finest grids (u, v, r) and the coarse
    levels' u and r, 0.29 of one together: k_up writes the new u over r.  The
    two change places every cycle, and the graph captured for another number
    of cycles leaves them where that number does."""
    import torch
    torch.zeros(1, device="cuda")
    lt = 8
    with cgb.Mg(5, 0):  # the library's own first allocations
        before = torch.cuda.mem_get_info()[0]
        with cgb.Mg(lt, 0):
            held = (before - torch.cuda.mem_get_info()[0]) / (8.0 * ((1 << lt) + 2) ** 3)
    assert 3.2 < held < 3.6, held
    with cgb.Mg(6, 0) as g:
        for nit in (1, 2, 0, 3):
            got = g.run(nit)
            want = oracle.mg_run(6, nit, 0, grids=True)
            assert np.array_equal(g.grid("u"), want["u"]), nit
            assert np.array_equal(g.grid("r"), want["r"]), nit
            assert got["rnmu"] == want["rnmu"], nit


def test_invalid_arguments(cgb):
    for lt, sm in ((1, 0), (11, 0), (5, 2)):
        with pytest.raises(cgb.CgbError) as e:
            cgb.Mg(lt, sm)
        assert e.value.status == cgb.ERR_INVALID
    with pytest.raises(cgb.CgbError):
        cgb.mg_apply(0, 7, np.zeros(343), np.zeros(343))  # odd side
