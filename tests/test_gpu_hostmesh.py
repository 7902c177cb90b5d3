"""The drop-in routines' mesh tables, formed on the device from the caller's inpoel, at the edges
of their tiles: the element table's blocks, the prefix sum's 4,096 points per block, the sort's 64
elements around a point (above it the host forms the lists), points without an element and
elements that name a point twice; and calcRHS at the edges of the pieces its arrays are copied in.
The lists are the reference's element order exactly, so the bar is bit-for-bit equality.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_inpoel(npoin, nelem, fan, seed):
    """Random 1-based elements; the last point lies on exactly `fan` of them."""
    rng = np.random.default_rng(seed)
    inp = rng.integers(1, max(npoin, 2), size=(nelem, 3), dtype=np.int32)
    if fan:
        inp[rng.permutation(nelem)[:fan], 1] = npoin
    return inp


@pytest.mark.parametrize("npoin,nelem,fan", [(1, 1, 0), (3, 1, 0), (12289, 5, 1), (4095, 255, 0),
                                             (4096, 8000, 64), (4097, 8001, 65), (8193, 40000, 5000),
                                             (300, 40000, 0)])
def test_lists_around_points(gpu_lib, oracle, npoin, nelem, fan):
    from cfd_gb300 import solver
    inp = random_inpoel(npoin, nelem, fan, npoin + nelem)
    area = np.random.default_rng(1).uniform(0.1, 1.0, nelem)
    assert np.array_equal(solver.MASAS(area, inp, npoin), oracle.masas(area, inp, npoin))


@pytest.mark.parametrize("nelem", [1, 32767, 32769, 98303, 98305, 262147])
def test_calcrhs_pieces(gpu_lib, oracle, nelem):
    from cfd_gb300 import solver
    rng = np.random.default_rng(nelem)
    n = max(3, nelem // 2)
    inp = random_inpoel(n, nelem, 0, nelem + 1)
    U = np.column_stack([rng.uniform(0.5, 2, n), rng.normal(size=(n, 2)), rng.uniform(2, 9, n)])
    dN = rng.normal(size=(2, nelem, 3))
    el = rng.uniform(1e-3, 1e-1, size=(6, nelem))
    T = rng.uniform(200, 400, n)
    gas = np.array([717.5, 0.025, 1.8e-5, 1.4, 300.0, 1.0])
    r0 = rng.normal(size=(n, 4))
    a = solver.calcRHS(r0.copy(), U, None, dN[0], dN[1], *el, inp, T, gas)
    b = oracle.calcrhs(r0, U, np.zeros((n, 4)), dN[0], dN[1], *el, inp, T, gas)
    assert np.array_equal(a, b)


def test_bad_index_leaves_the_result_alone(gpu_lib):
    from cfd_gb300 import abi, solver
    inp = random_inpoel(500, 900, 0, 5)
    inp[700, 2], inp[801, 0] = 501, 0
    M = np.full(500, 7.0)
    with pytest.raises(abi.CfdError) as e:
        abi.check(abi.lib().cfd_masas(abi.dptr(np.ones(900)), abi.iptr(inp), solver._ci(900),
                                      solver._ci(500), abi.dptr(M)), "cfd_masas")
    assert e.value.status == abi.CFD_ERR_MESH and "701" in str(e.value)
    assert np.all(M == 7.0)
