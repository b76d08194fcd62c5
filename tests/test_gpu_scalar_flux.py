"""The scalar-flux pass at the edges of its tiles: rows that do and do not
divide a tile of 256 elements, the longest rows, cells whose directions fill
less and more than a shared-memory stage, fewer cells than one tile and a last
tile of few.  FP64: phi is the quadrature sum of the resident psi in the order
of the directions, bit for bit.  FP32: within 1e-5 of the FP64 operator (its
rounding is of the order of 1e-7; a misplaced element is wrong in the first
digits)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(1, 2, 1), (1, 4, 64), (2, 16, 1), (4, 4, 1), (9, 8, 1), (5, 6, 2), (4, 8, 3), (6, 6, 5), (7, 4, 7),
         (8, 4, 8), (4, 10, 12), (3, 16, 16), (5, 4, 33), (4, 6, 63), (3, 8, 64),
         (6, 4, 36), (4, 6, 40), (5, 4, 41)]


def make(n, sn, G, fp32):
    import tycho2_b200 as ty
    sw = ty.SweeperCuda(ty.TychoMesh.kuhn_cube(n, 0.05, 5, 1.0), sn, G, fp32=fp32)
    rng = np.random.default_rng(7 * n + G)
    st = rng.lognormal(0.0, 0.3, sw.phi_shape[0])
    sw.set_cross_sections(st, 0.4 * st)
    sw.set_source(rng.uniform(0.5, 1.0, sw.phi_shape), "isotropic")
    return sw


@pytest.mark.parametrize("n,sn,G", CASES)
def test_scalar_flux_is_the_quadrature_sum(built, n, sn, G):
    import torch
    sw = make(n, sn, G, True)
    phi, psi, _ = sw.solve("si", iter_max=2, err_max=-1.0)
    want = np.zeros_like(phi)
    for a, w in enumerate(sw.quadrature.wt):
        want = want + psi[:, a] * w
    assert np.array_equal(phi, want)
    x = torch.tensor(phi, device="cuda")
    y = [torch.full_like(x, float("nan")) for _ in range(2)]
    sw.apply(x, y[0], 0)
    sw.apply(x, y[1], 1)
    assert float(((y[1] - y[0]).abs() / y[0].abs()).max()) <= 1e-5
    sw.close()


def test_batched_scalar_flux(built):
    import tycho2_b200 as ty
    members = [(5, 4, 1), (4, 4, 5), (3, 4, 33), (2, 4, 63), (7, 6, 8), (3, 2, 64), (1, 2, 1), (6, 4, 12)]
    sweepers = [make(n, sn, G, True) for n, sn, G in members]
    for method, tol in (("si", 0.0), ("mixed", 1e-8)):
        b = ty.BatchSolver()
        ids = [b.add(sw, method, err_max=1e-10) for sw in sweepers]
        b.run()
        for sw, i in zip(sweepers, ids):
            phi = b.result(i)[0]
            want = sw.solve("si", err_max=1e-10, want_psi=False)[0]
            assert np.abs(phi / want - 1.0).max() <= tol
        b.close()
    for sw in sweepers:
        sw.close()


@pytest.mark.parametrize("members", [[(18, 2, 8), (3, 4, 3)], [(24, 2, 16), (21, 2, 33), (5, 4, 1)],
                                     [(20, 2, 7), (22, 4, 1)]])
def test_batched_streaming_passes_of_larger_members(built, members):
    """Sums of chunks (4096 elements of phi) for which the streaming passes take a
    chunk whole and in quarters, and several tiles of cells one after the other:
    phi of the single solver's source iteration bit for bit, the mixed solve's to its
    tolerance (1e-9 of a sum; 1e-7 allowed of each element)."""
    import tycho2_b200 as ty
    sweepers = [make(n, sn, G, True) for n, sn, G in members]
    for method, tol in (("si", 0.0), ("mixed", 1e-7)):
        b = ty.BatchSolver()
        ids = [b.add(sw, method, err_max=1e-10 if method == "si" else 1e-9) for sw in sweepers]
        b.run()
        for sw, i in zip(sweepers, ids):
            phi = b.result(i)[0]
            want = sw.solve("si", err_max=1e-10, want_psi=False)[0]
            assert np.abs(phi / want - 1.0).max() <= tol
        b.close()
    for sw in sweepers:
        sw.close()
