"""The default launch form against the configured level launches: the block
kernel (shallow, deep and record-prefetching launches) and the direction
chains (128, 256 and 512 threads, the block's warps together or in turns), at the group counts where their tasks and rows
differ -- odd, even and multiples of four, more tasks per item than a warp has
lanes -- and at directions above one wave of blocks.  The configured direct
kernels are checked against the oracle elsewhere; phi must be the same bit for
bit in both precisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n, SN order, groups, precision, launches of one sweep: 1 for chains)
CASES = [
    (1, 4, 1, 0, True), (1, 4, 4, 1, True),         # six cells
    (1, 12, 3, 0, True), (4, 10, 2, 1, True),       # 288 and 200 directions: 256 threads
    (14, 8, 1, 1, True), (17, 8, 2, 0, True), (21, 8, 4, 1, True),  # 512, in turns and together
    (3, 4, 1, 1, True), (3, 4, 2, 0, True), (5, 4, 3, 1, True), (6, 8, 5, 0, True),
    (4, 6, 33, 1, None), (4, 6, 64, 0, None),       # 33 or 9, and 32 tasks per item
    (6, 8, 9, 1, True), (7, 6, 10, 1, True), (20, 8, 7, 1, None), (22, 8, 6, 1, False),  # padded FP32 rows
    (6, 4, 7, 1, True), (7, 6, 12, 1, True), (9, 8, 6, 1, True), (12, 8, 8, 1, True),
    (3, 16, 2, 1, True), (9, 16, 2, 0, True),       # 512 directions: one wave of 128-thread blocks
    (13, 16, 2, 0, False),                          # and more than one of 512-thread ones
    (12, 8, 8, 0, False), (13, 6, 5, 1, None), (18, 8, 12, 1, False), (16, 8, 3, 0, False),
    (14, 8, 64, 0, False), (14, 8, 63, 0, False),   # deep launches: several runs per warp; the record prefetch
    (5, 4, 16, 1, True), (12, 4, 16, 1, False), (18, 8, 16, 1, False), (18, 8, 20, 1, False), (12, 4, 64, 1, False),  # blocks in chains, else plain
]


@pytest.mark.parametrize("n,sn,G,prec,chains", CASES)
def test_default_form_equals_level_launches(built, n, sn, G, prec, chains):
    import torch
    import tycho2_b200 as ty
    mesh = ty.TychoMesh.kuhn_cube(n, 0.05, 5, 1.0)
    sw = ty.SweeperCuda(mesh, sn, G, fp32=prec == 1)
    rng = np.random.default_rng(n + G)
    st = rng.lognormal(0.0, 0.5, mesh.n_cells)
    sw.set_cross_sections(st, 0.6 * st)
    sw.set_source(rng.uniform(0.0, 1.0, sw.phi_shape), "isotropic")
    if chains is not None:
        assert (sw.launches(prec) == 3) == chains  # source, sweep, phi
    phi = torch.tensor(rng.uniform(0.0, 1.0, sw.phi_shape), device="cuda")
    out = [torch.full_like(phi, float("nan")) for _ in range(3)]
    sw.apply(phi, out[0], prec)
    st2 = 1.3 * st  # new cross sections: the records are made again
    sw.set_cross_sections(st2, 0.6 * st)
    sw.apply(phi, out[1], prec)
    even = G % 2 == 0
    sw.configure(prec, "levels", "compact", -172 if prec and even else -96, 0, 2)
    sw.apply(phi, out[2], prec)
    assert torch.equal(out[1].view(torch.int64), out[2].view(torch.int64))
    sw.set_cross_sections(st, 0.6 * st)
    sw.apply(phi, out[2], prec)
    assert torch.equal(out[0].view(torch.int64), out[2].view(torch.int64))
    sw.close()


@pytest.mark.parametrize("n,sn,G", [(13, 8, 2), (20, 8, 1), (20, 6, 2)])
def test_chunked_sweep_on_chain_records(built, n, sn, G):
    """Host sweeps of 64 MB and more go in chunks of directions, on the records of
    the sweeper's own form: between applications by chains, and against the level
    order of a configured sweeper, psi bit for bit."""
    import torch
    import tycho2_b200 as ty
    mesh = ty.TychoMesh.kuhn_cube(n, 0.05, 5, 1.0)
    sw = ty.SweeperCuda(mesh, sn, G)
    assert sw.launches(0) == 3  # chains
    rng = np.random.default_rng(n)
    st = rng.lognormal(0.0, 0.5, mesh.n_cells)
    sw.set_cross_sections(st, 0.4 * st)
    src = rng.uniform(0.0, 1.0, sw.psi_shape)
    assert src.nbytes >= 64 << 20
    x = torch.tensor(rng.uniform(0.0, 1.0, sw.phi_shape), device="cuda")
    y = [torch.empty_like(x) for _ in range(2)]
    psi = [np.full(sw.psi_shape, np.nan) for _ in range(3)]
    sw.apply(x, y[0])
    sw.sweep(psi[0], src)
    sw.apply(x, y[1])
    sw.sweep(psi[1], src)
    sw.configure(0, "levels", "compact", -96, 0, 2)
    sw.sweep(psi[2], src)
    assert torch.equal(y[0].view(torch.int64), y[1].view(torch.int64))
    for other in psi[1:]:
        assert np.array_equal(psi[0].view(np.uint64), other.view(np.uint64))
    sw.close()


@pytest.mark.parametrize("n,sn,G,solver", [(5, 4, 2, "NoPivot"), (20, 8, 7, "NoPivot"), (22, 8, 6, "NoPivot"),
                                           (4, 4, 3, "CramerGlu")])
def test_reported_shape_leads_back_to_the_default_form(built, n, sn, G, solver):
    """shape() of a sweeper in its own form, given to configure() later, is that
    form again: the same launches and the same bits."""
    import torch
    import tycho2_b200 as ty
    mesh = ty.TychoMesh.kuhn_cube(n, 0.05, 5, 1.0)
    sw = ty.SweeperCuda(mesh, sn, G, fp32=True, gauss_elim=solver)
    rng = np.random.default_rng(n)
    st = rng.lognormal(0.0, 0.5, mesh.n_cells)
    sw.set_cross_sections(st, 0.4 * st)
    x = torch.tensor(rng.uniform(0.0, 1.0, sw.phi_shape), device="cuda")
    for prec in (0, 1):
        kept, launches = sw.shape(prec), sw.launches(prec)
        y = [torch.empty_like(x) for _ in range(2)]
        sw.apply(x, y[0], prec)
        for shape in [("compact", -172 if prec and G % 2 == 0 else -96, 0, 2)] * (solver == "NoPivot") + [("direct", 128)]:
            sw.configure(prec, "levels", *shape)
            assert sw.shape(prec) != kept  # nor is it the name of another one
        sw.apply(x, y[1], prec)
        sw.configure(prec, **kept)
        assert sw.shape(prec) == kept and sw.launches(prec) == launches
        sw.apply(x, y[1], prec)
        assert torch.equal(y[0].view(torch.int64), y[1].view(torch.int64))
    sw.close()


def test_own_form_refuses_shapes_it_does_not_have(built):
    import tycho2_b200 as ty
    sw = ty.SweeperCuda(ty.TychoMesh.kuhn_cube(2, 0.05, 5, 1.0), 4, 4, fp32=True)
    for prec, args in ((0, ("levels", "compact", 0, 1)), (1, ("levels", "compact", 0, 2)),
                       (0, ("levels", "compact", 0, 0, 4)), (0, ("levels", "direct", 0)),
                       (0, ("dataflow", "compact", 0))):
        with pytest.raises(ty.TychoError) as e:
            sw.configure(prec, *args)
        assert e.value.status == 1, args
    sw.close()
