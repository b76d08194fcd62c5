"""The batched passes' forms against the persistent form (whose per-task
arithmetic and upwind reads are its own): direction chains in 512-thread blocks
(few directions) and 256-thread blocks, and level launches (few directions of a
large member, where one direction would outlast the levels), with every row
kind: one group, two, odd and even counts, whole and several vectors per row.
phi must be the same bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# members (n, SN order, groups) of each batch
BATCHES = {
    "chains-512": [(5, 4, 1), (4, 6, 2), (6, 4, 3)],
    "chains-256": [(6, 8, 1), (5, 8, 8), (7, 8, 6), (4, 8, 5), (1, 4, 2)],
    "levels-fp64": [(15, 2, 8), (3, 2, 1), (4, 2, 2), (5, 2, 3)],
    "levels-both": [(21, 2, 16), (3, 2, 1), (4, 2, 2), (5, 2, 5)],
    "levels-direct": [(21, 2, 16), (9, 2, 12), (4, 2, 20)],            # every row plain
    "levels-many-rows": [(21, 2, 16), (5, 2, 8), (4, 2, 4), (3, 2, 7), (6, 2, 6), (2, 2, 64)],
}


@pytest.mark.parametrize("method", ["si", "mixed"])
@pytest.mark.parametrize("batch", sorted(BATCHES))
def test_batch_forms_agree(built, batch, method):
    import tycho2_b200 as ty
    sweepers = []
    for k, (n, sn, G) in enumerate(BATCHES[batch]):
        mesh = ty.TychoMesh.kuhn_cube(n, 0.05, 50 + k, 1.0)
        sw = ty.SweeperCuda(mesh, sn, G, fp32=method == "mixed")
        rng = np.random.default_rng(k)
        st = rng.lognormal(0.0, 0.5, mesh.n_cells)
        sw.set_cross_sections(st, 0.4 * st)
        sw.set_source(rng.uniform(0.5, 1.5, sw.phi_shape), "isotropic")
        sweepers.append(sw)
    phis = []
    for persistent in (False, True, False):
        b = ty.BatchSolver(persistent=persistent)
        ids = [b.add(sw, method, err_max=1e-10) for sw in sweepers]
        b.run()
        phis.append([b.result(i)[0] for i in ids])
        b.close()
        sweepers[0].solve("si", iter_max=2, err_max=-1.0, want_psi=False)  # its own form in between
    for other in phis[1:]:
        for p, q in zip(phis[0], other):
            assert np.array_equal(p.view(np.uint64), q.view(np.uint64))
    for sw in sweepers:
        sw.close()


@pytest.mark.parametrize("change", ["work order", "cross sections and source"])
@pytest.mark.parametrize("method", ["si", "mixed"])
def test_member_changed_between_steps(built, method, change):
    """A member's buffers may be released and made anew between two steps of its
    batch: another work order (its chain plan), or scattering and source given
    again, and a sweep of its own that fills its records before the batch asks
    for them.  The batch reads the new ones; phi is that of a batch left alone."""
    import tycho2_b200 as ty
    import torch
    rng = np.random.default_rng(9)
    meshes = [ty.TychoMesh.kuhn_cube(n, 0.05, 50 + n, 1.0) for n in (6, 5, 4)]
    sweepers, inputs = [], []
    for k, mesh in enumerate(meshes):
        sw = ty.SweeperCuda(mesh, (4, 6, 8)[k], 3, fp32=True)
        st = rng.lognormal(0.0, 0.5, mesh.n_cells)
        inputs.append((st, 0.6 * st, np.tril(np.ones((3, 3))) / 3.0, rng.uniform(0.5, 1.5, sw.phi_shape)))
        sweepers.append(sw)

    def fresh(sw, inp):
        sw.set_cross_sections(*inp[:3])
        sw.set_source(inp[3], "isotropic")

    def run(between):
        for sw, inp in zip(sweepers, inputs):
            fresh(sw, inp)
        b = ty.BatchSolver()
        ids = [b.add(sw, method, err_max=1e-10) for sw in sweepers]
        b.step()
        b.step()
        others = between()
        b.run()
        phi = [b.result(i)[0] for i in ids]
        b.close()
        for o in others:
            o.close()
        return phi

    def touch():
        sw, others = sweepers[0], []
        if change == "work order":
            sw.set_work_order("random")
        else:
            sw.set_cross_sections(inputs[0][0], inputs[0][1])  # no scattering matrix: its buffer goes
            sw.set_source(None, "isotropic")
        for _ in range(3):  # what was released is used by others
            o = ty.SweeperCuda(meshes[0], 4, 3)
            o.set_cross_sections(np.ones(meshes[0].n_cells), np.zeros(meshes[0].n_cells), 7.0 * np.ones((3, 3)))
            o.set_source(np.full(o.phi_shape, 9.0), "isotropic")
            x = torch.zeros(o.phi_shape, dtype=torch.float64, device="cuda")
            o.apply(x, torch.empty_like(x))
            others.append(o)
        fresh(sw, inputs[0])
        x = torch.zeros(sw.phi_shape, dtype=torch.float64, device="cuda")
        for prec in (0, 1):
            sw.apply(x, torch.empty_like(x), prec)  # fills the records of its own form
        return others

    want, got = run(list), run(touch)
    for p, q in zip(want, got):
        assert np.array_equal(p.view(np.uint64), q.view(np.uint64))
    for sw in sweepers:
        sw.close()
