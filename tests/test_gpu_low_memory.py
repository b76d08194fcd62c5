"""Out of device memory for the direction-chain plan (its sort takes 16 bytes an
item): the sweep and the batch fall back to level launches with the same
results, and use chains again once there is room."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def fill_device(left):
    """Blocks that leave about `left` bytes of device memory."""
    import torch
    torch.cuda.empty_cache()
    blocks, size = [], 1 << 36
    while size >= 1 << 22:
        free = torch.cuda.mem_get_info()[0]
        if free - left < size:
            size //= 2
            continue
        try:
            blocks.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            torch.cuda.empty_cache()
            size //= 2
    return blocks


@pytest.mark.parametrize("entry", ["apply", "batch"])
def test_no_room_for_the_chain_plan(built, entry):
    import torch
    import tycho2_b200 as ty
    mesh = ty.TychoMesh.kuhn_cube(20, 0.05, 5, 1.0)  # 6.1 M items: 98 MB for the plan's sort
    rng = np.random.default_rng(3)
    st = rng.lognormal(0.0, 0.5, mesh.n_cells)
    q = rng.uniform(0.5, 1.0, (mesh.n_cells, 4, 1))

    def sweeper():
        s = ty.SweeperCuda(mesh, 8, 1)
        s.set_cross_sections(st, 0.4 * st)
        s.set_source(q, "isotropic")
        return s

    def result(s, levels=False):
        x = torch.tensor(q, device="cuda")
        if entry == "apply":
            y = torch.empty_like(x)
            s.apply(x, y)
            return y.cpu().numpy()
        b = ty.BatchSolver()
        i = b.add(s, "si", err_max=1e-3)
        b.run()
        phi = b.result(i)[0]
        b.close()
        return phi

    sw = sweeper()
    want = result(sw)
    assert sw.launches(0) == 3  # chains
    sw.configure(0, "levels", "compact", -96, 0, 2)
    result(sw)  # level kernels loaded
    sw.close()
    sw = sweeper()
    ty.release_cached_memory(0)
    torch.cuda.synchronize()
    blocks = fill_device(56 << 20)
    try:
        low = result(sw)
    finally:
        del blocks
        torch.cuda.empty_cache()
    assert bits_equal(low, want)
    assert bits_equal(result(sw), want)
    if entry == "apply":
        assert sw.launches(0) > 3  # level launches, kept
    sw.close()


def test_autotune_without_room_for_records(built):
    """Shapes whose records do not fit are left out, the sweeper's own form among
    them."""
    import torch
    import tycho2_b200 as ty
    mesh = ty.TychoMesh.kuhn_cube(20, 0.05, 5, 1.0)  # 688 MB of FP64 compact records
    rng = np.random.default_rng(3)
    st = rng.lognormal(0.0, 0.5, mesh.n_cells)
    q = rng.uniform(0.5, 1.0, (mesh.n_cells, 4, 1))
    x = torch.tensor(q, device="cuda")
    out = []
    for low in (False, True):
        sw = ty.SweeperCuda(mesh, 8, 1, **({"tpi64": 1} if low else {}))
        sw.set_cross_sections(st, 0.4 * st)
        sw.set_source(q, "isotropic")
        ty.release_cached_memory(0)
        blocks = fill_device(450 << 20) if low else []
        try:
            if low:
                best = sw.autotune(0, reps=1)
                assert best["variant"] in ("items", "tiles")
            out.append(torch.empty_like(x))
            sw.apply(x, out[-1])
        finally:
            del blocks
            torch.cuda.empty_cache()
        sw.close()
    assert torch.equal(out[0].view(torch.int64), out[1].view(torch.int64))
