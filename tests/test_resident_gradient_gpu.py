"""Gradients through the resident forward and adjoint (one launch each, the
state of a tile in shared memory for every step) against the tile kernels:
the cell arithmetic and the order of each shot's sums are the same, so with
one shot a group the gradients are the same numbers."""
import numpy as np
import pytest
import torch

from test_forward_gpu import _plan_of, synthetic_case

pytestmark = pytest.mark.gpu


def _gradient(c, device, order, fmt, rho, wavelet):
    from geobrain_b200.wave import acoustic_forward_kernel
    vp = torch.tensor(c["vp"], device=device, requires_grad=True)
    r = torch.tensor(c["rho"], device=device, requires_grad=rho)
    w = torch.tensor(c["src_v"], device=device, requires_grad=wavelet)
    out = acoustic_forward_kernel(
        nx=c["nx"], nz=c["nz"], dx=c["dx"], dz=c["dx"], nt=c["nt"], dt=c["dt"], nabc=c["nabc"],
        free_surface=c["free_surface"], src_x=c["src_x"], src_z=c["src_z"], src_n=len(c["src_x"]), src_v=w,
        rcv_x=c["rcv_x"], rcv_z=c["rcv_z"], rcv_n=len(c["rcv_x"]), damp=torch.as_tensor(c["damp"], device=device),
        vp=vp, rho=r, device=device, fd_order=order, imaging_dtype=fmt, imaging_cache="all")
    gen = torch.Generator().manual_seed(5)
    (out["p"] * torch.randn(out["p"].shape, generator=gen).to(device)).sum().backward()
    res = [out["p"].detach(), vp.grad] + ([r.grad] if rho else []) + ([w.grad] if wavelet else [])
    return [t.cpu().numpy() for t in res]


# (nz, nx, nabc, nt, shots), tile rows (0 automatic): one tile and a ragged
# remainder, several tiles both ways, tiles that are all boundary, tiles with
# interior rows; an even and an odd number of steps
@pytest.mark.parametrize("shape,tile_rows", [((37, 53, 4, 41, 1), 0), ((60, 250, 10, 40, 2), 0), ((90, 121, 12, 33, 3), 16),
                                             ((90, 130, 9, 30, 1), 4), ((70, 245, 8, 30, 2), 12),
                                             ((150, 330, 10, 26, 1), 36), ((150, 330, 10, 26, 1), 40)])
@pytest.mark.parametrize("order,fmt,free_surface,rho", [(4, "fp32", False, False), (8, "fp24", False, True),
                                                        (4, "bf16", True, True), (8, "fp32", True, False)])
def test_resident_gradient_is_the_tile_kernels(cuda_device, shape, tile_rows, order, fmt, free_surface, rho):
    nz, nx, nabc, nt, shots = shape
    nabc = max(nabc, order // 2)
    c = synthetic_case(nz, nx, nabc, nt, shots, seed=17, free_surface=free_surface)
    c["src_x"], c["src_z"] = np.full(shots, nx // 2), np.arange(shots) + 2
    # two receivers in one cell would add in either order
    _, keep = np.unique(c["rcv_z"] * 100003 + c["rcv_x"], return_index=True)
    c["rcv_x"], c["rcv_z"] = c["rcv_x"][np.sort(keep)], c["rcv_z"][np.sort(keep)]
    if free_surface:
        # a receiver in the mirror row adds to the row two below it: keep one of each pair
        mirror = c["rcv_z"] == -1
        below = np.isin(c["rcv_x"], c["rcv_x"][mirror]) & (c["rcv_z"] == 1)
        c["rcv_x"], c["rcv_z"] = c["rcv_x"][~below], c["rcv_z"][~below]
    plan = _plan_of(c, order // 2)
    wavelet = order == 4
    try:
        plan.set_tiling(16, 1)
        plan.set_resident(False)
        base = _gradient(c, cuda_device, order, fmt, rho, wavelet)
        try:
            plan.set_resident("global", tile_rows)
        except ValueError:
            pytest.skip("the mirror row's sources lie in another tile")
        assert plan.resident()["tile_rows"] > 0
        out = _gradient(c, cuda_device, order, fmt, rho, wavelet)
    finally:
        plan.set_resident("auto")
        plan.set_tiling(16, 0)
    for a, b in zip(out, base):
        assert np.abs(b).max() > 0
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("order,fmt,free_surface,rho", [(4, "fp32", False, False), (8, "fp24", True, True)])
def test_resident_adjoint_reads_what_the_tile_forward_wrote(cuda_device, order, fmt, free_surface, rho):
    """The adjoint's kernel is chosen when the backward runs: after
    set_resident between the two, the resident adjoint reads a store the tile
    forward made, which holds no imaging fields off the pressure mask.  With
    the store's bytes all ones before the forward (NaN in every format) the
    gradient is the one of a tile forward and a tile adjoint."""
    from geobrain_b200.wave import engine
    c = synthetic_case(70, 245, 9, 33, 1, seed=19, free_surface=free_surface)
    _, keep = np.unique(c["rcv_z"] * 100003 + c["rcv_x"], return_index=True)
    keep = np.sort(keep)[c["rcv_z"][np.sort(keep)] != -1]
    c["src_x"], c["src_z"] = np.array([c["nx"] // 2]), np.array([3])
    c["rcv_x"], c["rcv_z"] = c["rcv_x"][keep], c["rcv_z"][keep]
    t = {k: torch.as_tensor(c[k], device=cuda_device) for k in ("vp", "rho", "damp", "src_v")}
    geo = engine.Geometry(c["nz"], c["nx"], c["nabc"], c["nt"], c["dt"], c["dx"], order // 2, free_surface)
    plan = engine.Plan(geo, c["src_x"], c["src_z"], c["rcv_x"], c["rcv_z"])
    img = torch.full((plan.imaging_bytes(c["nt"], rho, fmt),), 255, dtype=torch.uint8, device=cuda_device)
    store = engine.make_store(None, c["nt"], "fp32", img, c["nt"], rho, fmt)
    plan.set_resident(False)
    p, *_ = engine.run_forward(plan, t["vp"], t["rho"], t["damp"], t["src_v"], want_energy=False, store=store)
    res = torch.randn(p.shape, generator=torch.Generator().manual_seed(5)).to(cuda_device)
    args = (plan, t["vp"], t["rho"], t["damp"], t["src_v"], res, None, None, store, rho)
    base = engine.run_backward(*args)
    assert float(base[0].abs().max()) > 0
    plan.set_resident("global", 16)
    plan.set_profiling(True)
    out = engine.run_backward(*args)
    assert plan.profile()["launches"] < c["nt"]          # one launch for all steps
    for a, b in zip(out, base):
        if b is not None:
            np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
