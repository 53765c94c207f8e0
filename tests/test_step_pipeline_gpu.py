"""The step kernels' launch forms at the sizes where each can go wrong: long
shot loops of a CTA (a stage refilled by the last warp to leave it), group
lanes that hold several groups, step graphs whose arguments are replaced, and
gradients of models one or two cells thick."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from conftest import oracle_kwargs
from test_forward_gpu import _plan_of, synthetic_case
from test_graphs_gpu import _unique_receivers

pytestmark = pytest.mark.gpu


def _run(c, device, order, **kw):
    from geobrain_b200.wave import acoustic_forward_kernel
    vp = torch.tensor(c["vp"], device=device, requires_grad=True)
    out = acoustic_forward_kernel(
        nx=c["nx"], nz=c["nz"], dx=c["dx"], dz=c["dx"], nt=c["nt"], dt=c["dt"], nabc=c["nabc"],
        free_surface=c["free_surface"], src_x=c["src_x"], src_z=c["src_z"], src_n=len(c["src_x"]),
        src_v=torch.as_tensor(c["src_v"], device=device), rcv_x=c["rcv_x"], rcv_z=c["rcv_z"],
        rcv_n=len(c["rcv_x"]), damp=torch.as_tensor(c["damp"], device=device), vp=vp,
        rho=torch.as_tensor(c["rho"], device=device), device=device, fd_order=order, imaging_cache="all", **kw)
    lin = torch.randn(out["p"].shape, generator=torch.Generator().manual_seed(3)).to(device)
    (out["p"] * lin).sum().backward()
    return out["p"].detach(), vp.grad


@pytest.mark.parametrize("order,free_surface,absorbing", [(4, False, "damping"), (8, True, "damping"),
                                                          (4, True, "cpml"), (8, False, "cpml")])
def test_shots_per_cta_do_not_change_results(cuda_device, order, free_surface, absorbing):
    """One to all of 7 shots in a CTA, layers that end inside, at and beyond
    a tile's edge: the traces are the same numbers; the gradient's sums over a
    CTA's shots round in another order, at most 6 roundings of 2^-24 of the
    terms' magnitudes a step, with room for cancellation 1e-5."""
    for nz, nx, nabc in ((41, 233, 12), (32, 104, 16)):
        c = _unique_receivers(synthetic_case(nz, nx, nabc, 37, 7, seed=61, free_surface=free_surface))
        plan = _plan_of(c, order // 2)
        try:
            plan.set_resident(False)
            plan.set_tiling(16, 1)
            p0, g0 = _run(c, cuda_device, order, absorbing=absorbing)
            for spc in (2, 3, 4, 7):
                plan.set_tiling(16, spc)
                p, g = _run(c, cuda_device, order, absorbing=absorbing)
                assert torch.equal(p, p0), spc
                assert float((g - g0).norm() / g0.norm()) < 1e-5, spc
        finally:
            plan.set_tiling(16, 0)
            plan.set_resident("auto")


@pytest.mark.parametrize("absorbing,fmt", [("damping", "fp32"), ("damping", "fp24"), ("cpml", "bf16")])
def test_graphs_with_replaced_arguments_and_lanes(cuda_device, absorbing, fmt):
    """Nine groups of one shot on four lanes, replayed from graphs whose
    buffers are others on every call (the earlier calls' are held), against
    one launch per step on one stream: the same numbers."""
    c = _unique_receivers(synthetic_case(45, 190, 10, 53, 9, seed=62))
    plan = _plan_of(c, 4)
    try:
        plan.set_resident(False)
        plan.set_tiling(16, 1)
        plan.set_group_streams(False)
        plan.set_graph_steps(0)
        p0, g0 = _run(c, cuda_device, 8, absorbing=absorbing, imaging_dtype=fmt)
        plan.set_group_streams(True)
        plan.set_graph_steps(16)
        held = []
        for _ in range(3):
            held.append((torch.empty(3_000_000, device=cuda_device), *_run(c, cuda_device, 8, absorbing=absorbing,
                                                                           imaging_dtype=fmt)))
        for _, p, g in held:
            assert torch.equal(p, p0) and torch.equal(g, g0)
    finally:
        plan.set_tiling(16, 0)
        plan.set_resident("auto")


@pytest.mark.parametrize("nz,nx", [(1, 40), (2, 33), (40, 1), (33, 2), (1, 1), (3, 130)])
def test_gradient_of_thin_models(cuda_device, nz, nx):
    """Every cell a rim cell: the padding's share is folded onto it from one
    or two sides (float64 oracle, the gradient tests' 1e-4)."""
    c = synthetic_case(nz, nx, 9, 40, 2, seed=63, edge_rcv=False)
    c["src_x"], c["src_z"] = np.array([0, nx - 1]), np.array([nz - 1, 0])
    c["rcv_x"], c["rcv_z"] = np.arange(nx), np.full(nx, nz - 1)
    p, g = _run(c, cuda_device, 4)
    lin = torch.randn(p.shape, generator=torch.Generator().manual_seed(3)).numpy()
    ref, _, _ = orc.gradient(**oracle_kwargs(c), res_p=lin, res_vx=np.zeros_like(lin), res_vz=np.zeros_like(lin),
                             half=2, dtype=np.float64)
    assert orc.rel_l2(g.cpu().numpy(), ref) < 1e-4
