"""CUDA-graph replay of the gradient's step loops and of the batched engine:
chunks of gb_plan_set_graph_steps steps replayed from one graph (the step
index, and the imaging fields' address, from a device counter) give the
results of one launch per step, bit for bit, with far fewer host launch
calls."""
import numpy as np
import pytest
import torch

from test_batched_gpu import cases, model_dict
from test_forward_gpu import _plan_of, synthetic_case

pytestmark = pytest.mark.gpu


def _unique_receivers(c):
    """Receivers that share a cell add their residuals with shared-memory
    atomics in the adjoint, in an order that varies between runs; keep one
    receiver per cell so that runs can be compared bit for bit."""
    _, keep = np.unique(np.stack([c["rcv_z"], c["rcv_x"]]), axis=1, return_index=True)
    keep = np.sort(keep)
    return dict(c, rcv_x=c["rcv_x"][keep], rcv_z=c["rcv_z"][keep])


def _grad(c, device, **kw):
    from geobrain_b200.wave import acoustic_forward_kernel
    vp = torch.tensor(c["vp"], device=device, requires_grad=True)
    rho = torch.tensor(c["rho"], device=device, requires_grad=kw.pop("want_rho", False))
    out = acoustic_forward_kernel(
        nx=c["nx"], nz=c["nz"], dx=c["dx"], dz=c["dx"], nt=c["nt"], dt=c["dt"], nabc=c["nabc"],
        free_surface=c["free_surface"], src_x=c["src_x"], src_z=c["src_z"], src_n=len(c["src_x"]),
        src_v=torch.as_tensor(c["src_v"], device=device), rcv_x=c["rcv_x"], rcv_z=c["rcv_z"],
        rcv_n=len(c["rcv_x"]), damp=torch.as_tensor(c["damp"], device=device), vp=vp, rho=rho, device=device,
        fd_order=8, **kw)
    lin = np.random.default_rng(5).standard_normal(out["p"].shape).astype(np.float32)
    (out["p"] * torch.as_tensor(lin, device=device)).sum().backward()
    torch.cuda.synchronize()
    return (vp.grad.cpu().numpy(), None if rho.grad is None else rho.grad.cpu().numpy(),
            out["p"].detach().cpu().numpy())


@pytest.mark.parametrize("nt,cache,want_rho", [(100, "all", False), (87, "all", True), (120, "partial", False)])
def test_gradient_graphs_are_bit_identical(cuda_device, nt, cache, want_rho):
    """The forward steps that keep their imaging fields and the adjoint over
    them, replayed in 16-step chunks (an odd cache start, a ragged last chunk,
    the density fields, and a cache over only part of the steps)."""
    c = _unique_receivers(synthetic_case(60, 250, 10, nt, 5, seed=51))
    plan = _plan_of(c, 4)
    ic = "all" if cache == "all" else plan.imaging_bytes(nt // 2 + 7, want_rho, "fp24")
    kw = dict(imaging_cache=ic, imaging_dtype="fp24", checkpoint_every=23, want_rho=want_rho)
    try:
        plan.set_graph_steps(0)
        plan.set_profiling(True)
        base = _grad(c, cuda_device, **kw)
        calls0 = plan.profile()["launch_calls"]
        plan.set_graph_steps(16)
        plan.set_profiling(True)
        outs = [_grad(c, cuda_device, **kw) for _ in range(2)]
        calls1 = plan.profile()["launch_calls"] / 2
    finally:
        plan.set_profiling(False)
        plan.set_graph_steps(16)
    for out in outs:
        for a, b in zip(out, base):
            if b is not None:
                np.testing.assert_array_equal(a, b)
    if cache == "all":
        assert calls1 * 5 < calls0, (calls1, calls0)


def test_batched_graphs_are_bit_identical(cuda_device):
    """Batched forward and adjoint chunks replayed from graphs (models of
    uneven size and step count), against one launch per step."""
    from geobrain_b200.wave import acoustic_forward_batched, acoustic_gradient_batched
    from geobrain_b200.wave.batched import _Prepared
    cs = [_unique_receivers(c) for c in cases()]
    plans = _Prepared([model_dict(c, cuda_device) for c in cs], 8, cuda_device).plans
    obs = [torch.as_tensor(np.random.default_rng(7 + i).standard_normal(
        (len(c["src_x"]), c["nt"], len(c["rcv_x"]))).astype(np.float32), device=cuda_device) for i, c in enumerate(cs)]

    def residual(i, p):
        r = p - obs[i]
        return 0.5 * (r * r).sum(), r

    def run():
        with torch.no_grad():
            fw = acoustic_forward_batched([model_dict(c, cuda_device) for c in cs], fd_order=8, want_energy=False)
        _, g = acoustic_gradient_batched([model_dict(c, cuda_device) for c in cs], residual, fd_order=8)
        return [o["p"].cpu().numpy() for o in fw], [x.cpu().numpy() for x in g]

    try:
        for p in plans:
            p.set_graph_steps(0)
        base = run()
        for p in plans:
            p.set_graph_steps(16)
        out = run()
        out2 = run()
    finally:
        for p in plans:
            p.set_graph_steps(16)
    for o in (out, out2):
        for a, b in zip(o[0] + o[1], base[0] + base[1]):
            np.testing.assert_array_equal(a, b)


def _plan_gradient(plan, t, res, ws, *, checkpoint_every, cached):
    """dL/dvp through the C ABI on the caller's workspace ws; res: the
    adjoint sources of p, vx, vz (None: unused)."""
    import ctypes

    from geobrain_b200 import _lib
    from geobrain_b200.wave import engine
    dev = t["vp"].device
    n_ck = -(-(plan.geo.nt - cached) // checkpoint_every)
    ck = torch.empty(max(n_ck * plan.checkpoint_bytes(plan.geo.nt, "fp32"), 256), dtype=torch.uint8, device=dev)
    img = torch.empty(max(plan.imaging_bytes(cached, False, "fp32"), 256), dtype=torch.uint8, device=dev)
    store = engine.make_store(ck if n_ck > 0 else None, checkpoint_every, "fp32", img, cached, False, "fp32")
    engine.run_forward(plan, t["vp"], t["rho"], t["damp"], t["src_v"], want_energy=False, store=store)
    g = torch.empty((plan.geo.nz, plan.geo.nx), device=dev)
    _lib.check(plan._lib.gb_backward(plan.h, t["vp"].data_ptr(), t["rho"].data_ptr(), t["damp"].data_ptr(),
                                     t["src_v"].data_ptr(), *[_lib.ptr(r) for r in res], ctypes.byref(store),
                                     g.data_ptr(), None, None, ws.data_ptr(), ws.numel(), engine.stream_handle(dev)))
    return g.cpu().numpy()


@pytest.mark.parametrize("change", ["resident", "checkpoint_every"])
def test_adjoint_graphs_follow_the_workspace_layout(cuda_device, change):
    """Gradients of one plan by the tile adjoint in one caller-owned
    workspace, before and after what can move the adjoint's buffers inside it:
    another resident mode or tiling (vx residuals keep the adjoint in the
    tile kernels), or another segment length of a partial cache.  Each equals
    a plan that never ran anything else, bit for bit."""
    from geobrain_b200.wave import engine
    c = _unique_receivers(synthetic_case(60, 200, 10, 55, 2, seed=53))
    t = {k: torch.as_tensor(c[k], device=cuda_device) for k in ("vp", "rho", "damp", "src_v")}
    shape = (2, c["nt"], len(c["rcv_x"]))
    rng = np.random.default_rng(9)
    rp, rv = (torch.as_tensor(rng.standard_normal(shape).astype(np.float32), device=cuda_device) for _ in range(2))
    geo = engine.Geometry(c["nz"], c["nx"], c["nabc"], c["nt"], c["dt"], c["dx"], 2, False)
    new = lambda: engine.Plan(geo, c["src_x"], c["src_z"], c["rcv_x"], c["rcv_z"])
    if change == "resident":
        runs = [(("auto", 0), 55, 55), ((False, 0), 55, 55), (("cluster", 0), 55, 55), (("global", 16), 55, 55),
                (("auto", 0), 55, 55)]
    else:
        runs = [((False, 0), k, 33) for k in (5, 11, 3, 5)]

    def bytes_of(plan, run):
        plan.set_resident(*run[0])
        return plan.gradient_workspace_bytes(False, max(1, min(run[1], c["nt"] - run[2])), "fp32")

    plan = new()
    sizes = [bytes_of(plan, r) for r in runs]
    assert change == "resident" or len(set(sizes)) == 3      # the layouts do differ
    ws = torch.empty(max(sizes), dtype=torch.uint8, device=cuda_device)
    for mode, every, cached in runs:
        fresh = new()
        for p in (plan, fresh):
            p.set_resident(*mode)
        base = _plan_gradient(fresh, t, (rp, rv, None), torch.empty_like(ws), checkpoint_every=every, cached=cached)
        out = _plan_gradient(plan, t, (rp, rv, None), ws, checkpoint_every=every, cached=cached)
        assert np.abs(base).max() > 0
        np.testing.assert_array_equal(out, base, err_msg=f"{mode} {every}")


def test_gradient_after_autotuning_keeps_its_step_graphs(cuda_device):
    """One shot on a small grid tunes to a resident forward, which uses no
    step graphs; the plan's gradients keep theirs (or run resident too): few
    host launch calls, and the untuned plan's numbers."""
    c = _unique_receivers(synthetic_case(70, 200, 10, 96, 1, seed=57))
    plan = _plan_of(c, 4)
    base = _grad(c, cuda_device, imaging_cache="all")
    try:
        _grad(c, cuda_device, imaging_cache="all", autotune=True)
        assert plan.config()["resident_rows"] > 0 and plan.config()["graph_steps"] == 16
        plan.set_profiling(True)
        out = _grad(c, cuda_device, imaging_cache="all")
        assert plan.profile()["launch_calls"] < c["nt"] // 2
    finally:
        plan.set_profiling(False)
        plan.tuned = None
        plan.set_tiling(16, 0)
        plan.set_graph_steps(16)
        plan.set_group_streams(True)
        plan.set_streaming(False)
        plan.set_resident("auto")
    for a, b in zip(out, base):
        if b is not None:
            np.testing.assert_array_equal(a, b)
