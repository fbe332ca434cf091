"""Bounded device waits: a wait that runs out ends the run with
LAPW1GPU_ERR_TIMEOUT and leaves the context usable.

The test hook lapw1gpu_test_wait_timeout makes the MMA issuer of the
split-precision spherical kernels wait on a barrier that nothing arrives at
(bounded to about half a millisecond); every other wait of the kernel keeps
its full bound, so the producer drains its copies in flight and TMEM is
freed before the kernel returns.  A clean run on the same context follows.
"""
import numpy as np
import pytest
import torch

from hack_wein2k_b200 import lapw1gpu, synth
from oracle import oracle as O
from tests.helpers import rel_errors


@pytest.mark.gpu
def test_timeout_status_then_clean_run(ctx):
    p = synth.small_case("lo")
    hs_o, hsd_o = O.setup(p)
    saved = ctx.tuning()
    ctx.set_precision(lapw1gpu.PREC_SPLIT, 5)
    ctx.set_tuning(sph_tc=1)
    try:
        ctx.test_wait_timeout(True)
        with pytest.raises(lapw1gpu.Lapw1GpuError) as e:
            ctx.setup(p)
        assert e.value.code == 5  # LAPW1GPU_ERR_TIMEOUT
        ctx.test_wait_timeout(False)
        for _ in range(2):
            hs, hsd = ctx.setup(p)
            err = rel_errors(hs, hsd, hs_o, hsd_o)
            assert err["H"] <= 2e-9 and err["S"] <= 2e-9, err
    finally:
        ctx.test_wait_timeout(False)
        ctx.set_tuning(sph_tc=saved["sph_tc"])
        ctx.set_precision(lapw1gpu.PREC_FP64)


@pytest.mark.gpu
@pytest.mark.parametrize("slices", [4, 6, 8])
@pytest.mark.parametrize("batch", [False, True])
def test_projection_timeout_and_nonfinite_status(ctx, slices, batch):
    """The adjoint's projections: the issuer's wait that runs out is
    LAPW1GPU_ERR_TIMEOUT, a NaN in the eigenvectors LAPW1GPU_ERR_NONFINITE,
    and the same call is clean again after either."""
    p = synth.small_case("lo")
    dev = torch.device("cuda", ctx.device)
    nb = 8
    rng = np.random.default_rng(3)
    c = torch.from_numpy(rng.standard_normal((nb, p.n)) + 1j * rng.standard_normal((nb, p.n))).to(dev)
    nan = c.clone()
    nan[nb - 1, p.nv - 1] = float("nan")
    eps = torch.linspace(-1.0, 1.0, nb, dtype=torch.float64, device=dev)
    occ = torch.ones(nb, dtype=torch.float64, device=dev)
    g = torch.empty((p.ndf, 3), dtype=torch.float64, device=dev)
    kp = ctx.upload(p)

    def forces(x):
        torch.cuda.synchronize()
        if batch:
            ctx.forces_batch([kp, kp], [c.data_ptr(), x.data_ptr()], [p.n] * 2, nb, occ.data_ptr(),
                             [eps.data_ptr()] * 2, [g.data_ptr()] * 2)
        else:
            kp.forces(x.data_ptr(), p.n, nb, occ.data_ptr(), eps.data_ptr(), g.data_ptr())
        return g.cpu().numpy().copy()

    try:
        ctx.set_precision(lapw1gpu.PREC_SPLIT, 5)
        ctx.set_force_projection(slices, 64)
        assert p.nv > 64
        ref = forces(c)
        for x, hook, code in ((c, True, 5), (nan, False, 4), (nan, True, 5)):
            ctx.test_wait_timeout(hook)
            with pytest.raises(lapw1gpu.Lapw1GpuError) as e:
                forces(x)
            assert e.value.code == code
            ctx.test_wait_timeout(False)
            assert np.abs(forces(c) - ref).max() <= 1e-12 * np.abs(ref).max()
    finally:
        ctx.test_wait_timeout(False)
        ctx.set_force_projection(-1, 1024)
        ctx.set_precision(lapw1gpu.PREC_FP64)
        kp.free()
