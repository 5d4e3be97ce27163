"""cvcb_time_stencil, the timing entry point behind the profiles and the
benchmark's stencil figures: every kind runs on a small lattice and returns a
positive time; an unknown kind is an argument error, not a launch."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [1, 2], ids=["fp32", "fp16"])
def test_every_kind_times(cb, prec):
    dims = (16, 8, 8, 8)
    lat = cb.Lattice(*dims, kappa=0.155, mu=0.005 / 0.31)
    lat.upload_gauge(cb.gauge_random(*dims, 0.25, 11))
    ms = ctypes.c_double()
    for kind in (0, 1, 2, 3):
        rc = lat._lib.cvcb_time_stencil(lat._h, kind, prec, 12, 6, 3, ctypes.byref(ms))
        assert rc == 0, (kind, cb.last_error())
        assert ms.value > 0, kind
    for kind in (-1, 4):
        ms.value = 0.0
        rc = lat._lib.cvcb_time_stencil(lat._h, kind, prec, 12, 6, 3, ctypes.byref(ms))
        assert rc == cb._lib.CVCB_ERR_ARG and ms.value == 0.0, kind
    lat.close()


@pytest.mark.parametrize("dims", [(8, 4, 4, 4), (12, 10, 10, 10)])
def test_kind_0_times_the_kernel_of_the_operator(cb, dims):
    """Kind 0 launches the kernel that Q_phi_tbc launches, on both sides of the
    volume where that one changes."""
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile
    lat = cb.Lattice(*dims, kappa=0.155, mu=0.005 / 0.31)
    lat.upload_gauge(cb.gauge_random(*dims, 0.25, 11))
    phi = torch.zeros(24 * lat.VOLUME, dtype=torch.float64, device="cuda")
    xi = torch.zeros_like(phi)
    ms = ctypes.c_double()

    def kernels(fn):
        fn()  # first-use tuning is over
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            fn()
            torch.cuda.synchronize()
        return {e.name for e in prof.events() if "k_tm_full" in e.name}

    op = kernels(lambda: lat.Q_phi_tbc(xi, phi))
    if not op:
        pytest.skip("the profiler reports no kernels")
    timed = kernels(lambda: lat._lib.cvcb_time_stencil(lat._h, 0, 0, 18, 1, 2, ctypes.byref(ms)))
    assert len(op) == 1 and timed == op
    lat.close()
