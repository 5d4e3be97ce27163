"""Operators and reductions on the GPU against the oracle (Q_phi.c,
invert_Qtm.c:28-84).  FP64 throughout; the CUDA kernels sum in a different
order (and use FMA), so agreement is to a few units of double rounding:
tolerance 1e-14 relative to the largest component."""
import numpy as np
import pytest

from conftest import rel_err, seeded

pytestmark = pytest.mark.gpu

TOL = 1e-14
CASES = [
    ((8, 4, 4, 4), 0.15, 0.01 / 0.3, (1.0, 0.0, 0.0, 0.0)),
    ((16, 8, 8, 8), 0.15, 0.01 / 0.3, (1.0, 0.0, 0.0, 0.0)),
    ((8, 6, 4, 2), 0.137, -0.05, (1.0, 0.5, 0.0, 0.25)),
]


@pytest.fixture(scope="module", params=CASES, ids=["4^3x8", "8^3x16", "8x6x4x2-bc"])
def setup(request, cb, oracle_mod):
    dims, kappa, mu, bc = request.param
    lat = cb.Lattice(*dims, kappa=kappa, mu=mu, bc_angle=bc)
    g = cb.gauge_random(*dims, 0.3, 1234)
    lat.upload_gauge(g)
    orc = oracle_mod.Oracle(*dims, kappa, mu, bc)
    orc.set_gauge(g)
    V = lat.VOLUME
    phi = seeded(11, 24 * V)
    yield lat, orc, phi, V, kappa, mu
    lat.close()


def test_Q_phi_tbc(setup):
    lat, orc, phi, V, *_ = setup
    xi = np.zeros_like(phi)
    lat.Q_phi_tbc(xi, phi)
    assert rel_err(xi, orc.Q_phi_tbc(phi)) < TOL


def test_Hopping(setup):
    lat, orc, phi, V, *_ = setup
    xi = np.zeros_like(phi)
    lat.Hopping(xi, phi)
    assert rel_err(xi, orc.Hopping(phi)) < TOL


@pytest.mark.parametrize("sgn", [1.0, -1.0])
def test_Qf5(setup, sgn):
    lat, orc, phi, V, kappa, mu = setup
    xi = np.zeros_like(phi)
    lat.Qf5(xi, phi, sgn * mu)
    assert rel_err(xi, orc.Qf5(phi, sgn * mu)) < TOL


def test_Q_phi_explicit_mu(setup):
    lat, orc, phi, *_ = setup
    xi = np.zeros_like(phi)
    lat.Q_phi(xi, phi, 0.0731)
    assert rel_err(xi, orc.Q_phi(phi, 0.0731)) < TOL


def test_g5_and_imu(setup):
    lat, orc, phi, V, *_ = setup
    a = phi.copy()
    lat.g5_phi(a)
    assert np.array_equal(a, orc.g5_phi(phi))
    for sign, nv in [(1.0, V), (-1.0, V), (1.0, V // 2 + 3)]:
        b = phi.copy()
        lat.mul_one_pm_imu_inv(b, sign, nv)
        assert rel_err(b, orc.mul_one_pm_imu_inv(phi, sign, nv)) < TOL


def test_scalar_products(setup):
    lat, orc, phi, V, *_ = setup
    psi = seeded(12, 24 * V)
    for nv in (V, V // 3, 1):
        w = lat.spinor_scalar_product_co(phi, psi, nv)
        ref = orc.scalar_product_co(phi, psi, nv)
        assert abs(w - ref) <= 1e-13 * max(abs(ref), 1.0)
        r = lat.spinor_scalar_product_re(phi, psi, nv)
        assert abs(r - ref.real) <= 1e-13 * max(abs(ref), 1.0)
    # deterministic: identical bits on repeated calls
    w1 = lat.spinor_scalar_product_co(phi, psi, V)
    w2 = lat.spinor_scalar_product_co(phi, psi, V)
    assert w1 == w2


def test_gamma5_hermiticity(setup):
    """Q(mu)^dagger = g5 Q(-mu) g5: <a, Q(mu) b> = <g5 Q(-mu) g5 a, b>."""
    lat, orc, phi, V, kappa, mu = setup
    psi = seeded(13, 24 * V)
    qb = np.zeros_like(phi)
    lat.Q_phi(qb, psi, mu)
    lhs = lat.spinor_scalar_product_co(phi, qb, V)
    t = phi.copy()
    lat.g5_phi(t)
    u = np.zeros_like(phi)
    lat.Qf5(u, t, -mu)  # g5 Q(-mu) g5 phi
    rhs = lat.spinor_scalar_product_co(u, psi, V)
    assert abs(lhs - rhs) <= 1e-12 * abs(lhs)


def test_device_pointers(setup):
    """The same entry points accept CUDA device memory (torch tensors)."""
    torch = pytest.importorskip("torch")
    lat, orc, phi, V, *_ = setup
    d_phi = torch.from_numpy(phi).cuda()
    d_xi = torch.zeros_like(d_phi)
    lat.Q_phi_tbc(d_xi, d_phi)
    torch.cuda.synchronize()
    assert rel_err(d_xi.cpu().numpy(), orc.Q_phi_tbc(phi)) < TOL
    w = lat.spinor_scalar_product_co(d_phi, d_xi, V)
    ref = orc.scalar_product_co(phi, d_xi.cpu().numpy(), V)
    assert abs(w - ref) <= 1e-13 * abs(ref)


def test_plaquette(setup):
    lat, orc, *_ = setup
    pl, ls = lat.plaquette()
    opl, ols = orc.plaquette()
    assert abs(pl - opl) < 1e-14
    assert abs(ls - ols) < 1e-12 * abs(ols)


def test_errors(cb):
    lat = cb.Lattice(4, 4, 4, 4)
    phi = np.zeros(24 * lat.VOLUME)
    with pytest.raises(cb.CvcbError) as e:
        lat.Q_phi_tbc(phi.copy(), phi)  # no gauge field yet
    assert e.value.code == -5
    with pytest.raises(cb.CvcbError):
        cb.Lattice(3, 4, 4, 4)  # odd extent
    lat.close()


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 6, 4, 10), (4, 2, 14, 6), (6, 10, 14, 12),
                                  (14, 2, 10, 34), (2, 2, 2, 1030)],
                         ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("where", ["host", "device", "device16", "to_host", "in_place"])
def test_operator_on_cvc_fields(cb, oracle_mod, dims, where):
    """The operator on site-major arrays, below and above the volume up to which
    a site's directions go to eight warps: extents of two (both hops reach the
    same site), rows that cross warps, a last block and a last warp that are not
    full, fields on 32- and on 16-byte boundaries, mixed memories, and input and
    output the same array."""
    torch = pytest.importorskip("torch")
    bc = (1.0, 0.0, 0.25, 0.5)
    lat = cb.Lattice(*dims, kappa=0.14, mu=0.03, bc_angle=bc)
    V = lat.VOLUME
    g = cb.gauge_random(*dims, 0.3, 4)
    lat.upload_gauge(g)
    orc = oracle_mod.Oracle(*dims, 0.14, 0.03, bc)
    orc.set_gauge(g)
    phi = seeded(6, 24 * V)

    def dev(off):
        t = torch.zeros(24 * V + 4, dtype=torch.float64, device="cuda")[off:24 * V + off]
        t.copy_(torch.from_numpy(phi))
        torch.cuda.synchronize()
        return t

    for name, extra in (("Q_phi_tbc", ()), ("Qf5", (-0.02,)), ("Hopping", ())):
        x = phi.copy() if where == "host" else dev(2 if where == "device16" else 0)
        y = x if where == "in_place" else np.zeros(24 * V) if where in ("host", "to_host") else \
            torch.zeros_like(x)
        torch.cuda.synchronize()
        getattr(lat, name)(y, x, *extra)
        got = y if isinstance(y, np.ndarray) else y.cpu().numpy()
        assert rel_err(got, getattr(orc, name)(phi, *extra)) < 1e-14
    lat.close()


def test_lattice_set_up_pins_no_memory(cb):
    """Making a lattice and freeing it takes less than one pinned allocation
    and its release alone, which it therefore cannot contain."""
    import ctypes
    import time
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    lib = ctypes.CDLL([line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line][0])
    p = ctypes.c_void_p()

    def pinned():
        assert lib.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(4), 2) == 0
        assert lib.cudaFreeHost(p) == 0

    def median(fn):
        t = []
        for _ in range(25):
            t0 = time.perf_counter()
            fn()
            t.append(time.perf_counter() - t0)
        return sorted(t)[12]

    def lattice():
        cb.Lattice(8, 4, 4, 4).close()

    lattice()
    pinned()
    made, pin = median(lattice), median(pinned)
    print(f"lattice {1e6 * made:.0f} us, pinned allocation {1e6 * pin:.0f} us")
    assert made < pin
