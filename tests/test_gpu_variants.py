"""Every launch variant of the batched stencil, pinned by CVCB_SHAPE in a
child process (the autotuner caches one shape per configuration and
process): one rhs per thread with per-thread links, shared-memory links
for several rows, 2 and 4 rhs per thread, packed FP32x2 rhs pairs, and
(FP32 only, CVCB_PAIRS=1) the pair-tiled fields with 12- and 18-real
links, with a thread per site and with a site's directions on eight warps (4th
shape field 2); other 4th fields, 3 and 4 among them, run the former.
A wrong sloppy operator would still be corrected by the FP64 reliable
updates, so each variant must also converge in the same number of inner
iterations as the plain one (the arithmetic differs only in rounding)."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import json, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import cvc_b200 as cb
prec = int(sys.argv[2])
recon = int(sys.argv[3])
dims = (16, 8, 8, 8)
V = 16 * 8 ** 3
lat = cb.Lattice(*dims, kappa=0.155, mu=0.005 / 0.31)
lat.upload_gauge(cb.gauge_random(*dims, 0.25, 11))
bs = []
for i in range(11):                       # odd count: a lone last rhs in pair kernels
    b = np.zeros(24 * V); b[24 * (37 * i) + 2 * (i % 12)] = 1.0; bs.append(b)
xs = [np.zeros(24 * V) for _ in bs]
p = cb.solver_defaults(); p.precision = prec; p.block_rhs = 11; p.link_recon = recon
st = lat.solve(xs, bs, p)
r = np.zeros(24 * V); lat.Q_phi_tbc(r, xs[4])
print(json.dumps({"iters": st.iterations, "conv": st.converged, "res": st.max_true_res,
                  "chk": float(np.linalg.norm(r - bs[4]) / np.linalg.norm(bs[4])),
                  "x4": float(np.abs(xs[4]).sum())}))
"""

VARIANTS = ["64,1,1", "32,4,1", "64,1,2", "32,1,4", "64,1,2,1", "32,2,2,1"]
# (shape, CVCB_PAIRS, link reals) of the pair-tiled fields
PAIR_VARIANTS = [("64,1,2,1", 1, 12), ("32,2,2,1", 1, 12), ("64,1,2,1", 1, 18),
                 ("128,1,2,1", 1, 18), ("128,1,2,2", 1, 12), ("128,1,2,2", 1, 18),
                 ("128,1,2,3", 1, 12), ("128,1,2,3", 1, 18), ("128,1,2,4", 1, 12),
                 ("128,1,2,4", 1, 18)]


def run(prec, shape, pairs=0, recon=12):
    env = dict(os.environ, CVCB_SHAPE=shape, CVCB_PAIRS=str(pairs))
    out = subprocess.run([sys.executable, "-c", CHILD, str(ROOT), str(prec), str(recon)],
                         env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    return json.loads(out.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("prec", [1, 2], ids=["fp32", "fp16"])
def test_stencil_variants_agree(prec):
    res = {v: run(prec, v) for v in VARIANTS}
    if prec == 1:
        res.update({f"pairs {v} {r}": run(prec, v, pt, r) for v, pt, r in PAIR_VARIANTS})
    base = res["64,1,1"]
    print({v: r["iters"] for v, r in res.items()})
    for v, r in res.items():
        assert r["conv"] == 11, (v, r)
        assert r["res"] <= 1e-10 and r["chk"] <= 1e-10, (v, r)
        assert abs(r["iters"] - base["iters"]) <= 0.1 * base["iters"], (v, r, base)
        assert abs(r["x4"] - base["x4"]) <= 1e-8 * base["x4"], (v, r, base)


@pytest.mark.parametrize("recon", [12, 18])
def test_half_pairs_agree(recon):
    """FP16 fields tiled by rhs pairs (11 rhs: a lone last one) against the
    per-rhs FP16 fields: the same solutions, and no more iterations than the
    tolerance of the other variants (the links are FP32 instead of FP16)."""
    base = run(2, "64,1,2,1", 0, recon)
    for shape in ("64,1,2,1", "32,2,2,1"):
        r = run(2, shape, 1, recon)
        assert r["conv"] == 11 and r["res"] <= 1e-10 and r["chk"] <= 1e-10, r
        assert r["iters"] <= 1.1 * base["iters"], (r, base)
        assert abs(r["x4"] - base["x4"]) <= 1e-8 * base["x4"], (r, base)


SPLIT_CHILD = r"""
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
sys.path.insert(0, sys.argv[1] + "/tests")
import cvc_b200 as cb
from conftest import seeded
dims = tuple(int(v) for v in sys.argv[3].split("x"))
lat = cb.Lattice(*dims, kappa=0.14, mu=0.02, bc_angle=(1.0, 0.0, 0.5, 0.0))
lat.upload_gauge(cb.gauge_random(*dims, 0.3, 3))
V = lat.VOLUME
out = {}
for recon in (12, 18):
    for n in (1, 3):
        ins = [seeded(10 + i, 24 * V) for i in range(n)]
        outs = [np.zeros(24 * V) for _ in range(n)]
        lat.sloppy_normal_op(ins, outs, cb.PREC_SINGLE, recon, 1)
        out["op%d_%d" % (recon, n)] = np.array(outs)
        p = cb.solver_defaults()
        p.link_recon, p.block_rhs = recon, n
        xs = [np.zeros(24 * V) for _ in range(n)]
        st = lat.solve(xs, ins, p)
        assert st.converged == n and st.max_true_res <= 1e-10
        out["x%d_%d" % (recon, n)] = np.array(xs)
        out["it%d_%d" % (recon, n)] = np.array([st.iterations])
np.savez(sys.argv[2], **out)
"""


@pytest.mark.parametrize("dims", ["2x2x2x2", "2x2x6x10", "6x4x2x14"])
def test_directions_on_warps_same_bits(tmp_path, dims):
    """The kernel with a site's directions on eight warps against the one with
    a thread per site: the operator to the last bit, the solves to their 1e-10
    residual (the norms sum in another order) and iteration count, on half
    volumes below and off whole tiles of 32, for lone and paired rhs."""
    import numpy as np
    got = []
    for shape in ("64,1,2,1", "32,1,2,2"):
        f = tmp_path / (shape.replace(",", "_") + ".npz")
        out = subprocess.run([sys.executable, "-c", SPLIT_CHILD, str(ROOT), str(f), dims],
                             env=dict(os.environ, CVCB_SHAPE=shape, CVCB_PAIRS="1"),
                             capture_output=True, text=True, timeout=600)
        assert out.returncode == 0, out.stderr[-2000:]
        got.append(np.load(f))
    a, b = got
    for k in a.files:
        if k.startswith("op"):
            assert np.array_equal(a[k], b[k]), k
        elif k.startswith("it"):
            assert abs(int(a[k][0]) - int(b[k][0])) <= 3 + 0.1 * a[k][0], k
        else:
            assert np.max(np.abs(a[k] - b[k])) <= 1e-8 * np.max(np.abs(a[k])), k


ODD_CHILD = r"""
import ctypes, json, os, sys
import numpy as np
for v in ("CVCB_SHAPE", "CVCB_PAIRS"):
    os.environ.pop(v, None)
sys.path.insert(0, sys.argv[1])
import cvc_b200 as cb
dims = (8, 4, 4, 6)
lat = cb.Lattice(*dims, kappa=0.14, mu=0.02)
lat.upload_gauge(cb.gauge_random(*dims, 0.3, 3))
V = lat.VOLUME
out = {}
for n in (1, 2, 3, 15, 17):
    bs = []
    for i in range(n):
        b = np.zeros(24 * V); b[24 * (11 * i % V) + 2 * (i % 12)] = 1.0; bs.append(b)
    xs = [np.zeros(24 * V) for _ in range(n)]
    p = cb.solver_defaults(); p.precision = cb.PREC_HALF; p.block_rhs = n
    st = lat.solve(xs, bs, p)
    v = [ctypes.c_int() for _ in range(4)]
    rc = lat._lib.cvcb_tuned_shape(lat._h, cb.PREC_HALF, 12, n, *[ctypes.byref(q) for q in v])
    r = np.zeros(24 * V); lat.Q_phi_tbc(r, xs[-1])
    out[n] = [rc, v[3].value, st.converged, float(np.linalg.norm(r - bs[-1]))]
print(json.dumps(out))
"""


def test_half_takes_pairs_only_where_no_lane_idles():
    """FP16 batches of an odd number of columns up to 15 run on the per-rhs
    fields (in pairs one column took up to twice the time), even and larger
    ones on pair-tiled fields (variant 3 of cvcb_tuned_shape)."""
    r = subprocess.run([sys.executable, "-c", ODD_CHILD, str(ROOT)], capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    for n, (rc, variant, conv, res) in json.loads(r.stdout.strip().splitlines()[-1]).items():
        n = int(n)
        assert rc == 0 and conv == n and res <= 1e-10, (n, rc, conv, res)
        assert (variant == 3) == (n % 2 == 0 or n > 15), (n, variant)


BITS_CHILD = r"""
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
sys.path.insert(0, sys.argv[1] + "/tests")
import cvc_b200 as cb
from conftest import seeded
dims, prec = tuple(int(v) for v in sys.argv[3].split("x")), int(sys.argv[4])
lat = cb.Lattice(*dims, kappa=0.14, mu=0.02, bc_angle=(1.0, 0.0, 0.5, 0.0))
lat.upload_gauge(cb.gauge_random(*dims, 0.3, 3))
V = lat.VOLUME
bs = [seeded(20 + i, 24 * V) for i in range(15)]
xs = [np.zeros(24 * V) for _ in bs]
p = cb.solver_defaults()
p.precision = prec
st = []
for k, n in [(i, 1) for i in range(12)] + [(12, 3)]:
    p.block_rhs = n
    s = lat.solve(xs[k:k + n], bs[k:k + n], p)
    assert s.converged == n
    st += [s.iterations, s.max_true_res]
np.savez(sys.argv[2], x=np.array(xs), st=np.array(st))
"""


@pytest.mark.parametrize("dims", ["2x2x6x10", "8x6x8x10"])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_solve_bits_do_not_depend_on_the_shape(tmp_path, prec, dims):
    """Two processes whose tuners take different shapes return the same bits,
    of the solutions and of the residuals: the norms behind alpha, beta and the
    residuals sum in one order for every shape (rows of 16 sites and of whole
    warps, one thread or eight warps a site), on half volumes of 120 and 1920
    sites, for lone columns and three together."""
    import numpy as np
    shapes = (["64,1,1", "16,1,1", "16,3,1", "32,3,1", "128,1,1"] if prec == 0 else
              ["64,1,2,1", "32,1,2,2", "32,2,2,1", "256,1,2,1"])
    got = []
    for shape in shapes:
        f = tmp_path / (shape.replace(",", "_") + ".npz")
        out = subprocess.run([sys.executable, "-c", BITS_CHILD, str(ROOT), str(f), dims, str(prec)],
                             env=dict(os.environ, CVCB_SHAPE=shape, CVCB_PAIRS="1"),
                             capture_output=True, text=True, timeout=600)
        assert out.returncode == 0, out.stderr[-2000:]
        got.append(np.load(f))
    for shape, g in zip(shapes[1:], got[1:]):
        assert np.array_equal(g["st"], got[0]["st"]), (shape, g["st"] - got[0]["st"])
        assert np.array_equal(g["x"], got[0]["x"]), shape


def test_half_takes_rows_that_are_no_whole_warps():
    """CVCB_SHAPE with 16 or 48 sites in a row: FP16 solves run whether their
    fields are tiled by pairs or not."""
    for shape in ("16,4,1", "48,1,1", "48,5,2,1"):
        for pairs in (0, 1):
            r = run(2, shape, pairs)
            assert r["conv"] == 11 and r["res"] <= 1e-10 and r["chk"] <= 1e-10, (shape, pairs, r)


CODE_CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import cvc_b200 as cb
lat = cb.Lattice(8, 4, 4, 4, kappa=0.14, mu=0.02)
lat.upload_gauge(cb.gauge_random(8, 4, 4, 4, 0.3, 3))
b = np.zeros(24 * 512); b[0] = 1.0
lat.solve([np.zeros(24 * 512)], [b])
v = [ctypes.c_int() for _ in range(4)]
lat._lib.cvcb_tuned_shape(lat._h, cb.PREC_SINGLE, 12, 1, *[ctypes.byref(q) for q in v])
print(*[q.value for q in v])
"""


@pytest.mark.parametrize("shape,want", [("64,1,2,1", [64, 1, 2, 3]), ("32,1,2,2", [32, 1, 2, 7])])
def test_variant_codes(shape, want):
    """cvcb_tuned_shape names the kernel that a pinned shape runs; the codes 4
    to 6 of kernels that are gone do not come back with another meaning."""
    r = subprocess.run([sys.executable, "-c", CODE_CHILD, str(ROOT)], capture_output=True, text=True,
                       env=dict(os.environ, CVCB_SHAPE=shape, CVCB_PAIRS="1"), timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    assert [int(t) for t in r.stdout.split()] == want
