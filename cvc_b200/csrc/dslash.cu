// Full-lattice FP64 twisted-mass Wilson operator with per-link boundary
// phases: k_tm_full_cvc and k_tm_full_cvc_split behind Q_phi_tbc, Q_phi, Qf5
// and Hopping, k_tm_full_f64 behind the FP64 solvers and the hopping expansion.
//
//   out(x) = a in(x) + i b g5 in(x)
//          + c sum_mu [ (1 - g_mu) U_mu(x) in(x+mu) + (1 + g_mu) U_mu(x-mu)^+ in(x-mu) ]
//   (then out = g5 out when g5out)
//
// Q_phi_tbc (Q_phi.c:38-188): a = 1/(2 kappa), b = mu, c = -1/2.
// Q_phi(mutm) (Q_phi.c:1092-1242): b = mutm.  Qf5(mutm) (Q_phi.c:789-934):
// b = mutm, g5out.  Hopping (Q_phi.c:399-528): a = b = 0, c = -kappa.
//
// One thread per output site; both parities in one launch.  The stencil is
// HBM-bound: per site it must read 8 neighbour spinors (mostly L1/L2 hits:
// each spinor is used by 8 sites), 8 links (each used by 2 sites), its own
// spinor, and write one spinor.  Compulsory traffic 2*192 + 4*144 = 960 B.
#include "bicgstab.cuh"
#include "cvcb_internal.h"
#include "spinor_ops.cuh"

namespace cvcb {

// DOT: the scalar products that BiCGStab takes of the result (TmDot) come from
// the registers of the sweep: one field read instead of two and a launch
// less.  Per-block partials, summed by the last block in block order.
template <int NT>
__device__ __forceinline__ void tm_dot_finish(const TmDot &D, double (&v)[3]) {
  __shared__ double sh[3][NT / 32];
  __shared__ bool last;
  auto reduce = [&] {
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int q = 0; q < 3; ++q) sh[q][threadIdx.x >> 5] = v[q];
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        v[q] = sh[q][0];
        for (int w = 1; w < NT / 32; ++w) v[q] += sh[q][w];
      }
  };
  reduce();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 3; ++q) D.partials[(size_t)blockIdx.x * 3 + q] = v[q];
    __threadfence();
    last = atomicAdd(D.counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += NT)
#pragma unroll
    for (int q = 0; q < 3; ++q) v[q] += __ldcg(D.partials + (size_t)b * 3 + q);
  __syncthreads();
  reduce();
  if (threadIdx.x == 0) {
    *D.counter = 0;
    if (D.kind == 1)
      epi_alpha(D.S, v[0], v[1]);
    else
      epi_omega(D.S, v[0], v[1], v[2]);
  }
}

template <bool G5OUT, bool DOT, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_tm_full_f64(double2 *__restrict__ out,
                                                     const double2 *__restrict__ in,
                                                     const double2 *__restrict__ U, Geom g,
                                                     double a, double b, double c,
                                                     const int *__restrict__ done, TmDot D) {
  if (done && *done) return;
  // Blocks alternate between the parities (block 2k: even sites of range k,
  // block 2k+1: odd sites of range k).  A link serves the forward hop of one
  // parity and the backward hop of the other; with the parities interleaved
  // its second use follows the first by a few MB of traffic and finds it in
  // L2, where parity after parity would read all links from DRAM twice.
  const int p = blockIdx.x & 1;
  const int i = (blockIdx.x >> 1) * blockDim.x + threadIdx.x;
  double dv[3] = {0.0, 0.0, 0.0};
  if (i < g.Vh) {
  const int s = p * g.Vh + i;
  const SiteCoord cd = site_coord(g, p, i);
  const size_t V = g.V;
  const int qoff = (1 - p) * g.Vh;

  Spinor<double> acc;
#pragma unroll
  for (int sp = 0; sp < 4; ++sp)
#pragma unroll
    for (int co = 0; co < 3; ++co) acc.c[sp][co] = cx(0.0, 0.0);

#pragma unroll
  for (int mu = 0; mu < 4; ++mu) {
    {  // backward: (1 + g_mu) U_mu(x-mu)^+ in(x-mu)
      const int j = qoff + (nb_lex(g, cd, mu, -1) >> 1);
      const HalfSpinor<double> h = project(mu, +1, load_spinor(in, V, j));
      const Link<double> W = load_link64(U, V, mu, j);
      accum_recon(mu, +1, acc, link_dag_mul(W, h));
    }
    {  // forward: (1 - g_mu) U_mu(x) in(x+mu)
      const int j = qoff + (nb_lex(g, cd, mu, +1) >> 1);
      const HalfSpinor<double> h = project(mu, -1, load_spinor(in, V, j));
      const Link<double> W = load_link64(U, V, mu, s);
      accum_recon(mu, -1, acc, link_mul(W, h));
    }
  }

  const Spinor<double> f = load_spinor(in, V, s);
  Spinor<double> r;
#pragma unroll
  for (int sp = 0; sp < 4; ++sp) {
    const double bs = sp < 2 ? b : -b;  // i b g5
#pragma unroll
    for (int co = 0; co < 3; ++co) {
      const Cx<double> v = f.c[sp][co];
      Cx<double> o;
      o.re = fma(c, acc.c[sp][co].re, fma(a, v.re, -bs * v.im));
      o.im = fma(c, acc.c[sp][co].im, fma(a, v.im, bs * v.re));
      if (G5OUT && sp >= 2) o = cx(-o.re, -o.im);
      r.c[sp][co] = o;
    }
  }
  store_spinor(out, V, s, r);
  if (DOT) {
    const Spinor<double> f2 = load_spinor(D.f, V, s);
    Cx<double> d = cx(0.0, 0.0);
#pragma unroll
    for (int sp = 0; sp < 4; ++sp)
#pragma unroll
      for (int co = 0; co < 3; ++co) {
        const Cx<double> o = r.c[sp][co];
        cfmac(d, f2.c[sp][co], o);  // <f, out>
        dv[2] = fma(o.re, o.re, dv[2]);
        dv[2] = fma(o.im, o.im, dv[2]);
      }
    dv[0] = d.re;
    dv[1] = D.kind == 1 ? d.im : -d.im;  // kind 2: <out, f>
  }
  }  // i < Vh
  if (DOT) tm_dot_finish<NT>(D, dv);
}

// Launch variants: blocks of 128 threads, with or without the registers capped
// for three resident blocks per SM (the caps for four and eight spill and were
// never chosen).  Chosen once per process by timing.
constexpr int kTmThreads = 128;
int tm_full_blocks(const Geom &g) { return 2 * ((g.Vh + kTmThreads - 1) / kTmThreads); }

template <int MINB>
static void launch_variant(cvcb_lattice *L, double2 *out, const double2 *in, double a, double b,
                           double c, bool g5out, const int *done, const TmDot *dot) {
  const Geom &g = L->g;
  const int blocks = tm_full_blocks(g);  // both parities, interleaved
  auto kern = g5out ? (dot ? k_tm_full_f64<true, true, kTmThreads, MINB> : k_tm_full_f64<true, false, kTmThreads, MINB>)
                    : (dot ? k_tm_full_f64<false, true, kTmThreads, MINB> : k_tm_full_f64<false, false, kTmThreads, MINB>);
  kern<<<blocks, kTmThreads, 0, L->stream>>>(out, in, L->U64, g, a, b, c, done, dot ? *dot : TmDot{});
}

static int g_tm_variant = -1;

static void launch_by_variant(int v, cvcb_lattice *L, double2 *out, const double2 *in, double a,
                              double b, double c, bool g5out, const int *done, const TmDot *dot) {
  if (v == 1)
    launch_variant<1>(L, out, in, a, b, c, g5out, done, dot);
  else
    launch_variant<3>(L, out, in, a, b, c, g5out, done, dot);
}

int launch_tm_full(cvcb_lattice *L, double2 *out, const double2 *in, double a, double b, double c,
                   bool g5out, const int *done, const TmDot *dot) {
  if (g_tm_variant < 0) {
    // one-time choice: time each variant on this lattice (output to `out`,
    // which the real launch below overwrites)
    cudaEvent_t e0, e1;
    CVCB_CUDA(cudaEventCreate(&e0));
    CVCB_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    int bestv = 0;
    for (int v = 0; v < 2; ++v) {
      launch_by_variant(v, L, out, in, a, b, c, g5out, nullptr, nullptr);
      CVCB_CUDA(cudaEventRecord(e0, L->stream));
      for (int k = 0; k < 5; ++k) launch_by_variant(v, L, out, in, a, b, c, g5out, nullptr, nullptr);
      CVCB_CUDA(cudaEventRecord(e1, L->stream));
      CVCB_CUDA(cudaEventSynchronize(e1));
      float ms;
      CVCB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      if (ms < best) {
        best = ms;
        bestv = v;
      }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    g_tm_variant = bestv;
  }
  launch_by_variant(g_tm_variant, L, out, in, a, b, c, g5out, done, dot);
  CVCB_LAUNCHED(L);
  return CVCB_OK;
}

// The same operator on CVC-layout fields (192 contiguous bytes per site), for
// the entry points that apply it once: no copy into and out of the device
// layout, which cost two field passes more than the operator itself.  Thread =
// lexicographic site; a spinor is six 32-byte loads (one whole sector each; V4)
// or twelve 16-byte ones (fields off a 32-byte boundary).  Same terms in the
// same order as k_tm_full_f64: the same bits.
template <bool V4>
__device__ __forceinline__ Spinor<double> load_spinor_cvc(const double2 *__restrict__ f, int lex) {
  const double2 *q = f + (size_t)lex * 12;
  Spinor<double> s;
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    Cx<double> a, b;
    if (V4) {
      asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                   : "=d"(a.re), "=d"(a.im), "=d"(b.re), "=d"(b.im)
                   : "l"(q + 2 * m));
    } else {
      const double2 v = __ldg(q + 2 * m), w = __ldg(q + 2 * m + 1);
      a = cx(v.x, v.y);
      b = cx(w.x, w.y);
    }
    s.c[(2 * m) / 3][(2 * m) % 3] = a;
    s.c[(2 * m + 1) / 3][(2 * m + 1) % 3] = b;
  }
  return s;
}

template <bool V4>
__device__ __forceinline__ void store_spinor_cvc(double2 *f, int lex, const Spinor<double> &s) {
  double2 *q = f + (size_t)lex * 12;
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const Cx<double> a = s.c[(2 * m) / 3][(2 * m) % 3], b = s.c[(2 * m + 1) / 3][(2 * m + 1) % 3];
    if (V4) {
      asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(q + 2 * m), "d"(a.re), "d"(a.im),
                   "d"(b.re), "d"(b.im)
                   : "memory");
    } else {
      q[2 * m] = make_double2(a.re, a.im);
      q[2 * m + 1] = make_double2(b.re, b.im);
    }
  }
}

constexpr int kCvcThreads = 128, kCvcWarps = kCvcThreads / 32;
constexpr int kCvcStage = 32 * 12;  // double2: the spinors of a warp's 32 sites in one direction
constexpr int kCvcSmem = kCvcWarps * 2 * kCvcStage * (int)sizeof(double2);  // 48 KB

__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// The spinors at lex index j of every lane's site into the warp's stage, in
// lane order: one bulk copy for each run of consecutive indices (a direction's
// neighbours of 32 consecutive sites are one run but for the periodic wraps).
__device__ __forceinline__ void cvc_fetch(double2 *stage, unsigned long long *bar,
                                          const double2 *__restrict__ in, int j, int lane) {
  const int before = __shfl_up_sync(0xffffffffu, j, 1);
  const bool first = lane == 0 || j != before + 1;
  const unsigned starts = __ballot_sync(0xffffffffu, first);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (lane == 0)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"((unsigned)(kCvcStage * sizeof(double2)))
                 : "memory");
  __syncwarp();
  if (first) {
    const unsigned later = lane == 31 ? 0u : starts >> (lane + 1);
    const int len = later ? __ffs(later) : 32 - lane;
    asm volatile(
        "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(stage + lane * 12)),
        "l"(in + (size_t)j * 12), "r"(len * 192), "r"(smem_addr(bar))
        : "memory");
  }
}
__device__ __forceinline__ bool cvc_landed(unsigned long long *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok;
}
// until the stage's copies have landed, for every lane; false after
// kCvcWaitSeconds (looked at once more then: the warp may have been paused in
// between)
__device__ __forceinline__ bool cvc_wait(unsigned long long *bar, unsigned parity) {
  if (__all_sync(0xffffffffu, cvc_landed(bar, parity))) return true;
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
  do {
    if (__all_sync(0xffffffffu, cvc_landed(bar, parity))) return true;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  } while (!__any_sync(0xffffffffu, t - t0 > (unsigned long long)(1e9 * kCvcWaitSeconds)));
  return __all_sync(0xffffffffu, cvc_landed(bar, parity));
}
// A lane's spinor.  Its 192 bytes start on one of two bank quarters, so lanes
// read their components from different starting points (lane / 2 mod 4) and
// rotate them into place afterwards: no bank conflicts.
__device__ __forceinline__ Spinor<double> cvc_spinor(const double2 *stage, int lane) {
  const int d = (lane >> 1) & 3;
  const double2 *q = stage + lane * 12;
  double2 v[12], w[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) v[k] = q[k + d < 12 ? k + d : k + d - 12];
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    w[k].x = d & 1 ? v[(k + 11) % 12].x : v[k].x;
    w[k].y = d & 1 ? v[(k + 11) % 12].y : v[k].y;
  }
  Spinor<double> s;
#pragma unroll
  for (int k = 0; k < 12; ++k)
    s.c[k / 3][k % 3] = cx(d & 2 ? w[(k + 10) % 12].x : w[k].x, d & 2 ? w[(k + 10) % 12].y : w[k].y);
  return s;
}

// A warp has 32 consecutive sites.  Their neighbours in a direction are brought
// into shared memory by bulk copies, two directions ahead of the arithmetic, and
// every lane reads its own from there.  Loads from the fields directly, 32 bytes
// a lane and 192 apart, keep the L1 data pipe 82 % busy: 29.4 us a call at
// 22 x 14 x 10 x 18 and 588 at 32^3 x 64, now 27.6 and 523 (with copies to and
// from the device layout 44 and 818); compulsory traffic there 2.0 GB, 0.31 ms.
// cp.async instead of bulk copies: 644.  More stages cost L1, which the links
// need: three 605, four 646.  Padding against bank conflicts instead of the
// rotation makes the copies small: 557 in fours, 581 in pairs.  A tile of the
// block's own sites for z, y and the diagonal term: 537.
template <bool G5OUT, bool V4>
__global__ void __launch_bounds__(kCvcThreads, 3)
    k_tm_full_cvc(double2 *__restrict__ out, const double2 *__restrict__ in,
                  const double2 *__restrict__ U, Geom g, double a, double b, double c, unsigned *late) {
  extern __shared__ __align__(128) double2 cvc_sm[];
  __shared__ unsigned long long bars[kCvcWarps][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2 *const st = cvc_sm + warp * 2 * kCvcStage;
  unsigned long long *const bar = bars[warp];
  const int want = blockIdx.x * kCvcThreads + threadIdx.x;
  if (want - lane >= g.V) return;  // the whole warp
  const bool valid = want < g.V;
  const int lex = valid ? want : g.V - 1;  // idle lanes take part in the copies
  if (lane < 2)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar + lane)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncwarp();
  SiteCoord cd;
  {
    const unsigned r0 = fdiv((unsigned)lex, g.dLZ), r1 = fdiv(r0, g.dLY), r2 = fdiv(r1, g.dLX);
    cd.lex = lex;
    cd.z = lex - (int)r0 * g.LZ;
    cd.y = (int)(r0 - r1 * g.LY);
    cd.x = (int)(r1 - r2 * g.LX);
    cd.t = (int)r2;
  }
  const int par = (cd.t + cd.x + cd.y + cd.z) & 1;
  const int self = par * g.Vh + (lex >> 1), qoff = (1 - par) * g.Vh;
  const size_t V = g.V;

  Spinor<double> acc;
#pragma unroll
  for (int sp = 0; sp < 4; ++sp)
#pragma unroll
    for (int co = 0; co < 3; ++co) acc.c[sp][co] = cx(0.0, 0.0);
  cvc_fetch(st, bar, in, nb_lex(g, cd, 0, -1), lane);
  cvc_fetch(st + kCvcStage, bar + 1, in, nb_lex(g, cd, 0, +1), lane);
#pragma unroll
  for (int d = 0; d < 8; ++d) {  // t-, t+, x-, x+, ...
    const int mu = d >> 1;
    const bool fwd = d & 1;
    const Link<double> W = load_link64(U, V, mu, fwd ? self : qoff + (nb_lex(g, cd, mu, -1) >> 1));
    if (!cvc_wait(bar + (d & 1), (d >> 1) & 1)) {
      *late = 1;
      cvc_wait(bar + (1 - (d & 1)), ((d + 1) >> 1) & 1);  // the copies in flight
      return;
    }
    const HalfSpinor<double> h = project(mu, fwd ? -1 : +1, cvc_spinor(st + (d & 1) * kCvcStage, lane));
    __syncwarp();  // every lane has read the stage
    if (d < 7)
      cvc_fetch(st + (d & 1) * kCvcStage, bar + (d & 1), in,
                d == 6 ? lex : nb_lex(g, cd, (d + 2) >> 1, fwd ? +1 : -1), lane);
    accum_recon(mu, fwd ? -1 : +1, acc, fwd ? link_mul(W, h) : link_dag_mul(W, h));
  }
  if (!cvc_wait(bar, 0)) {  // the fifth use of stage 0
    *late = 1;
    return;
  }
  const Spinor<double> f = cvc_spinor(st, lane);
  if (!valid) return;
  Spinor<double> r;
#pragma unroll
  for (int sp = 0; sp < 4; ++sp) {
    const double bs = sp < 2 ? b : -b;  // i b g5
#pragma unroll
    for (int co = 0; co < 3; ++co) {
      const Cx<double> v = f.c[sp][co];
      Cx<double> o;
      o.re = fma(c, acc.c[sp][co].re, fma(a, v.re, -bs * v.im));
      o.im = fma(c, acc.c[sp][co].im, fma(a, v.im, bs * v.re));
      if (G5OUT && sp >= 2) o = cx(-o.re, -o.im);
      r.c[sp][co] = o;
    }
  }
  store_spinor_cvc<V4>(out, lex, r);
}

// The same for small lattices, where the GPU waits for one site's directions one
// after the other: block = 32 lexicographic sites, warp d = direction (t-, t+,
// x-, ...), every warp loads one neighbour and leaves its transported half
// spinor in shared memory, warps 0..2 sum the sink colours 0..2 in the order
// of the kernels above (the same bits) and add the diagonal.
constexpr int kCvcSplitThreads = 256;
// Up to here: 14.2 against 16.7 us a call at 512 sites, 16.1 against 18.4 at
// 8192; at 12,000 18.8 against 18.2, at 55,440 32.6 against 27.
constexpr int kCvcSplitSites = 8192;

template <int MU, bool DAG, bool V4>
__device__ __forceinline__ void cvc_split_dir(double2 (*sh)[32], const double2 *__restrict__ in,
                                              const double2 *__restrict__ U, const Geom &g,
                                              const SiteCoord &cd, int self, int qoff, int lane) {
  const int j = nb_lex(g, cd, MU, DAG ? -1 : +1);
  const Link<double> W = load_link64(U, g.V, MU, DAG ? qoff + (j >> 1) : self);
  const HalfSpinor<double> h = project(MU, DAG ? +1 : -1, load_spinor_cvc<V4>(in, j));
  const HalfSpinor<double> u = DAG ? link_dag_mul(W, h) : link_mul(W, h);
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int c = 0; c < 3; ++c) sh[3 * b + c][lane] = make_double2(u.c[b][c].re, u.c[b][c].im);
}

// one colour of accum_recon: acc[spin] += (1 + S g_mu)-reconstruction of (u0, u1)
template <int MU, int S>
__device__ __forceinline__ void cvc_recon(Cx<double> (&acc)[4], double2 a, double2 b) {
  const Cx<double> u0 = cx(a.x, a.y), u1 = cx(b.x, b.y);
  acc[0] = acc[0] + u0;
  acc[1] = acc[1] + u1;
  if (MU == 0) {
    acc[2] = acc[2] + sgn(-S, u0);
    acc[3] = acc[3] + sgn(-S, u1);
  } else if (MU == 1) {
    acc[2] = acc[2] + sgn(S, mul_i(u1));
    acc[3] = acc[3] + sgn(S, mul_i(u0));
  } else if (MU == 2) {
    acc[2] = acc[2] + sgn(S, u1);
    acc[3] = acc[3] + sgn(-S, u0);
  } else {
    acc[2] = acc[2] + sgn(S, mul_i(u0));
    acc[3] = acc[3] + sgn(-S, mul_i(u1));
  }
}

template <bool G5OUT, bool V4>
__global__ void __launch_bounds__(kCvcSplitThreads)
    k_tm_full_cvc_split(double2 *__restrict__ out, const double2 *__restrict__ in,
                        const double2 *__restrict__ U, Geom g, double a, double b, double c) {
  __shared__ double2 sh[8][6][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lex = blockIdx.x * 32 + lane;
  const bool valid = lex < g.V;
  double2 f[4];  // the site's own spinor, one colour
  if (valid && warp < 3)
#pragma unroll
    for (int sp = 0; sp < 4; ++sp) f[sp] = __ldg(in + (size_t)lex * 12 + 3 * sp + warp);
  if (valid) {
    SiteCoord cd;
    const unsigned r0 = fdiv((unsigned)lex, g.dLZ), r1 = fdiv(r0, g.dLY), r2 = fdiv(r1, g.dLX);
    cd.lex = lex;
    cd.z = lex - (int)r0 * g.LZ;
    cd.y = (int)(r0 - r1 * g.LY);
    cd.x = (int)(r1 - r2 * g.LX);
    cd.t = (int)r2;
    const int par = (cd.t + cd.x + cd.y + cd.z) & 1;
    const int self = par * g.Vh + (lex >> 1), qoff = (1 - par) * g.Vh;
    switch (warp) {
      case 0: cvc_split_dir<0, true, V4>(sh[0], in, U, g, cd, self, qoff, lane); break;
      case 1: cvc_split_dir<0, false, V4>(sh[1], in, U, g, cd, self, qoff, lane); break;
      case 2: cvc_split_dir<1, true, V4>(sh[2], in, U, g, cd, self, qoff, lane); break;
      case 3: cvc_split_dir<1, false, V4>(sh[3], in, U, g, cd, self, qoff, lane); break;
      case 4: cvc_split_dir<2, true, V4>(sh[4], in, U, g, cd, self, qoff, lane); break;
      case 5: cvc_split_dir<2, false, V4>(sh[5], in, U, g, cd, self, qoff, lane); break;
      case 6: cvc_split_dir<3, true, V4>(sh[6], in, U, g, cd, self, qoff, lane); break;
      default: cvc_split_dir<3, false, V4>(sh[7], in, U, g, cd, self, qoff, lane); break;
    }
  }
  __syncthreads();
  if (!valid || warp >= 3) return;
  Cx<double> acc[4];
#pragma unroll
  for (int sp = 0; sp < 4; ++sp) acc[sp] = cx(0.0, 0.0);
  cvc_recon<0, +1>(acc, sh[0][warp][lane], sh[0][3 + warp][lane]);
  cvc_recon<0, -1>(acc, sh[1][warp][lane], sh[1][3 + warp][lane]);
  cvc_recon<1, +1>(acc, sh[2][warp][lane], sh[2][3 + warp][lane]);
  cvc_recon<1, -1>(acc, sh[3][warp][lane], sh[3][3 + warp][lane]);
  cvc_recon<2, +1>(acc, sh[4][warp][lane], sh[4][3 + warp][lane]);
  cvc_recon<2, -1>(acc, sh[5][warp][lane], sh[5][3 + warp][lane]);
  cvc_recon<3, +1>(acc, sh[6][warp][lane], sh[6][3 + warp][lane]);
  cvc_recon<3, -1>(acc, sh[7][warp][lane], sh[7][3 + warp][lane]);
#pragma unroll
  for (int sp = 0; sp < 4; ++sp) {
    const double bs = sp < 2 ? b : -b;  // i b g5
    double2 o;
    o.x = fma(c, acc[sp].re, fma(a, f[sp].x, -bs * f[sp].y));
    o.y = fma(c, acc[sp].im, fma(a, f[sp].y, bs * f[sp].x));
    if (G5OUT && sp >= 2) o = make_double2(-o.x, -o.y);
    out[(size_t)lex * 12 + 3 * sp + warp] = o;
  }
}

int launch_tm_full_cvc(cvcb_lattice *L, double *out, const double *in, double a, double b, double c,
                       bool g5out) {
  const Geom &g = L->g;
  const int blocks = (g.V + kCvcThreads - 1) / kCvcThreads;
  double2 *o = reinterpret_cast<double2 *>(out);
  const double2 *i = reinterpret_cast<const double2 *>(in);
  const bool v4 = ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(in)) & 31) == 0;
  if (g.V <= kCvcSplitSites) {
    auto kern = g5out ? (v4 ? k_tm_full_cvc_split<true, true> : k_tm_full_cvc_split<true, false>)
                      : (v4 ? k_tm_full_cvc_split<false, true> : k_tm_full_cvc_split<false, false>);
    kern<<<(g.V + 31) / 32, kCvcSplitThreads, 0, L->stream>>>(o, i, L->U64, g, a, b, c);
  } else {
    auto kern = g5out ? (v4 ? k_tm_full_cvc<true, true> : k_tm_full_cvc<true, false>)
                      : (v4 ? k_tm_full_cvc<false, true> : k_tm_full_cvc<false, false>);
    CVCB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kCvcSmem));
    kern<<<blocks, kCvcThreads, kCvcSmem, L->stream>>>(o, i, L->U64, g, a, b, c, L->red_counter + kLateFlag);
  }
  CVCB_LAUNCHED(L);
  return CVCB_OK;
}

// An expired wait of the call that has just been synchronised (a lattice has
// one call at a time); the next call starts afresh.
int tm_full_cvc_status(cvcb_lattice *L) {
  unsigned late = 0;
  unsigned *const flag = L->red_counter + kLateFlag;
  CVCB_CUDA(cudaMemcpyAsync(&late, flag, sizeof late, cudaMemcpyDeviceToHost, L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  if (late) {
    CVCB_CUDA(cudaMemsetAsync(flag, 0, sizeof late, L->stream));
    set_error("a copy of the operator's neighbours did not land in time");
    return CVCB_ERR_CUDA;
  }
  return CVCB_OK;
}

// f = g5 f on the first nsites sites (device layout: spins 2,3 are k = 6..11)
__global__ void k_g5(double2 *f, Geom g, int nsites_lex) {
  const int lex = blockIdx.x * blockDim.x + threadIdx.x;
  if (lex >= nsites_lex) return;
  const int j = lex_to_eo(g, lex);
#pragma unroll
  for (int k = 6; k < 12; ++k) {
    double2 v = f[(size_t)k * g.V + j];
    f[(size_t)k * g.V + j] = make_double2(-v.x, -v.y);
  }
}

int launch_g5(cvcb_lattice *L, double2 *f, int nsites) {
  k_g5<<<(nsites + 127) / 128, 128, 0, L->stream>>>(f, L->g, nsites);
  CVCB_LAUNCHED(L);
  return CVCB_OK;
}

// f = (1 - i sign m g5) f / (1 + m^2), m = 2 kappa mu  (Q_phi.c:576-589)
__global__ void k_one_pm_imu_inv(double2 *f, Geom g, int nsites_lex, double cm, double norminv) {
  const int lex = blockIdx.x * blockDim.x + threadIdx.x;
  if (lex >= nsites_lex) return;
  const int j = lex_to_eo(g, lex);
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    const double cc = k < 6 ? cm : -cm;  // cm * g5
    double2 v = f[(size_t)k * g.V + j];
    // v + i cc v
    const double re = v.x + (-cc * v.y);
    const double im = v.y + (cc * v.x);
    f[(size_t)k * g.V + j] = make_double2(re * norminv, im * norminv);
  }
}

int launch_one_pm_imu_inv(cvcb_lattice *L, double2 *f, double sign, int nsites) {
  const double m = 2.0 * L->kappa * L->mu;
  k_one_pm_imu_inv<<<(nsites + 127) / 128, 128, 0, L->stream>>>(f, L->g, nsites, -sign * m,
                                                                  1.0 / (1.0 + m * m));
  CVCB_LAUNCHED(L);
  return CVCB_OK;
}

}  // namespace cvcb
