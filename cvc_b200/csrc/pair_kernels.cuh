// Pair-tiled storage and its kernels for the inner iterations of the batched
// solver, in FP32 and, for FP16 storage, P16 below.
//
// Right-hand sides 2q and 2q+1 ("pair q") are stored interleaved per complex
// spin-colour component, so that 16 bytes hold both right-hand sides of a
// component in the register order of the packed FP32x2 instructions
// (FFMA2/FADD2/FMUL2), and two components of a site are adjacent:
//   float4 P[pair][tile = j / 32][component pair k / 2][j % 32][k % 2]
//   float4 = (re of rhs 2q, re of rhs 2q+1, im of rhs 2q, im of rhs 2q+1)
// One 256-bit load per thread reads components 2m and 2m+1 of its site; a
// warp reads 1 KB contiguous; the 6 component pairs of a site lie at fixed
// offsets (m * 1 KB) from one address, so a neighbour costs one address
// computation and six loads.  Links are tiled by 32 even/odd link indices
// too, with 18 reals (phase multiplied in; nothing to rebuild) or 12 reals
// (rows 0, 1; row 2 rebuilt in registers).
//
// Compared with per-rhs structure-of-arrays storage packed into FP32x2 pairs
// after the loads (k_eo_hop_x2), the stencil needs no register moves to form
// the pairs, projects and reconstructs both right-hand sides with packed
// additions, and applies the site-diagonal epilogue in packed arithmetic.
#pragma once

#include "eo_kernels.cuh"
#include "reduce.cuh"

namespace cvcb {

constexpr int kTile = 32;

__device__ __forceinline__ CP cp_of(float4 v) {
  CP c;
  c.re = make_float2(v.x, v.y);
  c.im = make_float2(v.z, v.w);
  return c;
}
__device__ __forceinline__ float4 f4_of(const CP &c) {
  return make_float4(c.re.x, c.re.y, c.im.x, c.im.y);
}

// 256-bit global accesses (sm_100): two float4 from 32-byte-aligned
// addresses in one instruction.  The asm statements are volatile with a
// memory clobber so that the compiler keeps them in order with the other
// memory accesses of the thread (a field is often read and then written by
// the same thread).
__device__ __forceinline__ void ldg_v8(const float4 *q, float4 &a, float4 &b) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z),
                 "=f"(b.w)
               : "l"(q)
               : "memory");
}
__device__ __forceinline__ void stg_v8(float4 *q, const float4 &a, const float4 &b) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(q), "f"(a.x),
               "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}

// FP32 pair-tiled field set: pair pr, half-lattice site j.  Within a tile of
// 32 sites, component k of the site in position l sits at float4
// comp(k) + 2 l = (k / 2) * 64 + k % 2 + 2 l: components 2m and 2m + 1 of a
// site are 32 contiguous bytes, read or written with one 256-bit access
// (a warp: 1 KB contiguous), six per site and rhs pair.
struct P32 {
  using R = float;
  static constexpr bool kScaled = false;  // no scale per site
  float4 *p;
  size_t pstride;  // float4 per pair (tiles x 12 x 32)
  __device__ __forceinline__ static constexpr int comp(int k) { return (k >> 1) * (2 * kTile) + (k & 1); }
  // the site's slot: component k at at(pr, j) + comp(k)
  __device__ __forceinline__ float4 *at(int pr, int j) const {
    return p + (size_t)pr * pstride + (size_t)(j >> 5) * (12 * kTile) + 2 * (j & (kTile - 1));
  }
  __device__ __forceinline__ SpinorPair load_pair(int pr, int j) const {
    const float4 *q = at(pr, j);
    SpinorPair s;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      float4 a, b;
      ldg_v8(q + m * 2 * kTile, a, b);
      s.c[(2 * m) / 3][(2 * m) % 3] = cp_of(a);
      s.c[(2 * m + 1) / 3][(2 * m + 1) % 3] = cp_of(b);
    }
    return s;
  }
  __device__ __forceinline__ SpinorPair load_pair_raw(int pr, int j, float2 &) const {
    return load_pair(pr, j);
  }
  __device__ __forceinline__ void store_pair(int pr, int j, const SpinorPair &s) const {
    float4 *q = at(pr, j);
#pragma unroll
    for (int m = 0; m < 6; ++m)
      stg_v8(q + m * 2 * kTile, f4_of(s.c[(2 * m) / 3][(2 * m) % 3]),
             f4_of(s.c[(2 * m + 1) / 3][(2 * m + 1) % 3]));
  }
  // one lane of a pair (lane 0: rhs 2 pr, lane 1: rhs 2 pr + 1); the other
  // lane's values are left as they are
  __device__ __forceinline__ void store_lane(int pr, int lane, int j, const SpinorPair &s) const {
    float *q = reinterpret_cast<float *>(at(pr, j)) + lane;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const CP &c = s.c[k / 3][k % 3];
      q[4 * comp(k)] = lane ? c.re.y : c.re.x;
      q[4 * comp(k) + 2] = lane ? c.im.y : c.im.x;
    }
  }
  // per-rhs access (for the kernels that run once per reliable update)
  __device__ __forceinline__ Spinor<float> load(int r, int j) const {
    const float4 *q = at(r >> 1, j);
    const bool b = r & 1;
    Spinor<float> s;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      float4 v[2];
      ldg_v8(q + m * 2 * kTile, v[0], v[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        s.c[(2 * m + h) / 3][(2 * m + h) % 3] = cx(b ? v[h].y : v[h].x, b ? v[h].w : v[h].z);
    }
    return s;
  }
};

inline size_t p32_pair_float4(int Vh) { return (size_t)((Vh + kTile - 1) / kTile) * 12 * kTile; }

// FP16 pair-tiled field set with one float scale per site and right-hand side
// (value = half * scale, |half| <= 1):
//   uint4 P[pair][tile][component quarter q = k / 4][j % 32][k / 2 % 2]
//   uint4 = components 2m, 2m + 1 as halves (re a, re b, im a, im b)
//   float2 scale[pair][tile][j % 32] = (rhs a, rhs b)
// A half2 is one operand pair of the FP32x2 instructions after one
// conversion; a spinor pair is three 256-bit loads and one 64-bit load, half
// the requests and 54 % of the bytes of the FP32 form.
struct P16 {
  using R = float;
  static constexpr bool kScaled = true;
  uint4 *p;
  float2 *scale;
  size_t pstride, sstride;  // uint4 and float2 per pair
  __device__ __forceinline__ uint4 *at(int pr, int j) const {
    return p + (size_t)pr * pstride + (size_t)(j >> 5) * (6 * kTile) + 2 * (j & (kTile - 1));
  }
  __device__ __forceinline__ float2 *scale_at(int pr, int j) const {
    return scale + (size_t)pr * sstride + j;
  }
  __device__ __forceinline__ static void unpack(unsigned w, float2 &f) {
    f = __half22float2(*reinterpret_cast<const __half2 *>(&w));
  }
  // the stored halves as floats, and the scales
  __device__ __forceinline__ SpinorPair load_pair_raw(int pr, int j, float2 &nm) const {
    const uint4 *q = at(pr, j);
    nm = __ldg(scale_at(pr, j));
    SpinorPair s;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      float4 a, b;
      ldg_v8(reinterpret_cast<const float4 *>(q + m * 2 * kTile), a, b);
      const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        CP &c = s.c[(4 * m + k) / 3][(4 * m + k) % 3];
        unpack(__float_as_uint(w[2 * k]), c.re);
        unpack(__float_as_uint(w[2 * k + 1]), c.im);
      }
    }
    return s;
  }
  __device__ __forceinline__ SpinorPair load_pair(int pr, int j) const {
    float2 nm;
    SpinorPair s = load_pair_raw(pr, j, nm);
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      CP &c = s.c[k / 3][k % 3];
      c.re = __fmul2_rn(nm, c.re);
      c.im = __fmul2_rn(nm, c.im);
    }
    return s;
  }
  // the scales of a spinor pair (its largest components) and their inverses
  __device__ __forceinline__ static void scales(const SpinorPair &s, float2 &mx, float2 &inv) {
    mx = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const CP &c = s.c[k / 3][k % 3];
      mx.x = fmaxf(mx.x, fmaxf(fabsf(c.re.x), fabsf(c.im.x)));
      mx.y = fmaxf(mx.y, fmaxf(fabsf(c.re.y), fabsf(c.im.y)));
    }
    // below the smallest normal float a site is stored as zero: 1 / mx would overflow
    if (!(mx.x >= 1.17549435e-38f)) mx.x = 0.f;
    if (!(mx.y >= 1.17549435e-38f)) mx.y = 0.f;
    inv = make_float2(mx.x > 0.f ? 1.f / mx.x : 0.f, mx.y > 0.f ? 1.f / mx.y : 0.f);
  }
  __device__ __forceinline__ static unsigned pack(float2 v, float2 inv) {
    const float2 t = __fmul2_rn(v, inv);
    const __half2 h = __floats2half2_rn(t.x, t.y);
    return *reinterpret_cast<const unsigned *>(&h);
  }
  __device__ __forceinline__ void store_pair(int pr, int j, const SpinorPair &s) const {
    float2 mx, inv;
    scales(s, mx, inv);
    uint4 *q = at(pr, j);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      float w[8];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const CP &c = s.c[(4 * m + k) / 3][(4 * m + k) % 3];
        w[2 * k] = __uint_as_float(pack(c.re, inv));
        w[2 * k + 1] = __uint_as_float(pack(c.im, inv));
      }
      stg_v8(reinterpret_cast<float4 *>(q + m * 2 * kTile), make_float4(w[0], w[1], w[2], w[3]),
             make_float4(w[4], w[5], w[6], w[7]));
    }
    *scale_at(pr, j) = mx;
  }
  __device__ __forceinline__ void store_lane(int pr, int lane, int j, const SpinorPair &s) const {
    float2 mx, inv;
    scales(s, mx, inv);
    __half *q = reinterpret_cast<__half *>(at(pr, j)) + lane;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const CP &c = s.c[k / 3][k % 3];
      __half *d = q + (k / 4) * (2 * kTile * 8) + (k % 4) * 4;
      d[0] = __float2half_rn(lane ? c.re.y * inv.y : c.re.x * inv.x);
      d[2] = __float2half_rn(lane ? c.im.y * inv.y : c.im.x * inv.x);
    }
    reinterpret_cast<float *>(scale_at(pr, j))[lane] = lane ? mx.y : mx.x;
  }
  // per-rhs access (for the kernels that run once per reliable update)
  __device__ __forceinline__ Spinor<float> load(int r, int j) const {
    const SpinorPair f = load_pair(r >> 1, j);
    const bool b = r & 1;
    Spinor<float> s;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const CP &c = f.c[k / 3][k % 3];
      s.c[k / 3][k % 3] = cx(b ? c.re.y : c.re.x, b ? c.im.y : c.im.x);
    }
    return s;
  }
};

// pair-tiled storage
template <class SF>
constexpr bool kPairTiled = std::is_same<SF, P32>::value || std::is_same<SF, P16>::value;

inline size_t tile_count(int Vh) { return (size_t)((Vh + kTile - 1) / kTile); }

// 18-real phased links, tiled: float2 U[idx / 32][mu][9][idx % 32]
struct LT32f {
  using R = float;
  static constexpr bool kPhased = true;
  const float2 *U;
  float2 ph[4];  // unused: the phase is multiplied in
  __device__ __forceinline__ Link<float> load(int mu, int idx) const {
    const float2 *q = U + (size_t)(idx >> 5) * (36 * kTile) + mu * 9 * kTile + (idx & (kTile - 1));
    Link<float> L;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const float2 v = __ldg(q + k * kTile);
      L.m[k / 3][k % 3] = cx(v.x, v.y);
    }
    return L;
  }
};

// 12-real phased links (rows 0, 1), tiled: float4 U[idx / 32][mu][3][idx % 32];
// row 2 = e^{3 i theta_mu} conj(row0 x row1) (ph = e^{3 i theta_mu})
struct LT32c {
  using R = float;
  static constexpr bool kPhased = true;
  const float4 *U;
  float2 ph[4];
  __device__ __forceinline__ Link<float> load(int mu, int idx) const {
    const float4 *q = U + (size_t)(idx >> 5) * (12 * kTile) + mu * 3 * kTile + (idx & (kTile - 1));
    Link<float> L;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 v = __ldg(q + k * kTile);
      L.m[(2 * k) / 3][(2 * k) % 3] = cx(v.x, v.y);
      L.m[(2 * k + 1) / 3][(2 * k + 1) % 3] = cx(v.z, v.w);
    }
    reconstruct_row2(L);
    apply_row2_phase(L, ph[mu]);
    return L;
  }
};

// h = (1 + s g_mu) f projected to spins 0, 1, both rhs (table in
// spinor_ops.cuh); with g5 on the input the sign of the lower spins flips
template <int MU, int S>
__device__ __forceinline__ HalfPair project_pair(const SpinorPair &f) {
  HalfPair h;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const CP &f0 = f.c[0][c], &f1 = f.c[1][c], &f2 = f.c[2][c], &f3 = f.c[3][c];
    if (MU == 0) {  // h0 = f0 - s f2, h1 = f1 - s f3
      h.c[0][c].re = S > 0 ? sub2(f0.re, f2.re) : add2(f0.re, f2.re);
      h.c[0][c].im = S > 0 ? sub2(f0.im, f2.im) : add2(f0.im, f2.im);
      h.c[1][c].re = S > 0 ? sub2(f1.re, f3.re) : add2(f1.re, f3.re);
      h.c[1][c].im = S > 0 ? sub2(f1.im, f3.im) : add2(f1.im, f3.im);
    } else if (MU == 1) {  // h0 = f0 - s i f3, h1 = f1 - s i f2; i z = (-z.im, z.re)
      h.c[0][c].re = S > 0 ? add2(f0.re, f3.im) : sub2(f0.re, f3.im);
      h.c[0][c].im = S > 0 ? sub2(f0.im, f3.re) : add2(f0.im, f3.re);
      h.c[1][c].re = S > 0 ? add2(f1.re, f2.im) : sub2(f1.re, f2.im);
      h.c[1][c].im = S > 0 ? sub2(f1.im, f2.re) : add2(f1.im, f2.re);
    } else if (MU == 2) {  // h0 = f0 - s f3, h1 = f1 + s f2
      h.c[0][c].re = S > 0 ? sub2(f0.re, f3.re) : add2(f0.re, f3.re);
      h.c[0][c].im = S > 0 ? sub2(f0.im, f3.im) : add2(f0.im, f3.im);
      h.c[1][c].re = S > 0 ? add2(f1.re, f2.re) : sub2(f1.re, f2.re);
      h.c[1][c].im = S > 0 ? add2(f1.im, f2.im) : sub2(f1.im, f2.im);
    } else {  // h0 = f0 - s i f2, h1 = f1 + s i f3
      h.c[0][c].re = S > 0 ? add2(f0.re, f2.im) : sub2(f0.re, f2.im);
      h.c[0][c].im = S > 0 ? sub2(f0.im, f2.re) : add2(f0.im, f2.re);
      h.c[1][c].re = S > 0 ? sub2(f1.re, f3.im) : add2(f1.re, f3.im);
      h.c[1][c].im = S > 0 ? add2(f1.im, f3.re) : sub2(f1.im, f3.re);
    }
  }
  return h;
}

// out = (a_s + i b_s) v per spin s (site-diagonal, per-spin coefficients)
__device__ __forceinline__ void diag_pair(SpinorPair &o, const SpinorPair &v, const float (&a)[4],
                                          const float (&b)[4], bool accumulate) {
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const CP &x = v.c[s][c];
      float2 re = accumulate ? __ffma2_rn(bc(a[s]), x.re, o.c[s][c].re) : __fmul2_rn(bc(a[s]), x.re);
      float2 im = accumulate ? __ffma2_rn(bc(a[s]), x.im, o.c[s][c].im) : __fmul2_rn(bc(a[s]), x.im);
      re = __ffma2_rn(bc(-b[s]), x.im, re);
      im = __ffma2_rn(bc(b[s]), x.re, im);
      o.c[s][c].re = re;
      o.c[s][c].im = im;
    }
}

// |v|^2 of one site for both right-hand sides, in FP64: the components of a
// colour in the order of their spins, then the colours 0, 1, 2.  Both sweeps
// below sum in this order, and take one partial per 32-site tile, so that alpha
// and beta do not depend on which of them the tuner took.
__device__ __forceinline__ void add_norm2(double2 &n, const CP &z) {
  n.x = fma((double)z.re.x, (double)z.re.x, n.x);
  n.x = fma((double)z.im.x, (double)z.im.x, n.x);
  n.y = fma((double)z.re.y, (double)z.re.y, n.y);
  n.y = fma((double)z.im.y, (double)z.im.y, n.y);
}
__device__ __forceinline__ double2 norm2_pair(const SpinorPair &v) {
  double2 n = make_double2(0.0, 0.0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double2 t = make_double2(0.0, 0.0);
#pragma unroll
    for (int s = 0; s < 4; ++s) add_norm2(t, v.c[s][c]);
    n = make_double2(n.x + t.x, n.y + t.y);
  }
  return n;
}

template <class PF>
__device__ __forceinline__ void store_active(const PF &f, int pr, int j, const SpinorPair &v,
                                             bool act_a, bool act_b) {
  if (act_a && act_b)
    f.store_pair(pr, j, v);
  else
    f.store_lane(pr, act_a ? 0 : 1, j, v);
}

// the scales of FP16 storage, on the projected half spinors (half the values)
template <class PF>
__device__ __forceinline__ void scale_half(HalfPair &h, float2 nm) {
  if (PF::kScaled) {
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        h.c[b][c].re = __fmul2_rn(nm, h.c[b][c].re);
        h.c[b][c].im = __fmul2_rn(nm, h.c[b][c].im);
      }
  }
}

template <int MU, class PF, class LF>
__device__ __forceinline__ void hop_pair_dir(SpinorPair &acc, const HopArgs<PF, LF> &A,
                                             const SiteCoord &cd, int pr, int self, int qoff,
                                             bool g5in) {
  const Geom &g = A.eg.g;
  float2 nm;
  {  // backward: (1 + g_mu) U_mu(x-mu)^+ in(x-mu)
    const int j = nb_lex(g, cd, MU, -1) >> 1;
    const Link<float> W = A.links.load(MU, qoff + j);
    const SpinorPair f = A.in.load_pair_raw(pr, j, nm);
    HalfPair h = g5in ? project_pair<MU, -1>(f) : project_pair<MU, +1>(f);
    scale_half<PF>(h, nm);
    accum_recon_pair(MU, +1, acc, link_mul_pair<true>(W, h));
  }
  {  // forward: (1 - g_mu) U_mu(x) in(x+mu)
    const int j = nb_lex(g, cd, MU, +1) >> 1;
    const Link<float> W = A.links.load(MU, self);
    const SpinorPair f = A.in.load_pair_raw(pr, j, nm);
    HalfPair h = g5in ? project_pair<MU, +1>(f) : project_pair<MU, -1>(f);
    scale_half<PF>(h, nm);
    accum_recon_pair(MU, -1, acc, link_mul_pair<false>(W, h));
  }
}

// The even/odd stencil sweep (same operator as k_eo_hop) on pair-tiled
// fields: thread = (site, rhs pair).  Directions in the order z, y, x, t (the
// z and y neighbours of a block's sites are in L1 after z-).  A pair with one
// inactive right-hand side computes both and stores only the active one;
// with dot_part, per-warp partials of |out|^2 per rhs (as k_eo_hop_x2).
// RUPD: the sweep that produces A p of a CG iteration updates the residual
// instead, r -= alpha A p, and its partials are those of |r|^2; A p itself
// is not stored (CG needs it for nothing else).
template <class PF, class LF, bool G5IN, bool G5HOP, bool AUX, bool RUPD = false>
__global__ void __launch_bounds__(kHopMaxThreads, 2) k_eo_hop_pt(HopArgs<PF, LF> A) {
  const int pr = blockIdx.x * blockDim.y + threadIdx.y;
  const int ra = 2 * pr;
  if (ra >= A.nrhs) return;
  const bool act_a = !(A.done && A.done[ra]);
  const bool has_b = ra + 1 < A.nrhs;
  const bool act_b = has_b && !(A.done && A.done[ra + 1]);
  if (!act_a && !act_b) return;
  const Geom &g = A.eg.g;
  const int p = A.eg.p;
  const int qoff = (1 - p) * g.Vh;
  // epilogue coefficients per spin: out = D1 (c [g5] hop) + D2 aux with
  // D = alpha + i beta g5; c and the optional g5 folded into D1
  float a1[4], b1[4], a2[4], b2[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const float g5 = s < 2 ? 1.f : -1.f;
    const float gh = G5HOP ? g5 : 1.f;
    a1[s] = (float)(A.c * A.d1a) * gh;
    b1[s] = (float)(A.c * A.d1b) * g5 * gh;
    a2[s] = (float)A.d2a;
    b2[s] = (float)A.d2b * g5;
  }
  for (int sb = blockIdx.y; sb * (int)blockDim.x < g.Vh; sb += gridDim.y) {
    const int i = sb * blockDim.x + threadIdx.x;
    double2 n2 = make_double2(0.0, 0.0);  // |out|^2 (or |r|^2) of this site, rhs a and b
    if (i < g.Vh) {
      const SiteCoord cd = site_coord(g, p, i);
      const int self = p * g.Vh + i;
      SpinorPair acc;
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int c = 0; c < 3; ++c) acc.c[s][c].re = acc.c[s][c].im = make_float2(0.f, 0.f);
      hop_pair_dir<3>(acc, A, cd, pr, self, qoff, G5IN);
      hop_pair_dir<2>(acc, A, cd, pr, self, qoff, G5IN);
      hop_pair_dir<1>(acc, A, cd, pr, self, qoff, G5IN);
      hop_pair_dir<0>(acc, A, cd, pr, self, qoff, G5IN);
      SpinorPair o;
      diag_pair(o, acc, a1, b1, false);
      if (AUX) diag_pair(o, A.aux.load_pair(pr, i), a2, b2, true);
      if (RUPD) {
        const float2 na = make_float2(-(float)A.alpha[ra], has_b ? -(float)A.alpha[ra + 1] : 0.f);
        SpinorPair rv = A.rup.load_pair(pr, i);
#pragma unroll
        for (int s = 0; s < 4; ++s)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            rv.c[s][c].re = __ffma2_rn(na, o.c[s][c].re, rv.c[s][c].re);
            rv.c[s][c].im = __ffma2_rn(na, o.c[s][c].im, rv.c[s][c].im);
          }
        if (A.dot_part) n2 = norm2_pair(rv);
        store_active(A.rup, pr, i, rv, act_a, act_b);
      } else {
        if (A.dot_part) n2 = norm2_pair(o);
        store_active(A.out, pr, i, o, act_a, act_b);
      }
    }
    if (A.dot_part) {  // the whole warp is here: one row, warp-aligned block width
      double da = n2.x, db = n2.y;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        da += __shfl_down_sync(0xffffffffu, da, o);
        db += __shfl_down_sync(0xffffffffu, db, o);
      }
      if ((threadIdx.x & 31) == 0) {
        const int w = sb * (blockDim.x >> 5) + (threadIdx.x >> 5);
        A.dot_part[(size_t)ra * A.dot_np + w] = da;
        if (has_b) A.dot_part[(size_t)(ra + 1) * A.dot_np + w] = db;
      }
    }
  }
}

// ---- the same sweep with a site's eight directions on eight warps -----------
// One thread per site and pair goes through the directions one after the
// other, eight load latencies in a row, and on a small lattice the GPU has
// nothing else to do meanwhile.  Here block = one 32-site tile of one pair,
// warp d = direction (z-, z+, y-, y+, x-, x+, t-, t+, the order of
// hop_pair_dir): every warp loads one neighbour, leaves its transported half
// spinors in shared memory, and warps 0..2 sum the colours 0..2 over the
// directions and run the epilogue.  The sums run in the order of k_eo_hop_pt:
// the same field values to the last bit.
constexpr int kSplitThreads = 256;

template <int MU, bool DAG, class LF>
__device__ __forceinline__ void split_dir(float4 (*sh)[kTile], const HopArgs<P32, LF> &A,
                                          const SiteCoord &cd, int pr, int self, int qoff,
                                          bool g5in, int lane) {
  const int j = nb_lex(A.eg.g, cd, MU, DAG ? -1 : +1) >> 1;
  const Link<float> W = A.links.load(MU, DAG ? qoff + j : self);
  const SpinorPair f = A.in.load_pair(pr, j);
  constexpr int S = DAG ? +1 : -1;
  const HalfPair h = g5in ? project_pair<MU, -S>(f) : project_pair<MU, S>(f);
  const HalfPair u = link_mul_pair<DAG>(W, h);
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int c = 0; c < 3; ++c) sh[3 * b + c][lane] = f4_of(u.c[b][c]);
}

// a (spin s of one colour) += (1 + S g_mu)-reconstruction of u (spins 0, 1 of
// the colour): accum_recon_pair, one component
template <int MU, int S>
__device__ __forceinline__ void recon_add(CP (&a)[4], const CP (&u)[2]) {
  auto add = [](CP &x, const CP &v, bool plus) {
    x.re = plus ? add2(x.re, v.re) : sub2(x.re, v.re);
    x.im = plus ? add2(x.im, v.im) : sub2(x.im, v.im);
  };
  auto add_i = [](CP &x, const CP &v, bool plus) {  // x += +-i v
    x.re = plus ? sub2(x.re, v.im) : add2(x.re, v.im);
    x.im = plus ? add2(x.im, v.re) : sub2(x.im, v.re);
  };
  add(a[0], u[0], true);
  add(a[1], u[1], true);
  if (MU == 0) {  // r2 = -S u0, r3 = -S u1
    add(a[2], u[0], S < 0);
    add(a[3], u[1], S < 0);
  } else if (MU == 1) {  // r2 = S i u1, r3 = S i u0
    add_i(a[2], u[1], S > 0);
    add_i(a[3], u[0], S > 0);
  } else if (MU == 2) {  // r2 = S u1, r3 = -S u0
    add(a[2], u[1], S > 0);
    add(a[3], u[0], S < 0);
  } else {  // r2 = S i u0, r3 = -S i u1
    add_i(a[2], u[0], S > 0);
    add_i(a[3], u[1], S < 0);
  }
}

// alpha or beta of right-hand side r from the sum t of a sweep's partials
__device__ __forceinline__ void dot_epilogue(const DotFinish &f, int r, double t) {
  if (f.kind == 1) {
    f.pAp[r] = t;
    // M^+ M is positive definite; a non-positive <p, M^+ M p> only comes from
    // rounding at the end of convergence: take no step and let the host's
    // reliable update refresh the residual.
    f.alpha[r] = (t > 0 && isfinite(t)) ? f.rr[r] / t : 0.0;
  } else {
    f.beta[r] = t / f.rr[r];
    f.rr[r] = t;
  }
}

static_assert(kSplitThreads == kRedThreads, "the last block reduces with block_sum");
template <class LF, bool G5IN, bool G5HOP, bool AUX, bool RUPD = false>
__global__ void __launch_bounds__(kSplitThreads) k_eo_hop_sp(const __grid_constant__ HopArgs<P32, LF> A) {
  __shared__ float4 sh[8][6][kTile];
  // |out|^2 per colour and site, for warp 0 to add up in k_eo_hop_pt's order.  On
  // lattices that fill the GPU the sweep takes 4 to 7 % longer than with a sum per
  // colour and warp, at 8^3 x 16 and below no longer; sums per colour in
  // k_eo_hop_pt too cost that one 0.2 % of M^+ M at 24^3 x 48.
  __shared__ double2 sn[3][kTile];
  const int pr = blockIdx.x, ra = 2 * pr;
  const bool act_a = !(A.done && A.done[ra]);
  const bool has_b = ra + 1 < A.nrhs;
  const bool act_b = has_b && !(A.done && A.done[ra + 1]);
  if (!act_a && !act_b) return;
  const Geom &g = A.eg.g;
  const int p = A.eg.p, qoff = (1 - p) * g.Vh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = (g.Vh + kTile - 1) / kTile;
  for (int tile = blockIdx.y; tile < tiles; tile += gridDim.y) {
    const int i = tile * kTile + lane;
    const bool valid = i < g.Vh;
    // the epilogue's own inputs are under way while the directions arrive
    float4 ax[4], rx[4];
    if (valid && warp < 3) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        if (AUX) ax[s] = __ldg(A.aux.at(pr, i) + P32::comp(3 * s + warp));
        if (RUPD) rx[s] = __ldg(A.rup.at(pr, i) + P32::comp(3 * s + warp));
      }
    }
    if (valid) {
      const SiteCoord cd = site_coord(g, p, i);
      const int self = p * g.Vh + i;
      switch (warp) {
        case 0: split_dir<3, true>(sh[0], A, cd, pr, self, qoff, G5IN, lane); break;
        case 1: split_dir<3, false>(sh[1], A, cd, pr, self, qoff, G5IN, lane); break;
        case 2: split_dir<2, true>(sh[2], A, cd, pr, self, qoff, G5IN, lane); break;
        case 3: split_dir<2, false>(sh[3], A, cd, pr, self, qoff, G5IN, lane); break;
        case 4: split_dir<1, true>(sh[4], A, cd, pr, self, qoff, G5IN, lane); break;
        case 5: split_dir<1, false>(sh[5], A, cd, pr, self, qoff, G5IN, lane); break;
        case 6: split_dir<0, true>(sh[6], A, cd, pr, self, qoff, G5IN, lane); break;
        default: split_dir<0, false>(sh[7], A, cd, pr, self, qoff, G5IN, lane); break;
      }
    }
    __syncthreads();
    if (warp < 3) {
      double2 n2 = make_double2(0.0, 0.0);
      if (valid) {
        CP acc[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) acc[s].re = acc[s].im = make_float2(0.f, 0.f);
        auto take = [&](int d, CP (&u)[2]) {
          u[0] = cp_of(sh[d][warp][lane]);
          u[1] = cp_of(sh[d][3 + warp][lane]);
        };
        CP u[2];
        take(0, u), recon_add<3, +1>(acc, u);
        take(1, u), recon_add<3, -1>(acc, u);
        take(2, u), recon_add<2, +1>(acc, u);
        take(3, u), recon_add<2, -1>(acc, u);
        take(4, u), recon_add<1, +1>(acc, u);
        take(5, u), recon_add<1, -1>(acc, u);
        take(6, u), recon_add<0, +1>(acc, u);
        take(7, u), recon_add<0, -1>(acc, u);
        float4 *dst = RUPD ? A.rup.at(pr, i) : A.out.at(pr, i);
        const float2 na = RUPD ? make_float2(-(float)A.alpha[ra], has_b ? -(float)A.alpha[ra + 1] : 0.f)
                               : make_float2(0.f, 0.f);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const float g5 = s < 2 ? 1.f : -1.f, gh = G5HOP ? g5 : 1.f;
          const float a1 = (float)(A.c * A.d1a) * gh, b1 = (float)(A.c * A.d1b) * g5 * gh;
          const float a2 = (float)A.d2a, b2 = (float)A.d2b * g5;
          CP o;  // diag_pair, one component
          o.re = __ffma2_rn(bc(-b1), acc[s].im, __fmul2_rn(bc(a1), acc[s].re));
          o.im = __ffma2_rn(bc(b1), acc[s].re, __fmul2_rn(bc(a1), acc[s].im));
          if (AUX) {
            const CP x = cp_of(ax[s]);
            o.re = __ffma2_rn(bc(-b2), x.im, __ffma2_rn(bc(a2), x.re, o.re));
            o.im = __ffma2_rn(bc(b2), x.re, __ffma2_rn(bc(a2), x.im, o.im));
          }
          if (RUPD) {
            CP rv = cp_of(rx[s]);
            rv.re = __ffma2_rn(na, o.re, rv.re);
            rv.im = __ffma2_rn(na, o.im, rv.im);
            o = rv;
          }
          add_norm2(n2, o);
          float4 *q = dst + P32::comp(3 * s + warp);
          if (act_a && act_b) {
            *q = f4_of(o);
          } else {
            float *f = reinterpret_cast<float *>(q) + (act_a ? 0 : 1);
            f[0] = act_a ? o.re.x : o.re.y;
            f[2] = act_a ? o.im.x : o.im.y;
          }
        }
      }
      if (A.dot_part) sn[warp][lane] = n2;
    }
    __syncthreads();  // also: the next tile overwrites sh
    if (A.dot_part && warp == 0) {
      double da = sn[0][lane].x + sn[1][lane].x + sn[2][lane].x;
      double db = sn[0][lane].y + sn[1][lane].y + sn[2][lane].y;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        da += __shfl_down_sync(0xffffffffu, da, o);
        db += __shfl_down_sync(0xffffffffu, db, o);
      }
      if (lane == 0) {
        A.dot_part[(size_t)ra * A.dot_np + tile] = da;
        if (has_b) A.dot_part[(size_t)(ra + 1) * A.dot_np + tile] = db;
      }
    }
  }
  if (!A.dot_part || !A.fin.kind) return;
  // the pair's last block sums the partials, in k_dot_finish's order
  __shared__ bool last;
  __shared__ double sr[2][kRedThreads / 32];
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(A.fin.counters + pr, 1u) == gridDim.y - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v[2] = {0.0, 0.0};
  for (int k = threadIdx.x; k < A.dot_np; k += kRedThreads) {
    v[0] += __ldcg(A.dot_part + (size_t)ra * A.dot_np + k);
    if (has_b) v[1] += __ldcg(A.dot_part + (size_t)(ra + 1) * A.dot_np + k);
  }
  block_sum<2>(v, sr);
  if (threadIdx.x == 0) {
    A.fin.counters[pr] = 0;
    if (act_a) dot_epilogue(A.fin, ra, v[0]);
    if (act_b) dot_epilogue(A.fin, ra + 1, v[1]);
  }
}

}  // namespace cvcb
