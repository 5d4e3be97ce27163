// Momentum-space Pi_mu_nu(q) from the position-space conn of
// cvc_exact2_xspace.c:577-861 -- the step the reference's momentum-space
// programs take after the path.  With the conserved currents at their link
// midpoints (x + mu/2 for J_mu(x), y + nu/2 at the source) and the contact
// term c_nu (cvc_exact2_xspace.c:697-716,837-855) subtracted,
//   Pi_mu_nu(q) = e^{i q.y} e^{-i q_mu/2} e^{+i q_nu/2} sum_x e^{-i q.x} Pi_mu_nu(x)
//                 - delta_mu_nu c_nu,          q_mu = 2 pi k_mu / L_mu,
// the lattice Ward identity (cvc_exact2_xspace.c:928-1008) becomes exact
// transversality: sum_mu 2 sin(q_mu/2) Pi_mu_nu(q) = 0 for every q.
//
// The Fourier sum is separable.  k_dft_pair transforms two directions at once
// in shared memory (y and z of one (t, x), then t and x of one (y, z)), so
// that the field crosses memory twice instead of four times, each direction
// L = n1 n2 as n2 transforms of length n1, a twiddle, and n1 of length n2 held
// in registers (Cooley and Tukey, Math. Comp. 19 (1965) 297).  Directions with
// a factor above 16 that does not split further, and planes that do not fit
// shared memory, take k_dft_axis: one direction a pass, O(L) per output.
// FP64 throughout.
#include <cmath>
#include <vector>

#include "cvcb_internal.h"

namespace cvcb {
namespace {

// out[a][k][b] = sum_x tw[(k x) mod L] in[a][x][b]
__global__ void k_dft_axis(const double2 *__restrict__ in, double2 *__restrict__ out,
                           const double2 *__restrict__ tw, long long A, int L, long long B) {
  const long long n = A * L * B;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long b = i % B;
    const long long r = i / B;
    const int k = (int)(r % L);
    const long long a = r / L;
    const double2 *src = in + a * L * B + b;
    double re = 0.0, im = 0.0;
    int kx = 0;  // (k x) mod L
    for (int x = 0; x < L; ++x) {
      const double2 w = __ldg(tw + kx), v = __ldg(src + (long long)x * B);
      re = fma(w.x, v.x, re);
      re = fma(-w.y, v.y, re);
      im = fma(w.x, v.y, im);
      im = fma(w.y, v.x, im);
      kx += k;
      if (kx >= L) kx -= L;
    }
    out[i] = make_double2(re, im);
  }
}

struct PhaseArgs {
  int T, LX, LY, LZ;
  // per direction e^{i q y} and e^{i q / 2} over its momenta
  const double2 *e[4], *h[4];
  double contact[8];
  int subtract;
};

__device__ __forceinline__ double2 mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// midpoint phases, source shift and contact subtraction of one entry
__device__ __forceinline__ double2 pi_phase(const PhaseArgs &P, int kt, int kx, int ky, int kz,
                                            int mn, double2 v) {
  const int mu = mn >> 2, nu = mn & 3;
  const double2 hm = __ldg(mu == 0 ? P.h[0] + kt : mu == 1 ? P.h[1] + kx : mu == 2 ? P.h[2] + ky : P.h[3] + kz);
  const double2 hn = __ldg(nu == 0 ? P.h[0] + kt : nu == 1 ? P.h[1] + kx : nu == 2 ? P.h[2] + ky : P.h[3] + kz);
  double2 z = mul(mul(__ldg(P.e[0] + kt), __ldg(P.e[1] + kx)), mul(__ldg(P.e[2] + ky), __ldg(P.e[3] + kz)));
  z = mul(mul(z, v), mul(make_double2(hm.x, -hm.y), hn));
  if (P.subtract && mu == nu) {
    z.x -= P.contact[2 * nu];
    z.y -= P.contact[2 * nu + 1];
  }
  return z;
}

// the same on the whole field f[k][16] (after k_dft_axis passes)
__global__ void k_pi_phases(double2 *__restrict__ f, PhaseArgs P, long long V) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < 16 * V;
       k += (long long)gridDim.x * blockDim.x) {
    long long r = k >> 4;
    const int kz = (int)(r % P.LZ);
    r /= P.LZ;
    const int ky = (int)(r % P.LY);
    r /= P.LY;
    const int kx = (int)(r % P.LX);
    f[k] = pi_phase(P, (int)(r / P.LX), kx, ky, kz, (int)(k & 15), f[k]);
  }
}

// A direction of length L = n1 n2 (n1, n2 <= kMaxRadix)
constexpr int kMaxRadix = 16;
struct Radix {
  int L, n1, n2;
};
// The split with the least n1 + n2 (which also has the least larger factor);
// false if there is none.
bool split_radix(int L, Radix *r) {
  r->L = L;
  r->n1 = 0;
  for (int a = 1; a <= kMaxRadix; ++a)
    if (L % a == 0 && L / a <= kMaxRadix && (!r->n1 || a + L / a < r->n1 + r->n2)) {
      r->n1 = a;
      r->n2 = L / a;
    }
  return r->n1 != 0;
}

// cos and sin of 2 pi j / n for n <= 8, as constants of the unrolled transforms
// (no registers for the roots, and no arithmetic for 0 and +-1)
__host__ __device__ constexpr double root_cos(int n, int j) {
  constexpr double c5[3] = {1.0, 0.30901699437494742410, -0.80901699437494742410};
  constexpr double c7[4] = {1.0, 0.62348980185873353053, -0.22252093395631440429,
                            -0.90096886790241912624};
  constexpr double h = 0.70710678118654752440;
  constexpr double c8[5] = {1.0, h, 0.0, -h, -1.0};
  const int m = j > n - j ? n - j : j;  // cos is even about n / 2
  return n == 5 ? c5[m] : n == 7 ? c7[m] : n == 8 ? c8[m] : n == 4 ? c8[2 * m]
       : n == 2 ? c8[4 * m] : n == 1 ? 1.0
       : (n == 3 ? 2 * m : m) == 0 ? 1.0 : (n == 3 ? 2 * m : m) == 1 ? 0.5
       : (n == 3 ? 2 * m : m) == 2 ? -0.5 : -1.0;  // 3, 6
}
__host__ __device__ constexpr double root_sin(int n, int j) {
  constexpr double s5[3] = {0.0, 0.95105651629515357212, 0.58778525229247312917};
  constexpr double s7[4] = {0.0, 0.78183148246802980871, 0.97492791218182360702,
                            0.43388373911755812048};
  constexpr double h = 0.70710678118654752440, q = 0.86602540378443864676;
  constexpr double s8[5] = {0.0, h, 1.0, h, 0.0};
  const bool up = 2 * j > n;
  const int m = up ? n - j : j;  // odd about n / 2
  const double v = n == 5 ? s5[m] : n == 7 ? s7[m] : n == 8 ? s8[m] : n == 4 ? s8[2 * m]
                 : n <= 2 ? 0.0
                 : (n == 3 ? 2 * m : m) == 0 || (n == 3 ? 2 * m : m) == 3 ? 0.0 : q;
  return up ? -v : v;
}
// (re, im) += e^{-2 pi i j / n} v, all but v known to the compiler
__device__ __forceinline__ void add_root(double &re, double &im, int n, int j, double2 v) {
  const double c = root_cos(n, j), s = -root_sin(n, j);
  if (s == 0.0) {
    re = c == 1.0 ? re + v.x : c == -1.0 ? re - v.x : fma(c, v.x, re);
    im = c == 1.0 ? im + v.y : c == -1.0 ? im - v.y : fma(c, v.y, im);
  } else if (c == 0.0) {
    re = s == 1.0 ? re - v.y : re + v.y;
    im = s == 1.0 ? im + v.x : im - v.x;
  } else {
    re = fma(-s, v.y, fma(c, v.x, re));
    im = fma(s, v.x, fma(c, v.y, im));
  }
}

// n values at p[k * stride] -> their transform, in place; roots[j * step] =
// e^{-2 pi i j / n}; entry k is multiplied by tw[k * m] (tw null: not)
template <int N>
__device__ __forceinline__ void dft_reg(double2 *p, int stride, const double2 *roots, int step,
                                        const double2 *tw, int m) {
  double2 v[N];
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = p[k * stride];
  double2 w[N > 8 ? N : 1];
  if constexpr (N > 8)
#pragma unroll
    for (int k = 0; k < N; ++k) w[k] = roots[k * step];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double re = v[0].x, im = v[0].y;
#pragma unroll
    for (int x = 1; x < N; ++x) {
      if constexpr (N > 8) {
        const double2 c = w[(x * k) % N];
        re = fma(c.x, v[x].x, re);
        re = fma(-c.y, v[x].y, re);
        im = fma(c.x, v[x].y, im);
        im = fma(c.y, v[x].x, im);
      } else {
        add_root(re, im, N, (x * k) % N, v[x]);
      }
    }
    if (tw) {
      const double2 c = tw[k * m];
      const double t = c.x * re - c.y * im;
      im = c.x * im + c.y * re;
      re = t;
    }
    p[k * stride] = make_double2(re, im);
  }
}
template <int MAXR>
__device__ __forceinline__ void dft_any(int n, double2 *p, int stride, const double2 *roots,
                                        int step, const double2 *tw, int m) {
  switch (n) {
    case 1: dft_reg<1>(p, stride, roots, step, tw, m); return;
    case 2: dft_reg<2>(p, stride, roots, step, tw, m); return;
    case 3: dft_reg<3>(p, stride, roots, step, tw, m); return;
    case 4: dft_reg<4>(p, stride, roots, step, tw, m); return;
    case 5: dft_reg<5>(p, stride, roots, step, tw, m); return;
    case 6: dft_reg<6>(p, stride, roots, step, tw, m); return;
    case 7: dft_reg<7>(p, stride, roots, step, tw, m); return;
    case 8: dft_reg<8>(p, stride, roots, step, tw, m); return;
  }
  if constexpr (MAXR > 8) {
    switch (n) {
      case 9: dft_reg<9>(p, stride, roots, step, tw, m); return;
      case 10: dft_reg<10>(p, stride, roots, step, tw, m); return;
      case 11: dft_reg<11>(p, stride, roots, step, tw, m); return;
      case 12: dft_reg<12>(p, stride, roots, step, tw, m); return;
      case 13: dft_reg<13>(p, stride, roots, step, tw, m); return;
      case 14: dft_reg<14>(p, stride, roots, step, tw, m); return;
      case 15: dft_reg<15>(p, stride, roots, step, tw, m); return;
      default: dft_reg<16>(p, stride, roots, step, tw, m); return;
    }
  }
}

// One direction of the block's plane: element (outer, l, inner) at
// (outer * L + l) * ni + inner.  l = n2 x1 + x2 on entry; on exit momentum
// k1 + n1 k2 stands at l = n2 k1 + k2.
template <int MAXR>
__device__ __forceinline__ void dft_plane(double2 *sm, const double2 *tw, Radix r, int no, int ni) {
  const int lines = no * ni;
  for (int q = threadIdx.x; q < lines * r.n2; q += blockDim.x) {
    const int inner = q % ni, x2 = (q / ni) % r.n2, o = q / (ni * r.n2);
    dft_any<MAXR>(r.n1, sm + (o * r.L + x2) * ni + inner, r.n2 * ni, tw, r.n2, tw, x2);
  }
  __syncthreads();
  if (r.n2 > 1) {
    for (int q = threadIdx.x; q < lines * r.n1; q += blockDim.x) {
      const int inner = q % ni, k1 = (q / ni) % r.n1, o = q / (ni * r.n1);
      dft_any<MAXR>(r.n2, sm + (o * r.L + r.n2 * k1) * ni + inner, ni, tw, r.n1, nullptr, 0);
    }
    __syncthreads();
  }
}

// Two directions (a, b) of every plane.  Element (i, j) of plane o, entry c:
// (i Lb + j) es + o os + c; a block takes one plane o and nc of its 16 entries,
// consecutive blocks the entries of one plane (they share its cache lines:
// DRAM reads of the second launch 336 -> 170 MB).  phases: midpoint phases on
// the way out (the planes are then (t, x) and o = (y, z)).  MAXR: largest
// factor held in registers; up to 8, which covers 2, 4, ... 16, 20, 24, 28, 30,
// 32, 36, 40, 42, 48, 56, 64, the roots are constants and three blocks fit an
// SM (larger ones keep them in registers, 236 in all).
// Moves 0.68 GB at 24^3 x 48 in the two launches, 0.10 ms at 6.55 TB/s;
// measured 0.13 and 0.22 ms (0.37 ms for the call), issue-bound on index
// arithmetic and FP64; 2.85 ms with four k_dft_axis passes, a phase pass and
// two copies.  With two blocks per SM 0.41 ms, with four 0.41 (spills).
constexpr int kDftThreads = 256;
constexpr size_t kDftSmem = 220 * 1024;
struct DftPair {
  const double2 *in, *ta, *tb;  // roots of both directions
  double2 *out;
  Radix a, b;
  long long es, os;
  int lnc, phases;  // nc = 1 << lnc
};
template <int MAXR>
__global__ void __launch_bounds__(kDftThreads, MAXR > 8 ? 1 : 3)
    k_dft_pair(const __grid_constant__ DftPair D, const __grid_constant__ PhaseArgs P) {
  extern __shared__ double2 sm[];
  const int La = D.a.L, Lb = D.b.L, nc = 1 << D.lnc, n = La * Lb * nc;
  double2 *ta = sm + n, *tb = ta + La;
  const int plane = blockIdx.x / (16 >> D.lnc), c0 = blockIdx.x % (16 >> D.lnc) * nc;
  const long long base = plane * D.os + c0;
  for (int q = threadIdx.x; q < La + Lb; q += kDftThreads) ta[q] = q < La ? D.ta[q] : D.tb[q - La];
#pragma unroll 4
  for (int q = threadIdx.x; q < n; q += kDftThreads)
    sm[q] = __ldg(D.in + base + (q >> D.lnc) * D.es + (q & (nc - 1)));
  __syncthreads();
  dft_plane<MAXR>(sm, tb, D.b, La, nc);
  dft_plane<MAXR>(sm, ta, D.a, 1, Lb * nc);
  for (int q = threadIdx.x; q < n; q += kDftThreads) {
    const int c = q & (nc - 1), ka = (q >> D.lnc) / Lb, kb = (q >> D.lnc) - ka * Lb;
    // where momentum k = k1 + n1 k2 of each direction stands
    const int a2 = ka / D.a.n1, b2 = kb / D.b.n1;
    const int sa = D.a.n2 * (ka - a2 * D.a.n1) + a2, sb = D.b.n2 * (kb - b2 * D.b.n1) + b2;
    double2 v = sm[((sa * Lb + sb) << D.lnc) + c];
    if (D.phases)
      v = pi_phase(P, ka, kb, plane / P.LZ, plane % P.LZ, c0 + c, v);
    D.out[base + (q >> D.lnc) * D.es + c] = v;
  }
}

// log2 of the entries per block: the most (up to 8 entries) that leave room for two
// blocks on an SM, at least two (32-byte sectors); 0 if not even two fit one
// block.
int dft_entries(int La, int Lb) {
  auto bytes = [&](int l) { return (((size_t)La * Lb << l) + La + Lb) * sizeof(double2); };
  for (int l = 3; l >= 1; --l)
    if (bytes(l) <= kDftSmem / 2) return l;
  return bytes(1) <= kDftSmem ? 1 : 0;
}

int launch_dft_pair(cvcb_lattice *L, const DftPair &D, const PhaseArgs &P, long long planes) {
  auto kern = std::max(std::max(D.a.n1, D.a.n2), std::max(D.b.n1, D.b.n2)) <= 8 ? k_dft_pair<8>
                                                                               : k_dft_pair<kMaxRadix>;
  CVCB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDftSmem));
  kern<<<(unsigned)(planes * (16 >> D.lnc)), kDftThreads,
         (((size_t)D.a.L * D.b.L << D.lnc) + D.a.L + D.b.L) * sizeof(double2), L->stream>>>(D, P);
  CVCB_LAUNCHED(L);
  return CVCB_OK;
}

}  // namespace
}  // namespace cvcb

using namespace cvcb;

extern "C" int cvcb_pi_momentum(cvcb_lattice *L, const double *conn, int source_site,
                                const double *contact, double *pimom) {
  if (!L || !conn || !pimom) return CVCB_ERR_NULL;
  const Geom &g = L->g;
  if (source_site < 0 || source_site >= g.V) {
    set_error("source site %d outside the lattice", source_site);
    return CVCB_ERR_ARG;
  }
  CVCB_CUDA(cudaSetDevice(L->device));
  const size_t bytes = (size_t)g.V * 16 * sizeof(double2);
  void *a, *b, *t;
  CVCB_TRY(ensure_buffer(L, SLOT_F0, bytes, &a));
  CVCB_TRY(ensure_buffer(L, SLOT_F1, bytes, &b));
  const int ext[4] = {g.T, g.LX, g.LY, g.LZ};
  const int off[4] = {0, g.T, g.T + g.LX, g.T + g.LX + g.LY}, ntw = off[3] + g.LZ;
  CVCB_TRY(ensure_buffer(L, SLOT_F2, (size_t)3 * ntw * sizeof(double2), &t));
  double2 *buf[2] = {static_cast<double2 *>(a), static_cast<double2 *>(b)};
  double2 *tw = static_cast<double2 *>(t);
  // arrays of this device on 16-byte boundaries are read and written in place
  auto here = [&](const double *p) {
    return is_own_device_ptr(L, p) && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
  };
  const double2 *cur = reinterpret_cast<const double2 *>(conn);
  if (!here(conn)) {
    CVCB_CUDA(cudaMemcpyAsync(buf[0], conn, bytes, cudaMemcpyDefault, L->stream));
    cur = buf[0];
  }
  const bool direct = here(pimom);
  // per direction and FP64 on the host: the roots e^{-2 pi i j / L}, the
  // source shifts e^{i q y} (angle reduced exactly) and e^{i q / 2}
  PhaseArgs P{};
  P.T = g.T;
  P.LX = g.LX;
  P.LY = g.LY;
  P.LZ = g.LZ;
  const int y[4] = {source_site / g.s3, source_site / g.s2 % g.LX, source_site / g.s1 % g.LY,
                    source_site % g.LZ};
  std::vector<double2> htw((size_t)3 * ntw);
  for (int d = 0; d < 4; ++d) {
    for (int j = 0; j < ext[d]; ++j) {
      const double ph = -2.0 * M_PI * j / ext[d];
      const double sh = 2.0 * M_PI * (double)((long long)j * y[d] % ext[d]) / ext[d];
      htw[off[d] + j] = make_double2(std::cos(ph), std::sin(ph));
      htw[ntw + off[d] + j] = make_double2(std::cos(sh), std::sin(sh));
      htw[2 * ntw + off[d] + j] = make_double2(std::cos(M_PI * j / ext[d]), std::sin(M_PI * j / ext[d]));
    }
    P.e[d] = tw + ntw + off[d];
    P.h[d] = tw + 2 * ntw + off[d];
  }
  CVCB_CUDA(cudaMemcpyAsync(tw, htw.data(), htw.size() * sizeof(double2), cudaMemcpyHostToDevice,
                            L->stream));
  P.subtract = contact != nullptr;
  if (contact)
    for (int i = 0; i < 8; ++i) P.contact[i] = contact[i];
  // y and z first, then t and x; `last`: into the caller's array if possible
  bool phased = false;
  for (int first = 2; first >= 0; first -= 2) {
    const int La = ext[first], Lb = ext[first + 1];
    DftPair D;
    D.lnc = dft_entries(La, Lb);
    const bool last = first == 0;
    if (D.lnc && split_radix(La, &D.a) && split_radix(Lb, &D.b)) {
      D.in = cur;
      D.out = last && direct ? reinterpret_cast<double2 *>(pimom) : cur == buf[0] ? buf[1] : buf[0];
      D.ta = tw + off[first];
      D.tb = tw + off[first + 1];
      const long long plane = (long long)La * Lb, planes = g.V / plane;
      D.es = last ? planes * 16 : 16;
      D.os = last ? 16 : plane * 16;
      D.phases = phased = last;
      CVCB_TRY(launch_dft_pair(L, D, P, planes));
      cur = D.out;
      continue;
    }
    for (int d = first; d < first + 2; ++d) {
      long long A = 1, B = 16;
      for (int e = 0; e < d; ++e) A *= ext[e];
      for (int e = d + 1; e < 4; ++e) B *= ext[e];
      const long long n = A * ext[d] * B;
      const int blocks = (int)std::min<long long>((n + 255) / 256, 148LL * 32);
      double2 *out = cur == buf[0] ? buf[1] : buf[0];
      k_dft_axis<<<blocks, 256, 0, L->stream>>>(cur, out, tw + off[d], A, ext[d], B);
      CVCB_LAUNCHED(L);
      cur = out;
    }
  }
  if (!phased) {
    k_pi_phases<<<(int)std::min<long long>((16LL * g.V + 255) / 256, 148LL * 32), 256, 0,
                  L->stream>>>(cur == buf[0] ? buf[0] : buf[1], P, g.V);
    CVCB_LAUNCHED(L);
  }
  if (cur != reinterpret_cast<const double2 *>(pimom))
    CVCB_CUDA(cudaMemcpyAsync(pimom, cur, bytes, cudaMemcpyDefault, L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  return CVCB_OK;
}
