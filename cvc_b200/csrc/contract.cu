// Conserved-vector-current contraction Pi_mu_nu(x) (cvc_exact2_xspace.c:
// 577-861), Ward-identity divergence (:928-1008), the P->gamma gamma
// sequential source (p2gg_xspace.c:525-539) and the plaquette
// (cvc_utils.c:384-436).
//
// Restructuring of the reference's 4608 volume sweeps.  For one source
// index nu and one of the two parts, the reference accumulates
//   sum_{g,ir,ia,ib} k(g,ir) us(ia,ib) [ chi_d(x)^+ g5 (g_mu - 1) U_mu(x) phi_c(x+mu)
//                                       + chi_d(x+mu)^+ g5 (g_mu + 1) U_mu(x)^+ phi_c(x) ]
// with c = (ir,ia), d = (gperm_g(ir), ib), k = +-1 or +-i and us an entry of
// the (phased) source link.  Per part and nu the coefficients are K (x) us
// with K = X_nu -+ g5, X_nu = g_nu g5, which has rank two like the vertex
// (g_nu -+ 1) itself: its rows r and r' = partner of r are proportional.  One
// of the two columns of a bracket belongs to the four shifted source points
// (it depends on nu), the other to the source point itself (it does not).
// k_pi therefore keeps the former local to the site a thread works on and
// lets it meet the latter at the eight neighbours (the complex conjugate of
// the bracket exchanges the roles for the second part):
//   Z_{a,o}  = sum_i conj(Us_nu[o][i]) (f_{a,i}(x) - lam f_{a',i}(x)),  a = 0, 1
//   u_{c,+-} = [half spinor of] (1 -+ g_mu) W g_c(x +- mu)
//   T_{mu nu,+-}(x) = sum_{a,o} <Z_{a,o}, g5 (u_{(a,o),+-} + lam u_{(a',o),+-})>
// with f the 12 columns of the point shifted by nu, g those of the source
// point, and lam = conj(X_nu[a][a']) = +-1 or +-i, and
//   Pi_mu_nu(x) = T_{mu nu,+}(x) - T_{mu nu,-}(x + mu),
// T summed over the two parts (conjugated for the second).  (For the other
// kernels of the path, which want the columns of all nu in the coefficient
// form, k_cvc_z_sites or k_cvc_z builds the 24 columns
// Z_c(x) = sum_{g,ib} conj(k us) chi_{d(g,ir,ib)}(x) of one nu.)
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "cvcb_internal.h"
#include "contract_plan.h"
#include "reduce.cuh"
#include "spinor_ops.cuh"

namespace cvcb {


// Z columns of one nu: thread per site, reads 12 or 24 dn columns, writes 24.
__global__ void __launch_bounds__(128) k_cvc_z(double2 *__restrict__ Z,
                                               const double2 *__restrict__ dn, ZPlan plan,
                                               int V) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const size_t fs = (size_t)12 * V;  // field stride
  for (int col = 0; col < 24; ++col) {
    Cx<double> acc[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) acc[k] = cx(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const ZTerm tm = plan.t[col][q];
      const double2 *f = dn + tm.src * fs;
      const Cx<double> cf = cx(tm.coef.x, tm.coef.y);
#pragma unroll
      for (int k = 0; k < 12; ++k) {
        const double2 v = __ldg(f + (size_t)k * V + s);
        cfma(acc[k], cf, cx(v.x, v.y));
      }
    }
    double2 *z = Z + col * fs;
#pragma unroll
    for (int k = 0; k < 12; ++k) z[(size_t)k * V + s] = make_double2(acc[k].re, acc[k].im);
  }
}

// The same Z columns with each dn column that one nu needs read once per
// site: thread = (site, spinor component k = blockIdx.y).  Its inputs (at
// most 24 columns) are staged in shared memory, because the plan picks them
// at run time, and every output is formed with the same terms in the same
// order as k_cvc_z (the same bits).  k_cvc_z reads 6 inputs per output
// column, 144 field reads per nu, most of them from L2 or DRAM again.
constexpr int kZThreads = 128;
struct ZPlanLocal {
  double2 coef[24][6];
  int field[24];             // dn column (0..59) of local input f
  unsigned char loc[24][6];  // local input of term q of output column col
  int nin;                   // local inputs in use
};

__global__ void __launch_bounds__(kZThreads) k_cvc_z_sites(double2 *__restrict__ Z,
                                                          const double2 *__restrict__ dn,
                                                          ZPlanLocal plan, int V) {
  __shared__ double2 in[24][kZThreads];
  const int s = blockIdx.x * kZThreads + threadIdx.x;
  if (s >= V) return;  // each thread reads only its own slots: no barrier below
  const size_t fs = (size_t)12 * V, off = (size_t)blockIdx.y * V + s;
  for (int f = 0; f < plan.nin; ++f) in[f][threadIdx.x] = __ldg(dn + plan.field[f] * fs + off);
  for (int col = 0; col < 24; ++col) {
    Cx<double> acc = cx(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const double2 v = in[plan.loc[col][q]][threadIdx.x];
      cfma(acc, cx(plan.coef[col][q].x, plan.coef[col][q].y), cx(v.x, v.y));
    }
    Z[col * fs + off] = make_double2(acc.re, acc.im);
  }
}

// ---- the contraction kernel ------------------------------------------------
// A block takes 8 consecutive lexicographic sites (V is a multiple of 16).
// Per part it stages in shared memory the Z columns of all four nu (2 x 3
// columns each, formed from the 48 shifted columns, every element read once
// and coalesced although the fields are site-major) and the projected and
// transported half spinors u of the 12 columns of the source point for the 8
// neighbours; then each thread (colour of the sink, pair of nu with the same
// spin partners, site, a, sign of the hop) forms its dots.  u is formed once
// for all four nu, and the local columns need neither a copy in another
// layout nor Z columns in memory.
// Bounds at 24^3 x 48: 15.9 GB of compulsory traffic (2.4 ms at 6.55 TB/s) and
// 42.6 k FP64 instructions per site (1.5 ms at 64 per SM and clock).  Measured
// 7.5 ms (the whole contraction 9.2 ms; 44.6 ms with the columns copied to
// component-major order, Z columns in memory and one thread per site; 0.27
// against 2.41 ms at 8^3 x 16): load latency between the barriers at 12 warps
// per SM bounds it (FP64 pipe 22 % busy).  Tried, no faster: all of a part's
// local loads in flight at once and the links kept in registers (9.4 and
// 9.7 ms), and bringing the next block's local columns to L2 (10.1 ms, DRAM
// reads 1.5 times as many).
constexpr int kPiSites = 8;
constexpr int kPiThreads = 192;
constexpr int kPiZ = 4 * 2 * 3 * 12 * kPiSites;  // double2: [nu][a][o][comp][site]
constexpr int kPiU = 3 * 4 * 8 * 6 * kPiSites;   // double2: [ia][ir][dir][spin][colour][site]
constexpr size_t kPiSmem = (kPiZ + kPiU) * sizeof(double2);

struct PiArgs {
  const double2 *loc[2][48];  // part 0: dn, part 1: up columns of the shifted points, site-major
  const double2 *fix;         // [part][12 columns][12][V], lexicographic: columns of the source point
  const double2 *U;
  double2 *F, *B;   // T_+ and T_-, [V][mu][nu]
  double2 us[4][9]; // conj of the phased source links
  double lam[4][2]; // lam = lam (nu = 0, 2) or i lam (nu = 1, 3), per a
  Geom g;
};

// slot of component comp of site s inside one Z column: the sites of a
// component are permuted by it, so that both the writers (consecutive
// components) and the readers (consecutive sites) spread over the banks
__device__ __forceinline__ int z_slot(int comp, int s) { return comp * kPiSites + (s ^ (comp & 7)); }

// u of one column and direction for the thread's site
template <int MU, int S>
__device__ __forceinline__ void pi_transport(const PiArgs &A, const SiteCoord &cd, int par,
                                             const double2 *col, double2 *u) {
  const Geom &g = A.g;
  const int j = nb_lex(g, cd, MU, S < 0 ? +1 : -1);
  Spinor<double> f;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    const double2 v = __ldg(col + (size_t)k * g.V + j);
    f.c[k / 3][k % 3] = cx(v.x, v.y);
  }
  const int at = S < 0 ? par * g.Vh + (cd.lex >> 1) : (1 - par) * g.Vh + (j >> 1);
  const Link<double> W = load_link64(A.U, g.V, MU, at);
  const HalfSpinor<double> h = project(MU, S, f);
  const HalfSpinor<double> r = S < 0 ? link_mul(W, h) : link_dag_mul(W, h);
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      u[(3 * b + c) * kPiSites] = make_double2(r.c[b][c].re, r.c[b][c].im);
}

// acc += conj(z) v
__device__ __forceinline__ void dot_acc(Cx<double> &acc, Cx<double> z, Cx<double> v) {
  cfmac(acc, z, v);
}
// z + s w and z + s i w
__device__ __forceinline__ Cx<double> add_s(Cx<double> z, double s, Cx<double> w) {
  return cx(fma(s, w.re, z.re), fma(s, w.im, z.im));
}
__device__ __forceinline__ Cx<double> add_si(Cx<double> z, double s, Cx<double> w) {
  return cx(fma(-s, w.im, z.re), fma(s, w.re, z.im));
}

__global__ void __launch_bounds__(kPiThreads, 2) k_pi(const __grid_constant__ PiArgs A) {
  extern __shared__ double2 sm[];
  double2 *sz = sm, *su = sm + kPiZ;
  const Geom &g = A.g;
  const int base = blockIdx.x * kPiSites;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int site = lane & 7;
  SiteCoord cd;
  {
    cd.lex = base + site;
    const unsigned r0 = fdiv((unsigned)cd.lex, g.dLZ), r1 = fdiv(r0, g.dLY), r2 = fdiv(r1, g.dLX);
    cd.z = cd.lex - (int)r0 * g.LZ;
    cd.y = (int)(r0 - r1 * g.LY);
    cd.x = (int)(r1 - r2 * g.LX);
    cd.t = (int)r2;
  }
  const int par = (cd.t + cd.x + cd.y + cd.z) & 1;
  // the dots' role of the thread
  const int si = warp % 3, cls = warp / 3;           // colour of the sink; nu in {0,3} or {2,1}
  const int a = (lane >> 3) & 1, sg = lane >> 4;     // source spin; forward or backward hop
  const int ap = cls == 0 ? a + 2 : 3 - a;           // its partner
  const int nur = cls == 0 ? 0 : 2, nui = cls == 0 ? 3 : 1;
  const double lr = A.lam[nur][a], li = A.lam[nui][a];
  const double s = sg ? 1.0 : -1.0;
  Cx<double> acc[2][4];
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) acc[n][mu] = cx(0.0, 0.0);

#pragma unroll 1
  for (int part = 0; part < 2; ++part) {
    // Z: 8 (nu, a) x 96 elements (site, component), six columns in, three out
#pragma unroll 1
    for (int q = warp; q < 24; q += kPiThreads / 32) {
      const int na = q / 3, nu = na >> 1, za = na & 1;
      const int zp = nu == 0 || nu == 3 ? za + 2 : 3 - za;
      const int e = (q % 3) * 32 + lane, es = e / 12, ec = e - 12 * es;
      const size_t off = (size_t)base * 12 + e;
      const double l = A.lam[nu][za];
      Cx<double> y[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double2 v = __ldg(A.loc[part][12 * nu + 3 * za + i] + off);
        const double2 w = __ldg(A.loc[part][12 * nu + 3 * zp + i] + off);
        y[i] = nu & 1 ? add_si(cx(v.x, v.y), -l, cx(w.x, w.y)) : add_s(cx(v.x, v.y), -l, cx(w.x, w.y));
      }
#pragma unroll
      for (int o = 0; o < 3; ++o) {
        Cx<double> z = cx(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < 3; ++i) cfma(z, cx(A.us[nu][3 * o + i].x, A.us[nu][3 * o + i].y), y[i]);
        sz[(na * 3 + o) * 12 * kPiSites + z_slot(ec, es)] = make_double2(z.re, z.im);
      }
    }
    // u: 8 directions x 3 colours, lanes = 8 sites x 4 source spins
#pragma unroll 1
    for (int q = warp; q < 24; q += kPiThreads / 32) {
      const int dir = q / 3, ia = q % 3, ir = lane >> 3;
      const double2 *col = A.fix + (size_t)(part * 12 + 3 * ir + ia) * 12 * g.V;
      double2 *u = su + ((ia * 4 + ir) * 8 + dir) * 6 * kPiSites + site;
      switch (dir) {
        case 0: pi_transport<0, -1>(A, cd, par, col, u); break;
        case 1: pi_transport<1, -1>(A, cd, par, col, u); break;
        case 2: pi_transport<2, -1>(A, cd, par, col, u); break;
        case 3: pi_transport<3, -1>(A, cd, par, col, u); break;
        case 4: pi_transport<0, +1>(A, cd, par, col, u); break;
        case 5: pi_transport<1, +1>(A, cd, par, col, u); break;
        case 6: pi_transport<2, +1>(A, cd, par, col, u); break;
        default: pi_transport<3, +1>(A, cd, par, col, u); break;
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int o = 0; o < 3; ++o) {
      Cx<double> zr[4], zi[4];
#pragma unroll
      for (int sp = 0; sp < 4; ++sp) {
        const int sl = z_slot(3 * sp + si, site);
        const double2 v = sz[((nur * 2 + a) * 3 + o) * 12 * kPiSites + sl];
        const double2 w = sz[((nui * 2 + a) * 3 + o) * 12 * kPiSites + sl];
        zr[sp] = cx(v.x, v.y);
        zi[sp] = cx(w.x, w.y);
      }
#pragma unroll
      for (int mu = 0; mu < 4; ++mu) {
        const int d = sg * 4 + mu;
        const double2 *u1 = su + (((o * 4 + a) * 8 + d) * 6 + si) * kPiSites + site;
        const double2 *u2 = su + (((o * 4 + ap) * 8 + d) * 6 + si) * kPiSites + site;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const double2 p = u1[3 * b * kPiSites], q = u2[3 * b * kPiSites];
          const Cx<double> vr = add_s(cx(p.x, p.y), lr, cx(q.x, q.y));
          const Cx<double> vi = add_si(cx(p.x, p.y), li, cx(q.x, q.y));
          // the conjugate-transposed reconstruction of spins 2, 3 with g5
          const int hi = mu == 0 || mu == 3 ? 2 + b : 3 - b;
          const double sb = (mu >= 2 && b == 1) ? -s : s;
          const bool im = mu & 1;
          dot_acc(acc[0][mu], im ? add_si(zr[b], sb, zr[hi]) : add_s(zr[b], sb, zr[hi]), vr);
          dot_acc(acc[1][mu], im ? add_si(zi[b], sb, zi[hi]) : add_s(zi[b], sb, zi[hi]), vi);
        }
      }
    }
    __syncthreads();
    // the second part enters conjugated: conj(conj(T_0) + T_1)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int mu = 0; mu < 4; ++mu) acc[n][mu].im = -acc[n][mu].im;
  }
  // sum over a (lanes) and the sink's colour (warps), in a fixed order
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
      Cx<double> t = acc[n][mu];
      t.re += __shfl_xor_sync(0xffffffffu, t.re, 8);
      t.im += __shfl_xor_sync(0xffffffffu, t.im, 8);
      if (a == 0)
        sm[((si * 8 + sg * 4 + mu) * 4 + (n ? nui : nur)) * kPiSites + site] = make_double2(t.re, t.im);
    }
  __syncthreads();
  for (int k = threadIdx.x; k < 256; k += kPiThreads) {
    const int ks = (k >> 4) & 7, slot = (((k >> 7) * 4 + ((k >> 2) & 3)) * 4 + (k & 3)) * kPiSites + ks;
    const double2 x = sm[slot], y = sm[slot + 32 * kPiSites], z = sm[slot + 64 * kPiSites];
    double2 *o = (k >> 7) ? A.B : A.F;
    o[(size_t)(base + ks) * 16 + (k & 15)] = make_double2(x.x + y.x + z.x, x.y + y.y + z.y);
  }
}

// conn_mu_nu(x) = -1/4 (T_+(x) - T_-(x + mu))   (normalisation, :861)
__global__ void k_pi_combine(double2 *__restrict__ conn, const double2 *__restrict__ F,
                             const double2 *__restrict__ B, Geom g) {
  const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (k >= (size_t)g.V * 16) return;
  SiteCoord cd;
  cd.lex = (int)(k >> 4);
  const unsigned r0 = fdiv((unsigned)cd.lex, g.dLZ), r1 = fdiv(r0, g.dLY), r2 = fdiv(r1, g.dLX);
  cd.z = cd.lex - (int)r0 * g.LZ;
  cd.y = (int)(r0 - r1 * g.LY);
  cd.x = (int)(r1 - r2 * g.LX);
  cd.t = (int)r2;
  const int m = (int)(k & 15);
  const double2 f = F[k], b = B[(size_t)nb_lex(g, cd, m >> 2, +1) * 16 + m];
  conn[k] = make_double2(-0.25 * (f.x - b.x), -0.25 * (f.y - b.y));
}

// columns of the source point from CVC layout to component-major:
// dst[column][component][V], lexicographic
struct FixCols {
  const double2 *src[24];
};
constexpr int kFixTile = 64;
__global__ void __launch_bounds__(128) k_fix_columns(double2 *__restrict__ dst,
                                                    const __grid_constant__ FixCols c, int V) {
  __shared__ double2 t[kFixTile * 13];
  const int base = blockIdx.x * kFixTile, n = min(kFixTile, V - base);
  const double2 *src = c.src[blockIdx.y] + (size_t)base * 12;
  for (int q = threadIdx.x; q < n * 12; q += blockDim.x) {
    const int s = q / 12;
    t[q + s] = __ldg(src + q);
  }
  __syncthreads();
  double2 *d = dst + (size_t)blockIdx.y * 12 * V + base;
  for (int q = threadIdx.x; q < kFixTile * 12; q += blockDim.x) {
    const int k = q / kFixTile, s = q % kFixTile;
    if (s < n) d[(size_t)k * V + s] = t[s * 13 + k];
  }
}

// the 96 spinors of the contact term (:697-704, :837-844)
struct ContactCols {
  const double *src[60];  // up columns
  int iup[4], site;
};
__global__ void k_contact_gather(double *__restrict__ out, const __grid_constant__ ContactCols c) {
  const int q = blockIdx.x, part = q / 48, nu = (q / 12) % 4, col = q % 12;
  const double *f = part == 0 ? c.src[48 + col] : c.src[nu * 12 + col];
  if (threadIdx.x < 24)
    out[q * 24 + threadIdx.x] = f[24 * (size_t)(part == 0 ? c.iup[nu] : c.site) + threadIdx.x];
}

// Ward identity divergence on the CVC-layout conn (cvc_exact2_xspace.c:938-953)
__global__ void k_cvc_ward(double *__restrict__ wi, const double *__restrict__ conn, Geom g) {
  const int lex = blockIdx.x * blockDim.x + threadIdx.x;
  if (lex >= g.V) return;
  SiteCoord cd;
  cd.z = lex % g.LZ;
  int r = lex / g.LZ;
  cd.y = r % g.LY;
  r /= g.LY;
  cd.x = r % g.LX;
  cd.t = r / g.LX;
  cd.lex = lex;
  int dn[4];
#pragma unroll
  for (int mu = 0; mu < 4; ++mu) dn[mu] = nb_lex(g, cd, mu, -1);
  for (int nu = 0; nu < 4; ++nu)
    for (int ri = 0; ri < 2; ++ri) {
      double w = 0;
#pragma unroll
      for (int mu = 0; mu < 4; ++mu) w += conn[(size_t)lex * 32 + 2 * (4 * mu + nu) + ri];
#pragma unroll
      for (int mu = 0; mu < 4; ++mu) w -= conn[(size_t)dn[mu] * 32 + 2 * (4 * mu + nu) + ri];
      wi[(size_t)lex * 8 + 2 * nu + ri] = w;
    }
}

// Sequential source (p2gg_xspace.c:525-539): on timeslice t,
// source(x) = exp(i phase(x)) Gamma prop(x); elsewhere zero.  Works on the
// CVC layout directly (one thread per site of the whole lattice).
struct GammaTab {
  int perm[24];
  int sign[24];
};
__global__ void k_seq_source(double *__restrict__ src, const double *__restrict__ prop, Geom g,
                             int t0, int m0, int m1, int m2, double sgn2pi, GammaTab gt) {
  const int lex = blockIdx.x * blockDim.x + threadIdx.x;
  if (lex >= g.V) return;
  double *o = src + (size_t)lex * 24;
  const int t = lex / g.s3;
  if (t != t0) {
#pragma unroll
    for (int k = 0; k < 24; ++k) o[k] = 0.0;
    return;
  }
  const int x1 = (lex / g.s2) % g.LX, x2 = (lex / g.s1) % g.LY, x3 = lex % g.LZ;
  // same operation order as the reference: int products, then / (double)L
  const double phase =
      sgn2pi * ((x1 * m0) / (double)g.LX + (x2 * m1) / (double)g.LY + (x3 * m2) / (double)g.LZ);
  double sn, cs;
  sincos(phase, &sn, &cs);
  const double *pp = prop + (size_t)lex * 24;
  double s1[24];
#pragma unroll
  for (int k = 0; k < 24; ++k) s1[k] = pp[gt.perm[k]] * gt.sign[k];
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    const double re = s1[2 * k], im = s1[2 * k + 1];
    o[2 * k] = re * cs - im * sn;
    o[2 * k + 1] = re * sn + im * cs;
  }
}

// Plaquette: sum over sites and mu < nu of Re tr(U_mu(x) U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+)
struct PlaqF {
  const double2 *U;  // raw (unphased) links, device layout, as cvc_utils.c:393-394 uses
  Geom g;
  __device__ void operator()(size_t s, double (&acc)[1]) const {
    const int p = (int)s >= g.Vh;
    const SiteCoord cd = site_coord(g, p, (int)s - p * g.Vh);
    const int qoff = (1 - p) * g.Vh;
    double sum = 0;
    for (int mu = 0; mu < 3; ++mu)
      for (int nu = mu + 1; nu < 4; ++nu) {
        const int jm = qoff + (nb_lex(g, cd, mu, +1) >> 1);
        const int jn = qoff + (nb_lex(g, cd, nu, +1) >> 1);
        const Link<double> A = load_link64(U, g.V, mu, (int)s);
        const Link<double> B = load_link64(U, g.V, nu, jm);
        const Link<double> C = load_link64(U, g.V, nu, (int)s);
        const Link<double> D = load_link64(U, g.V, mu, jn);
        // Re tr[(A B)(C D)^+] = sum_ij Re (AB)_ij conj((CD)_ij)
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j) {
            Cx<double> ab = cx(0.0, 0.0), cdm = cx(0.0, 0.0);
            for (int k = 0; k < 3; ++k) {
              cfma(ab, A.m[i][k], B.m[k][j]);
              cfma(cdm, C.m[i][k], D.m[k][j]);
            }
            sum += ab.re * cdm.re + ab.im * cdm.im;
          }
      }
    acc[0] += sum;
  }
};

// raw links in device layout straight from the host copy (exact, no phase)
__global__ void k_gauge_raw_eo(double2 *__restrict__ out, const double2 *__restrict__ raw, Geom g) {
  const int lex = blockIdx.x * blockDim.x + threadIdx.x;
  if (lex >= g.V) return;
  const int eo = lex_to_eo(g, lex);
  for (int mu = 0; mu < 4; ++mu)
    for (int k = 0; k < 9; ++k)
      out[(size_t)(mu * 9 + k) * g.V + eo] = raw[((size_t)lex * 4 + mu) * 9 + k];
}

struct LinkSumF {
  const double2 *raw;
  __device__ void operator()(size_t k, double (&acc)[2]) const {
    const double2 v = __ldg(raw + k);
    acc[0] += v.x;
    acc[1] += v.y;
  }
};

// phased source links Usource[nu] (cvc_exact2_xspace.c:293-304)
static void source_links(const cvcb_lattice *L, int src, double Us[4][18]) {
  const double *G = L->gauge_host.data();
  for (int nu = 0; nu < 4; ++nu)
    for (int k = 0; k < 9; ++k) {
      const double re = G[18 * (4 * (size_t)src + nu) + 2 * k],
                   im = G[18 * (4 * (size_t)src + nu) + 2 * k + 1];
      const double pr = L->phase[2 * nu], pi = L->phase[2 * nu + 1];
      Us[nu][2 * k] = re * pr - im * pi;
      Us[nu][2 * k + 1] = re * pi + im * pr;
    }
}

// Coefficient plans of the Z columns for the four nu (see the file comment),
// and the phased source links Usource[nu] (cvc_exact2_xspace.c:293-304).
int make_zplans(cvcb_lattice *L, int src, ZPlan plans[4], double Us[4][18], ZMeta *meta) {
  // the reference's gamma bookkeeping (cvc_exact2_xspace.c:336-383)
  int perm[16][24], sign[16][24];
  gamma_tables(perm, sign);
  int gperm[5][4], isimag[4];
  double gsign[5][4];
  for (int ir = 0; ir < 4; ++ir) {
    gperm[4][ir] = perm[5][6 * ir] / 6;
    gsign[4][ir] = sign[5][6 * ir];
  }
  for (int nu = 0; nu < 4; ++nu) {
    for (int ir = 0; ir < 4; ++ir) {
      gperm[nu][ir] = perm[6 + nu][6 * ir] / 6;
      gsign[nu][ir] = sign[6 + nu][6 * ir];
    }
    isimag[nu] = perm[6 + nu][0] % 2;
  }
  source_links(L, src, Us);
  for (int nu = 0; nu < 4; ++nu) {
    ZPlan &plan = plans[nu];
    for (int part = 0; part < 2; ++part)
      for (int ir = 0; ir < 4; ++ir)
        for (int ia = 0; ia < 3; ++ia) {
          const int col = part * 12 + 3 * ir + ia;
          int q = 0;
          for (int gg = 0; gg < 2; ++gg) {
            const int gi = gg == 0 ? nu : 4;
            // k: +-1 or +-i
            double kr, ki;
            if (gg == 0) {
              kr = isimag[nu] ? 0.0 : gsign[nu][ir];
              ki = isimag[nu] ? -gsign[nu][ir] : 0.0;
            } else {
              kr = part == 0 ? -gsign[4][ir] : gsign[4][ir];
              ki = 0.0;
            }
            for (int ib = 0; ib < 3; ++ib) {
              double ur, ui;  // us
              if (part == 0) {
                ur = Us[nu][2 * (3 * ia + ib)];
                ui = Us[nu][2 * (3 * ia + ib) + 1];
              } else {
                ur = Us[nu][2 * (3 * ib + ia)];
                ui = -Us[nu][2 * (3 * ib + ia) + 1];
              }
              const double cr = kr * ur - ki * ui, ci = kr * ui + ki * ur;
              const int d = 3 * gperm[gi][ir] + ib;
              // chi: part 0 -> dn shifted by nu (block nu), part 1 -> dn unshifted (block 4)
              plan.t[col][q].src = (part == 0 ? nu * 12 : 48) + d;
              plan.t[col][q].coef = make_double2(cr, -ci);
              if (meta) {
                ZMeta &m = meta[(nu * 24 + col) * 6 + q];
                m.k = make_double2(kr, ki);
                m.ia = ia;
                m.ib = ib;
                m.part = part;
              }
              ++q;
            }
          }
        }
  }
  return CVCB_OK;
}

// Z columns of one nu into Z (24 fields), from the 60 dn fields at dn:
// k_cvc_z_sites when the plan draws on at most 24 distinct dn columns (one
// nu: the 12 shifted by nu and the 12 unshifted ones), else k_cvc_z.
int launch_cvc_z(cvcb_lattice *L, double2 *Z, const double2 *dn, const ZPlan &plan) {
  ZPlanLocal lp{};
  bool fits = true;
  for (int col = 0; col < 24 && fits; ++col)
    for (int q = 0; q < 6 && fits; ++q) {
      const int src = plan.t[col][q].src;
      int f = 0;
      while (f < lp.nin && lp.field[f] != src) ++f;
      if (f == lp.nin) {
        if (lp.nin == 24) {
          fits = false;
          break;
        }
        lp.field[lp.nin++] = src;
      }
      lp.loc[col][q] = (unsigned char)f;
      lp.coef[col][q] = plan.t[col][q].coef;
    }
  if (fits) {
    dim3 grid((L->g.V + kZThreads - 1) / kZThreads, 12);
    k_cvc_z_sites<<<grid, kZThreads, 0, L->stream>>>(Z, dn, lp, L->g.V);
  } else {
    k_cvc_z<<<(L->g.V + 127) / 128, 128, 0, L->stream>>>(Z, dn, plan, L->g.V);
  }
  CVCB_LAUNCHED(L);
  return CVCB_OK;
}

static int need_gauge(cvcb_lattice *L) {
  if (!L->have_gauge) {
    set_error("no gauge field uploaded");
    return CVCB_ERR_STATE;
  }
  return CVCB_OK;
}

int cvc_contract(cvcb_lattice *L, const double *const *fields, int src, double *conn,
                 double *contact) {
  CVCB_TRY(need_gauge(L));
  const Geom &g = L->g;
  if (src < 0 || src >= g.V) {
    set_error("source site %d outside [0, %d)", src, g.V);
    return CVCB_ERR_ARG;
  }
  int nhost = 0;
  bool on_host[120];
  for (int f = 0; f < 120; ++f) {
    if (!fields[f]) {
      set_error("field %d is NULL", f);
      return CVCB_ERR_NULL;
    }
    on_host[f] = !is_device_ptr(fields[f]);
    nhost += on_host[f];
  }
  const size_t fs = (size_t)12 * g.V;  // double2 per field
  void *fixb, *cb, *hb = nullptr;
  if (nhost) CVCB_TRY(ensure_buffer(L, SLOT_PROPS, nhost * fs * sizeof(double2), &hb));
  CVCB_TRY(ensure_buffer(L, SLOT_F2, 24 * fs * sizeof(double2), &fixb));
  // T_+, T_-, and the contact term's spinors
  const size_t piv = (size_t)g.V * 16;
  CVCB_TRY(ensure_buffer(L, SLOT_CONN, 2 * piv * sizeof(double2) + 96 * 24 * sizeof(double), &cb));
  const double *dev[120];
  for (int f = 0, h = 0; f < 120; ++f) {
    dev[f] = fields[f];
    if (on_host[f]) {
      double2 *d = static_cast<double2 *>(hb) + fs * h++;
      CVCB_CUDA(cudaMemcpyAsync(d, fields[f], fs * sizeof(double2), cudaMemcpyHostToDevice,
                                L->stream));
      dev[f] = reinterpret_cast<const double *>(d);
    }
  }

  // phased source links Usource[nu] (:293-304) and the spin structure of the vertex
  int perm[16][24], sign[16][24];
  gamma_tables(perm, sign);
  double Us[4][18];
  source_links(L, src, Us);
  PiArgs A;
  FixCols fc;
  for (int nu = 0; nu < 4; ++nu) {
    for (int k = 0; k < 9; ++k) A.us[nu][k] = make_double2(Us[nu][2 * k], -Us[nu][2 * k + 1]);
    for (int a = 0; a < 2; ++a) {
      const int ap = nu == 0 || nu == 3 ? a + 2 : 3 - a, *pm = perm[6 + nu] + 6 * a;
      const bool imag = pm[0] % 2;
      if (pm[0] / 6 != ap || imag != (bool)(nu & 1)) {  // the kernel's table of partners
        set_error("unexpected gamma table");
        return CVCB_ERR_STATE;
      }
      // lam = conj(X_nu[a][a']), X = sign (real) or -i sign (imaginary)
      A.lam[nu][a] = sign[6 + nu][6 * a];
    }
  }
  for (int c = 0; c < 48; ++c) {
    A.loc[0][c] = reinterpret_cast<const double2 *>(dev[60 + c]);
    A.loc[1][c] = reinterpret_cast<const double2 *>(dev[c]);
  }
  for (int c = 0; c < 12; ++c) {
    fc.src[c] = reinterpret_cast<const double2 *>(dev[48 + c]);
    fc.src[12 + c] = reinterpret_cast<const double2 *>(dev[108 + c]);
  }
  A.fix = static_cast<const double2 *>(fixb);
  A.U = L->U64;
  A.F = static_cast<double2 *>(cb);
  A.B = A.F + piv;
  A.g = g;
  k_fix_columns<<<dim3((g.V + kFixTile - 1) / kFixTile, 24), 128, 0, L->stream>>>(
      static_cast<double2 *>(fixb), fc, g.V);
  CVCB_LAUNCHED(L);
  CVCB_CUDA(cudaFuncSetAttribute(k_pi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPiSmem));
  k_pi<<<g.V / kPiSites, kPiThreads, kPiSmem, L->stream>>>(A);
  CVCB_LAUNCHED(L);
  // contact term (:697-704, :837-844) from a handful of spinors
  double *ctb = reinterpret_cast<double *>(A.B + piv);
  std::vector<double> sp;
  if (contact) {
    sp.resize(96 * 24);
    ContactCols cc;
    for (int c = 0; c < 60; ++c) cc.src[c] = dev[c];
    const int z = src % g.LZ, y = (src / g.LZ) % g.LY, x = (src / g.s2) % g.LX, t = src / g.s3;
    cc.iup[0] = ((t + 1) % g.T) * g.s3 + x * g.s2 + y * g.s1 + z;
    cc.iup[1] = t * g.s3 + ((x + 1) % g.LX) * g.s2 + y * g.s1 + z;
    cc.iup[2] = t * g.s3 + x * g.s2 + ((y + 1) % g.LY) * g.s1 + z;
    cc.iup[3] = t * g.s3 + x * g.s2 + y * g.s1 + (z + 1) % g.LZ;
    cc.site = src;
    k_contact_gather<<<96, 32, 0, L->stream>>>(ctb, cc);
    CVCB_LAUNCHED(L);
  }
  // Pi in CVC layout straight into the caller's array where that is memory of
  // this device on a 16-byte boundary, else through the (spent) column buffer
  const bool direct = is_own_device_ptr(L, conn) && (reinterpret_cast<uintptr_t>(conn) & 15) == 0;
  double2 *out = direct ? reinterpret_cast<double2 *>(conn) : static_cast<double2 *>(fixb);
  k_pi_combine<<<(int)((piv + 255) / 256), 256, 0, L->stream>>>(out, A.F, A.B, g);
  CVCB_LAUNCHED(L);
  if (!direct)
    CVCB_CUDA(cudaMemcpyAsync(conn, out, piv * sizeof(double2), cudaMemcpyDefault, L->stream));
  if (contact)
    CVCB_CUDA(cudaMemcpyAsync(sp.data(), ctb, sp.size() * sizeof(double), cudaMemcpyDeviceToHost,
                              L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  if (contact) {
    double ct[8] = {0};
    for (int part = 0; part < 2; ++part)
      for (int nu = 0; nu < 4; ++nu)
        for (int ir = 0; ir < 4; ++ir)
          for (int ia = 0; ia < 3; ++ia) {
            const double *phi = sp.data() + 24 * ((part * 4 + nu) * 12 + 3 * ir + ia);
            double s1[24], s2[24];
            for (int a = 0; a < 4; ++a)
              for (int i = 0; i < 3; ++i) {
                double re = 0, im = 0;
                for (int j = 0; j < 3; ++j) {
                  // part 0: Usource phi; part 1: Usource^+ phi
                  double ur, ui;
                  if (part == 0) { ur = Us[nu][2 * (3 * i + j)]; ui = Us[nu][2 * (3 * i + j) + 1]; }
                  else { ur = Us[nu][2 * (3 * j + i)]; ui = -Us[nu][2 * (3 * j + i) + 1]; }
                  const double vr = phi[2 * (3 * a + j)], vi = phi[2 * (3 * a + j) + 1];
                  re += ur * vr - ui * vi;
                  im += ur * vi + ui * vr;
                }
                s1[2 * (3 * a + i)] = re;
                s1[2 * (3 * a + i) + 1] = im;
              }
            for (int k = 0; k < 24; ++k) s2[k] = s1[perm[nu][k]] * sign[nu][k];
            const int k0 = 2 * (3 * ir + ia);
            if (part == 0) {
              ct[2 * nu] += -0.5 * (s2[k0] - s1[k0]);
              ct[2 * nu + 1] += -0.5 * (s2[k0 + 1] - s1[k0 + 1]);
            } else {
              ct[2 * nu] += 0.5 * (s2[k0] + s1[k0]);
              ct[2 * nu + 1] += 0.5 * (s2[k0 + 1] + s1[k0 + 1]);
            }
          }
    std::memcpy(contact, ct, sizeof ct);
  }
  return CVCB_OK;
}

int cvc_ward(cvcb_lattice *L, const double *conn, double *wi) {
  const Geom &g = L->g;
  void *cb, *wb;
  CVCB_TRY(ensure_buffer(L, SLOT_CONN, (size_t)g.V * 32 * sizeof(double), &cb));
  CVCB_TRY(ensure_buffer(L, SLOT_STAGE_B, (size_t)g.V * 24 * sizeof(double), &wb));
  CVCB_CUDA(cudaMemcpyAsync(cb, conn, (size_t)g.V * 32 * sizeof(double), cudaMemcpyDefault,
                            L->stream));
  k_cvc_ward<<<(g.V + 127) / 128, 128, 0, L->stream>>>(static_cast<double *>(wb),
                                                        static_cast<const double *>(cb), g);
  CVCB_LAUNCHED(L);
  CVCB_CUDA(cudaMemcpyAsync(wi, wb, (size_t)g.V * 8 * sizeof(double), cudaMemcpyDefault,
                            L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  return CVCB_OK;
}

int p2gg_seq_source(cvcb_lattice *L, double *source, const double *prop, int t, const int mom[3],
                    int gamma_id, int pos) {
  const Geom &g = L->g;
  if (t < 0 || t >= g.T || gamma_id < 0 || gamma_id > 15) {
    set_error("timeslice %d or gamma id %d out of range", t, gamma_id);
    return CVCB_ERR_ARG;
  }
  const double *dprop = prop;
  double *dsrc = source;
  void *a, *b;
  const size_t bytes = (size_t)g.V * 24 * sizeof(double);
  if (!is_device_ptr(prop)) {
    CVCB_TRY(ensure_buffer(L, SLOT_STAGE_A, bytes, &a));
    CVCB_CUDA(cudaMemcpyAsync(a, prop, bytes, cudaMemcpyHostToDevice, L->stream));
    dprop = static_cast<const double *>(a);
  }
  const bool host_out = !is_device_ptr(source);
  if (host_out) {
    CVCB_TRY(ensure_buffer(L, SLOT_STAGE_B, bytes, &b));
    dsrc = static_cast<double *>(b);
  }
  int perm[16][24], sign[16][24];
  gamma_tables(perm, sign);
  GammaTab gt;
  for (int k = 0; k < 24; ++k) {
    gt.perm[k] = perm[gamma_id][k];
    gt.sign[k] = sign[gamma_id][k];
  }
  const double sgn2pi = (1. - 2. * pos) * 2. * M_PI;
  k_seq_source<<<(g.V + 127) / 128, 128, 0, L->stream>>>(dsrc, dprop, g, t, mom[0], mom[1], mom[2],
                                                          sgn2pi, gt);
  CVCB_LAUNCHED(L);
  if (host_out)
    CVCB_CUDA(cudaMemcpyAsync(source, dsrc, bytes, cudaMemcpyDeviceToHost, L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  return CVCB_OK;
}

struct StorePlaq {
  double *out;
  __device__ void operator()(const double (&t)[1]) const { out[0] = t[0]; }
};
struct StoreLinksum {
  double *out;
  __device__ void operator()(const double (&t)[2]) const {
    out[1] = t[0];
    out[2] = t[1];
  }
};

int plaquette(cvcb_lattice *L, double *plaq, double *linksum) {
  CVCB_TRY(need_gauge(L));
  const Geom &g = L->g;
  void *raw, *eo;
  CVCB_TRY(ensure_buffer(L, SLOT_STAGE_A, (size_t)g.V * 72 * sizeof(double), &raw));
  CVCB_TRY(ensure_buffer(L, SLOT_F0, (size_t)g.V * 36 * sizeof(double2), &eo));
  CVCB_CUDA(cudaMemcpyAsync(raw, L->gauge_host.data(), (size_t)g.V * 72 * sizeof(double),
                            cudaMemcpyHostToDevice, L->stream));
  k_gauge_raw_eo<<<(g.V + 127) / 128, 128, 0, L->stream>>>(static_cast<double2 *>(eo),
                                                            static_cast<const double2 *>(raw), g);
  CVCB_LAUNCHED(L);
  CVCB_TRY(launch_reduce<1>(L, PlaqF{static_cast<const double2 *>(eo), g},
                            StorePlaq{L->red_result}, (size_t)g.V));
  CVCB_TRY(launch_reduce<2>(L, LinkSumF{static_cast<const double2 *>(raw)},
                            StoreLinksum{L->red_result}, (size_t)g.V * 36));
  double r[3];
  CVCB_CUDA(cudaMemcpyAsync(r, L->red_result, 3 * sizeof(double), cudaMemcpyDeviceToHost,
                            L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  if (plaq) *plaq = r[0] / ((double)g.V * 18.0);
  if (linksum) {
    linksum[0] = r[1];
    linksum[1] = r[2];
  }
  return CVCB_OK;
}

}  // namespace cvcb

using namespace cvcb;

extern "C" {

int cvcb_cvc_contract(cvcb_lattice *L, const double *const *fields, int source_site, double *conn,
                      double *contact) {
  if (!L || !fields || !conn) return CVCB_ERR_NULL;
  CVCB_CUDA(cudaSetDevice(L->device));
  return cvc_contract(L, fields, source_site, conn, contact);
}

int cvcb_cvc_ward(cvcb_lattice *L, const double *conn, double *wi) {
  if (!L || !conn || !wi) return CVCB_ERR_NULL;
  CVCB_CUDA(cudaSetDevice(L->device));
  return cvc_ward(L, conn, wi);
}

int cvcb_p2gg_seq_source(cvcb_lattice *L, double *source, const double *prop, int timeslice,
                         const int momentum[3], int gamma_id, int propagator_position) {
  if (!L || !source || !prop || !momentum) return CVCB_ERR_NULL;
  CVCB_CUDA(cudaSetDevice(L->device));
  return p2gg_seq_source(L, source, prop, timeslice, momentum, gamma_id, propagator_position);
}

int cvcb_plaquette(cvcb_lattice *L, double *plaq, double *linksum) {
  if (!L) return CVCB_ERR_NULL;
  CVCB_CUDA(cudaSetDevice(L->device));
  return plaquette(L, plaq, linksum);
}

}  // extern "C"
