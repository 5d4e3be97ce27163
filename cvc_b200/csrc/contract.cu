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
#include <algorithm>
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
// One block per SM walks through groups of 8 consecutive lexicographic sites
// (V is a multiple of 16), two stages (parts) per group.  A stage forms in
// shared memory the Z columns of all four nu (2 x 3 columns each) from the 48
// shifted columns, and the projected and transported half spinors u of the 12
// columns of the source point for the 8 neighbours; then each thread (colour
// of the sink, nu, site, a, sign of the hop) forms its dots.  u is formed once
// for all four nu, and the local columns need neither a copy in another
// layout nor Z columns in memory.
//
// The SM holds only 12 warps of this (registers, shared memory), so a stage's
// shifted columns (site-major, read once and coalesced) come to shared memory
// by cp.async during the stage before, and so do the next group's links; the
// first of a warp's two neighbour tasks is loaded into registers before the
// dots of the stage before, the second before the Z columns are formed.
//
// Bounds at 24^3 x 48: 15.9 GB of compulsory traffic (2.4 ms at 6.55 TB/s) and
// 42.6 k FP64 instructions per site (1.5 ms at 64 per SM and clock).  Measured
// 7.1 ms (the whole contraction 8.3 ms; 44.6 ms with the columns copied to
// component-major order, Z columns in memory and one thread per site; 0.26
// against 2.41 ms at 8^3 x 16).  The shared-memory and load queues bound it
// (L1 data pipe 51 %, FP64 pipe 21 % busy).  Measured against it: two blocks
// of 6 warps without the asynchronous copies 8.8 ms, of 12 warps at 80
// registers 9.7; one nu and all mu per thread, half again the reads of u, 8.6;
// the source point's columns not tiled (below) 8.5; the shifted columns by
// bulk copies 9.3; both neighbour tasks in flight together 11.4; another
// order of the groups, with the neighbours' timeslices in L2, no change.
constexpr int kPiSites = 8;
constexpr int kPiThreads = 384, kPiWarps = kPiThreads / 32;
constexpr int kPiZPitch = 13;                    // components of a site and one to spread the banks
constexpr int kPiZ = 4 * 2 * 3 * kPiZPitch * kPiSites;  // double2: [nu][a][o][site][comp]
constexpr int kPiU = 3 * 4 * 8 * 6 * kPiSites;   // double2: [ia][ir][dir][spin][colour][site]
constexpr int kPiRaw = 48 * 12 * kPiSites;       // double2: [column][site][comp]
constexpr int kPiRed = 3 * 8 * 4 * kPiSites;     // double2: [sink colour][dir][nu][site]
constexpr int kPiW = 8 * 9 * kPiSites;           // double2: [dir][entry][site], of this and the next group
constexpr size_t kPiSmem = (kPiZ + kPiU + kPiRaw + kPiRed + 2 * kPiW) * sizeof(double2);

struct PiArgs {
  const double2 *loc[2][48];  // part 0: dn, part 1: up columns of the shifted points, site-major
  const double2 *fix;         // columns of the source point (fix_slot)
  const double2 *U;
  double2 *F, *B;   // T_+ and T_-, [V][mu][nu]
  double2 us[4][9]; // conj of the phased source links
  double lam[4][2]; // lam = lam (nu = 0, 2) or i lam (nu = 1, 3), per a
  Geom g;
};

__device__ __forceinline__ SiteCoord lex_coord(const Geom &g, int lex) {
  SiteCoord cd;
  const unsigned r0 = fdiv((unsigned)lex, g.dLZ), r1 = fdiv(r0, g.dLY), r2 = fdiv(r1, g.dLX);
  cd.lex = lex;
  cd.z = lex - (int)r0 * g.LZ;
  cd.y = (int)(r0 - r1 * g.LY);
  cd.x = (int)(r1 - r2 * g.LX);
  cd.t = (int)r2;
  return cd;
}

// Columns of the source point, tiled by 8 lexicographic sites with all 24
// columns (12 up, 12 dn) of a tile together: [tile][column][component][site].
// A group's neighbours in one direction are then one or two runs of 37 KB;
// with the columns apart, every 128 bytes came from another page.
__device__ __forceinline__ size_t fix_slot(int lex, int col) {
  return ((size_t)(lex >> 3) * 24 + col) * 12 * kPiSites + (lex & 7);
}

__device__ __forceinline__ void cp_async16(double2 *dst, const double2 *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}

// the 64 links of a group's hops: dir = mu (forward, at the site) or 4 + mu
// (backward, at the neighbour)
__device__ __forceinline__ void pi_fetch_links(const PiArgs &A, double2 *sw, int base) {
  const Geom &g = A.g;
  for (int k = threadIdx.x; k < kPiW; k += kPiThreads) {
    const int site = k % kPiSites, q = k / kPiSites, e = q % 9, dir = q / 9, mu = dir & 3;
    const SiteCoord cd = lex_coord(g, base + site);
    const int par = (cd.t + cd.x + cd.y + cd.z) & 1;
    const int at = dir < 4 ? par * g.Vh + (cd.lex >> 1) : (1 - par) * g.Vh + (nb_lex(g, cd, mu, -1) >> 1);
    cp_async16(sw + k, A.U + (size_t)(mu * 9 + e) * g.V + at);
  }
}

// One neighbour task q = 3 direction + colour: the column of the lane's source
// spin at the neighbour of the lane's site.
__device__ __forceinline__ void pi_load(double2 (&f)[12], const PiArgs &A, int lex, int part, int q, int ir) {
  const Geom &g = A.g;
  const int j = nb_lex(g, lex_coord(g, lex), q / 3 & 3, q < 12 ? +1 : -1);
  const double2 *col = A.fix + fix_slot(j, part * 12 + 3 * ir + q % 3);
#pragma unroll
  for (int k = 0; k < 12; ++k) f[k] = __ldg(col + k * kPiSites);
}
template <int MU, int S>
__device__ __forceinline__ void pi_transport(const double2 (&fv)[12], const double2 *w, double2 *u) {
  Spinor<double> f;
#pragma unroll
  for (int k = 0; k < 12; ++k) f.c[k / 3][k % 3] = cx(fv[k].x, fv[k].y);
  const HalfSpinor<double> h = project(MU, S, f);
  Link<double> W;
#pragma unroll
  for (int k = 0; k < 9; ++k) W.m[k / 3][k % 3] = cx(w[k * kPiSites].x, w[k * kPiSites].y);
  const HalfSpinor<double> r = S < 0 ? link_mul(W, h) : link_dag_mul(W, h);
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      u[(3 * b + c) * kPiSites] = make_double2(r.c[b][c].re, r.c[b][c].im);
}
__device__ __forceinline__ void pi_store(const double2 (&f)[12], const double2 *sw, double2 *su, int q,
                                         int ir, int site) {
  const int dir = q / 3, ia = q % 3;
  double2 *u = su + ((ia * 4 + ir) * 8 + dir) * 6 * kPiSites + site;
  const double2 *w = sw + dir * 9 * kPiSites + site;
  switch (dir) {
    case 0: pi_transport<0, -1>(f, w, u); break;
    case 1: pi_transport<1, -1>(f, w, u); break;
    case 2: pi_transport<2, -1>(f, w, u); break;
    case 3: pi_transport<3, -1>(f, w, u); break;
    case 4: pi_transport<0, +1>(f, w, u); break;
    case 5: pi_transport<1, +1>(f, w, u); break;
    case 6: pi_transport<2, +1>(f, w, u); break;
    default: pi_transport<3, +1>(f, w, u); break;
  }
}

// z + s w and z + s i w
__device__ __forceinline__ Cx<double> add_s(Cx<double> z, double s, Cx<double> w) {
  return cx(fma(s, w.re, z.re), fma(s, w.im, z.im));
}
__device__ __forceinline__ Cx<double> add_si(Cx<double> z, double s, Cx<double> w) {
  return cx(fma(-s, w.im, z.re), fma(s, w.re, z.im));
}

// a stage's 48 local columns of the 8 sites from lexicographic site `base`
__device__ __forceinline__ void pi_fetch_local(const PiArgs &A, double2 *raw, int base, int part) {
  for (int k = threadIdx.x; k < kPiRaw; k += kPiThreads) {
    const int col = k / (12 * kPiSites), e = k % (12 * kPiSites);
    cp_async16(raw + k, A.loc[part][col] + (size_t)base * 12 + e);
  }
}

// Z columns: 8 (nu, a) x 96 elements (site, component), six columns in, three out
__device__ __forceinline__ void pi_z(const PiArgs &A, double2 *sz, const double2 *raw, int warp, int lane) {
#pragma unroll 1
  for (int q = warp; q < 24; q += kPiWarps) {
    const int na = q / 3, nu = na >> 1, za = na & 1;
    const int zp = nu == 0 || nu == 3 ? za + 2 : 3 - za;
    const int e = (q % 3) * 32 + lane, es = e / 12, ec = e - 12 * es;
    const double2 *f = raw + 12 * nu * 12 * kPiSites + e;
    const double l = A.lam[nu][za];
    Cx<double> y[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double2 v = f[(3 * za + i) * 12 * kPiSites], w = f[(3 * zp + i) * 12 * kPiSites];
      y[i] = nu & 1 ? add_si(cx(v.x, v.y), -l, cx(w.x, w.y)) : add_s(cx(v.x, v.y), -l, cx(w.x, w.y));
    }
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      Cx<double> z = cx(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < 3; ++i) cfma(z, cx(A.us[nu][3 * o + i].x, A.us[nu][3 * o + i].y), y[i]);
      sz[((na * 3 + o) * kPiSites + es) * kPiZPitch + ec] = make_double2(z.re, z.im);
    }
  }
}

// The dots of one thread: both nu of a class (zr with a real lam, zi with an
// imaginary one: they share the u that they read) and mu = 2 MH, 2 MH + 1.
template <int MH>
__device__ __forceinline__ void pi_dots(Cx<double> (&acc)[2][2], const double2 *zr, const double2 *zi,
                                        const double2 *su, double lr, double li, double s, int si,
                                        int site, int a, int ap, int sg) {
#pragma unroll 1
  for (int o = 0; o < 3; ++o) {
    Cx<double> z[2][4];
#pragma unroll
    for (int sp = 0; sp < 4; ++sp) {
      const int k = (o * kPiSites + site) * kPiZPitch + 3 * sp + si;
      z[0][sp] = cx(zr[k].x, zr[k].y);
      z[1][sp] = cx(zi[k].x, zi[k].y);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int mu = 2 * MH + m, d = sg * 4 + mu;
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
        cfmac(acc[0][m], (mu & 1) ? add_si(z[0][b], sb, z[0][hi]) : add_s(z[0][b], sb, z[0][hi]), vr);
        cfmac(acc[1][m], (mu & 1) ? add_si(z[1][b], sb, z[1][hi]) : add_s(z[1][b], sb, z[1][hi]), vi);
      }
    }
  }
}

__global__ void __launch_bounds__(kPiThreads, 1) k_pi(const __grid_constant__ PiArgs A) {
  extern __shared__ double2 sm[];
  double2 *sz = sm, *su = sz + kPiZ, *raw = su + kPiU, *red = raw + kPiRaw, *sw = red + kPiRed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int site = lane & 7, ir = lane >> 3;  // of the neighbour tasks
  // the dots' role of the thread
  const int si = warp % 3, cls = warp / 3 & 1, mh = warp / 6;  // colour of the sink; nu in {0,3} or {2,1}; mu
  const int a = (lane >> 3) & 1, sg = lane >> 4;               // source spin; forward or backward hop
  const int ap = cls == 0 ? a + 2 : 3 - a;                     // its partner
  const int nur = cls == 0 ? 0 : 2, nui = cls == 0 ? 3 : 1;
  const double lr = A.lam[nur][a], li = A.lam[nui][a], s = sg ? 1.0 : -1.0;
  const double2 *zr = sz + (nur * 2 + a) * 3 * kPiSites * kPiZPitch;
  const double2 *zi = sz + (nui * 2 + a) * 3 * kPiSites * kPiZPitch;
  const int step = gridDim.x * kPiSites;
  int base = blockIdx.x * kPiSites, wb = 0;  // wb: which half of sw holds this group's links
  if (base >= A.g.V) return;
  double2 f[12];
  pi_fetch_local(A, raw, base, 0);
  pi_fetch_links(A, sw, base);
  pi_load(f, A, base + site, 0, warp, ir);
  for (;; base += step, wb = kPiW - wb) {
    Cx<double> acc[2][2];
#pragma unroll
    for (int n = 0; n < 2; ++n) acc[n][0] = acc[n][1] = cx(0.0, 0.0);
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();  // raw and the links are complete; the dots of the stage before are done
      pi_store(f, sw + wb, su, warp, ir, site);
      pi_load(f, A, base + site, part, warp + kPiWarps, ir);
      pi_z(A, sz, raw, warp, lane);
      pi_store(f, sw + wb, su, warp + kPiWarps, ir, site);
      __syncthreads();  // sz and su are complete, raw is free
      const int nbase = part ? base + step : base;  // the next stage
      if (nbase < A.g.V) {
        pi_fetch_local(A, raw, nbase, 1 - part);
        if (part) pi_fetch_links(A, sw + (kPiW - wb), nbase);
        pi_load(f, A, nbase + site, 1 - part, warp, ir);
      }
      if (mh)
        pi_dots<1>(acc, zr, zi, su, lr, li, s, si, site, a, ap, sg);
      else
        pi_dots<0>(acc, zr, zi, su, lr, li, s, si, site, a, ap, sg);
      // the second part enters conjugated: conj(conj(T_0) + T_1)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int m = 0; m < 2; ++m) acc[n][m].im = -acc[n][m].im;
    }
    // sum over a (lanes) and the sink's colour (warps), in a fixed order
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        Cx<double> v = acc[n][m];
        v.re += __shfl_xor_sync(0xffffffffu, v.re, 8);
        v.im += __shfl_xor_sync(0xffffffffu, v.im, 8);
        if (a == 0)
          red[((si * 8 + sg * 4 + 2 * mh + m) * 4 + (n ? nui : nur)) * kPiSites + site] = make_double2(v.re, v.im);
      }
    __syncthreads();
    if (threadIdx.x < 256) {
      const int k = threadIdx.x, ks = (k >> 4) & 7;
      const int slot = (((k >> 7) * 4 + ((k >> 2) & 3)) * 4 + (k & 3)) * kPiSites + ks;
      const double2 x = red[slot], y = red[slot + kPiRed / 3], w = red[slot + 2 * (kPiRed / 3)];
      double2 *o = (k >> 7) ? A.B : A.F;
      o[(size_t)(base + ks) * 16 + (k & 15)] = make_double2(x.x + y.x + w.x, x.y + y.y + w.y);
    }
    if (base + step >= A.g.V) break;
  }
}

// conn_mu_nu(x) = -1/4 (T_+(x) - T_-(x + mu))   (normalisation, :861)
__global__ void k_pi_combine(double2 *__restrict__ conn, const double2 *__restrict__ F,
                             const double2 *__restrict__ B, Geom g) {
  const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (k >= (size_t)g.V * 16) return;
  const SiteCoord cd = lex_coord(g, (int)(k >> 4));
  const int m = (int)(k & 15);
  const double2 f = F[k], b = B[(size_t)nb_lex(g, cd, m >> 2, +1) * 16 + m];
  conn[k] = make_double2(-0.25 * (f.x - b.x), -0.25 * (f.y - b.y));
}

// columns of the source point from CVC layout to the tiles of fix_slot
struct FixCols {
  const double2 *src[24];
};
constexpr int kFixTile = 64;
__global__ void __launch_bounds__(128) k_fix_columns(double2 *__restrict__ dst,
                                                    const __grid_constant__ FixCols c, int V) {
  __shared__ double2 t[kFixTile * 13];
  const int base = blockIdx.x * kFixTile, n = min(kFixTile, V - base);
  const double2 *src = c.src[blockIdx.y] + (size_t)base * 12;
  for (int q = threadIdx.x; q < n * 12; q += blockDim.x) t[q + q / 12] = __ldg(src + q);
  __syncthreads();
  for (int q = threadIdx.x; q < n * 12; q += blockDim.x) {
    const int tile = q / (12 * kPiSites), r = q % (12 * kPiSites), k = r / kPiSites, s = r % kPiSites;
    dst[fix_slot(base + tile * kPiSites, blockIdx.y) + r] = t[(tile * kPiSites + s) * 13 + k];
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
  int sms = 0;
  CVCB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, L->device));
  k_pi<<<std::min(g.V / kPiSites, sms), kPiThreads, kPiSmem, L->stream>>>(A);
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
