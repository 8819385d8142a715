// Two-level adaptive aggregation multigrid for the full Wilson or clover
// operator M = A - kappa D (A = 1 without clover).  qcu's own multigrid file
// is empty (src/multgrid.cu); the method is the aggregation multigrid that
// PyQuda configures for QUDA in python/PyQuda/pyquda/dslash/general.py:121-230
// (aggregates of geo_block_size sites, n_vec near-null vectors, chirality
// kept, MR smoother, loosely solved coarse system, flexible GCR outside).
//
// Set-up
//   * near-null vectors: for k = 1..n_vec, a Gaussian v0 and the error left
//     by a short solve of M y = M v0 (FP32 BiCGSTAB on the even-odd system,
//     setup_maxiter iterations), v = v0 - y: the slowly converging, low modes;
//   * aggregates: blocks of geo_block_size sites (both parities), each split
//     by chirality (spins 0,1 and 2,3: gamma_5 is diagonal in the DeGrand-Rossi
//     basis), so the coarse space keeps gamma_5's block structure;
//   * P: the vectors orthonormalised on every aggregate and chirality
//     (modified Gram-Schmidt with FP64 sums), stored in FP32;
//   * the Galerkin operator A_c = P^dag M P, built directly from the fine
//     hops: per aggregate a self block X (the local term A and the hops that
//     stay inside the aggregate) and one block Y_d per direction (the hops
//     that leave it), each 2 n_vec x 2 n_vec complex, FP32.
// Solve: flexible GCR in FP64 on the full system, preconditioned by one
// two-level cycle: nu_pre MR steps, the coarse correction P A_c^-1 P^dag r
// (FP32 BiCGSTAB on A_c to coarse_tol, at most coarse_maxiter iterations),
// nu_post MR steps.  The FP64 true residual decides convergence.
#include <chrono>
#include <cmath>
#include <cstddef>
#include <memory>
#include <vector>

#include "gridbar.cuh"
#include "mg.h"

namespace qcu {

namespace {

constexpr int MG_MAXVEC = 16;
constexpr int MG_MAXBLOCK = 512;  // sites per aggregate, at most
constexpr int MG_RED = 256;
constexpr int MG_RED_GRID = 148 * 4;

struct MGGeom {
  int L[4];    // fine full extents (x, y, z, t)
  int b[4];    // aggregate extents
  int nb[4];   // aggregates per direction
  int nblocks;
  int bsites;  // sites per aggregate (both parities)
  int Vh, Vp;  // sites per parity, and padded to the site blocks of 32
  int nvec;
  int nc;      // coarse degrees of freedom per aggregate (2 nvec)
};

struct SiteC {
  int x[4];  // full coordinates
  int par, s;
};

// site t (< bsites) of aggregate B: full coordinates, parity, half-lattice
// index i = ((t Lz + z) Ly + y) Lx/2 + x/2 (the PyQuda/qcu ordering)
__device__ __forceinline__ SiteC mg_site(const MGGeom &m, int B, int t) {
  SiteC c;
  int r = B, q = t;
#pragma unroll
  for (int d = 0; d < 4; d++) {
    c.x[d] = (r % m.nb[d]) * m.b[d] + q % m.b[d];
    r /= m.nb[d];
    q /= m.b[d];
  }
  c.par = (c.x[0] + c.x[1] + c.x[2] + c.x[3]) & 1;
  c.s = ((c.x[3] * m.L[2] + c.x[2]) * m.L[1] + c.x[1]) * (m.L[0] / 2) + (c.x[0] >> 1);
  return c;
}
__device__ __forceinline__ int mg_block_of(const MGGeom &m, const int x[4]) {
  return ((x[3] / m.b[3] * m.nb[2] + x[2] / m.b[2]) * m.nb[1] + x[1] / m.b[1]) * m.nb[0] + x[0] / m.b[0];
}
// the aggregate next to B in direction d = 2 mu + (0 forward, 1 backward); d = 8: B itself
__device__ __forceinline__ int mg_cnbr(const MGGeom &m, int B, int d) {
  if (d == 8) return B;
  const int mu = d >> 1;
  int stride = 1, n = m.nb[0];  // selects, not an indexed array: no local memory
  if (mu >= 1) stride *= m.nb[0], n = m.nb[1];
  if (mu >= 2) stride *= m.nb[1], n = m.nb[2];
  if (mu >= 3) stride *= m.nb[2], n = m.nb[3];
  const int c = (B / stride) % n;
  const int cn = (d & 1) ? (c == 0 ? n - 1 : c - 1) : (c == n - 1 ? 0 : c + 1);
  return B + (cn - c) * stride;
}

// a full fine vector: two site-blocked parity slabs in the SOA64 element
// order, parity p at p * Vp * 12
__device__ __forceinline__ size_t fidx(const MGGeom &m, int par, int s, int comp) {
  return (size_t)par * m.Vp * 12 + blk_base<12>(s) + (size_t)comp * SB;
}
// near-null vector k, FP32, aggregate-major: component comp of site t of
// aggregate B at ((k nblocks + B) 12 + comp) bsites + t, so the threads of
// an aggregate (one per site) read each component as one contiguous run
__device__ __forceinline__ size_t nidx(const MGGeom &m, int k, int B, int t, int comp) {
  return (((size_t)k * m.nblocks + B) * 12 + comp) * m.bsites + t;
}
// the index within its aggregate of the site with full coordinates x (inverse of mg_site)
__device__ __forceinline__ int mg_local(const MGGeom &m, const int x[4]) {
  return ((x[3] % m.b[3] * m.b[2] + x[2] % m.b[2]) * m.b[1] + x[1] % m.b[1]) * m.b[0] + x[0] % m.b[0];
}

// the coarse operator of aggregate B as a 9 nc x nc complex matrix
// (column j = d nc + col: d = 0..7 the directions Y_d, d = 8 the self block
// X), stored with the columns in pairs: element (j, row) at float2 index
// ((B * 9 nc / 2 + j / 2) * nc + row) * 2 + j % 2, so a lane reading its row
// takes the entries of two columns in one 16-byte load
__host__ __device__ __forceinline__ size_t yidx(const MGGeom &m, int B, int j, int row) {
  return (((size_t)B * (9 * m.nc / 2) + j / 2) * m.nc + row) * 2 + (j & 1);
}

// sum of N doubles over the thread block, every thread gets the totals
// (sh: blockDim / 32 * N doubles)
template <int N>
__device__ __forceinline__ void mg_block_sum(double (&v)[N], double *sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < N; k++)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  __syncthreads();  // sh may still be read by an earlier call
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < N; k++) sh[w * N + k] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; k++) {
    double t = 0;
    for (int q = 0; q < nw; q++) t += sh[q * N + k];
    v[k] = t;
  }
}

// ---------------------------------------------------------------- P and P^dag
// modified Gram-Schmidt of the near-null vectors on every aggregate and
// chirality (one thread block per aggregate, one thread per site)
__global__ void __launch_bounds__(MG_MAXBLOCK) k_mg_orth(MGGeom m, float2 *nv) {
  __shared__ double sh[(MG_MAXBLOCK / 32) * 4];
  const int B = blockIdx.x, t = threadIdx.x;
  for (int k = 0; k < m.nvec; k++) {
    for (int j = 0; j <= k; j++) {
      double v[4] = {0, 0, 0, 0};  // per chirality: Re, Im of <v_j, v_k> (j == k: |v_k|^2)
      for (int comp = 0; comp < 12; comp++) {
        const int ch = comp / 6;
        const float2 a = nv[nidx(m, j, B, t, comp)], b = nv[nidx(m, k, B, t, comp)];
        v[2 * ch] += (double)a.x * b.x + (double)a.y * b.y;
        v[2 * ch + 1] += (double)a.x * b.y - (double)a.y * b.x;
      }
      mg_block_sum<4>(v, sh);
      for (int comp = 0; comp < 12; comp++) {
        const int ch = comp / 6;
        float2 &b = nv[nidx(m, k, B, t, comp)];
        if (j < k) {  // v_k -= <v_j, v_k> v_j
          const float2 a = nv[nidx(m, j, B, t, comp)];
          const double dr = v[2 * ch], di = v[2 * ch + 1];
          b = make_float2((float)(b.x - (dr * a.x - di * a.y)), (float)(b.y - (dr * a.y + di * a.x)));
        } else {
          const double inv = v[2 * ch] > 0 ? 1.0 / sqrt(v[2 * ch]) : 0.0;
          b = make_float2((float)(b.x * inv), (float)(b.y * inv));
        }
      }
    }
  }
}

// A fine FP64 vector as two parity slabs (SOA64 element order); a null
// slab reads as zero and is not written.
struct FineVec {
  double2 *p[2];
};
__device__ __forceinline__ size_t hidx(int s, int comp) { return blk_base<12>(s) + (size_t)comp * SB; }

// The sums over the warp of 16 values, value lane / 2 in each lane: a halving
// exchange, 16 shuffles where a butterfly per value takes 80.
__device__ __forceinline__ double warp_sum16(double (&v)[16]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int w = 8, off = 16; w >= 1; w >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (i < w) {
        const double send = up ? v[i] : v[i + w], keep = up ? v[i + w] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// coarse c[B][ch nvec + k] = <v_k^ch, r>_B: warp sums for four vectors at a
// time, then one pass over the warps.  Bound by the near-null vectors' bytes
// (96 n_vec a site): 16^3 x 32, n_vec 12: 77 -> 46 us.
__global__ void __launch_bounds__(MG_MAXBLOCK) k_mg_restrict(MGGeom m, const float2 *nv, FineVec r, float2 *cv) {
  __shared__ double red[MG_MAXBLOCK / 32][MG_MAXVEC][4];
  const int B = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5, nw = blockDim.x >> 5;
  const SiteC c = mg_site(m, B, t);
  const double2 *rp = c.par ? r.p[1] : r.p[0];  // a select: no local copy of r
  double2 rv[12];
#pragma unroll
  for (int comp = 0; comp < 12; comp++) rv[comp] = rp ? rp[hidx(c.s, comp)] : make_double2(0, 0);
  for (int k0 = 0; k0 < m.nvec; k0 += 4) {
    double v[16];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = 0.0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (rp && k0 + q < m.nvec) {
        const float2 *p = nv + nidx(m, k0 + q, B, t, 0);
#pragma unroll
        for (int comp = 0; comp < 12; comp++) {
          const int i = 4 * q + 2 * (comp / 6);
          const float2 a = p[comp * m.bsites];
          v[i] += (double)a.x * rv[comp].x + (double)a.y * rv[comp].y;
          v[i + 1] += (double)a.x * rv[comp].y - (double)a.y * rv[comp].x;
        }
      }
    }
    const double tot = warp_sum16(v);
    if (!(lane & 1) && k0 + (lane >> 3) < m.nvec) red[w][k0 + (lane >> 3)][(lane >> 1) & 3] = tot;
  }
  __syncthreads();
  for (int i = t; i < 2 * m.nvec; i += blockDim.x) {  // i = ch nvec + k
    const int ch = i / m.nvec, k = i % m.nvec;
    double re = 0, im = 0;
    for (int q = 0; q < nw; q++) {
      re += red[q][k][2 * ch];
      im += red[q][k][2 * ch + 1];
    }
    cv[(size_t)B * m.nc + i] = make_float2((float)re, (float)im);
  }
}

// e = P c (e += P c when add)
__global__ void __launch_bounds__(MG_MAXBLOCK) k_mg_prolong(MGGeom m, const float2 *nv, const float2 *cv, FineVec e,
                                                          int add) {
  const int B = blockIdx.x, t = threadIdx.x;
  const SiteC c = mg_site(m, B, t);
  double2 *ep = c.par ? e.p[1] : e.p[0];
  if (!ep) return;
  const float2 *cb = cv + (size_t)B * m.nc;
#pragma unroll
  for (int comp = 0; comp < 12; comp++) {
    const int ch = comp / 6;
    double re = 0, im = 0;
    for (int k = 0; k < m.nvec; k++) {
      const float2 a = nv[nidx(m, k, B, t, comp)];
      const float2 q = cb[ch * m.nvec + k];
      re += (double)a.x * q.x - (double)a.y * q.y;
      im += (double)a.x * q.y + (double)a.y * q.x;
    }
    double2 &o = ep[hidx(c.s, comp)];
    if (add) o = make_double2(o.x + re, o.y + im);
    else o = make_double2(re, im);
  }
}

// ---------------------------------------------------------------- coarse operator
// h = the hop of direction MU (forward or backward) at site (par, s) applied
// to near-null vector k2 restricted to chirality ch2, taken at the neighbour
// n (site tn of aggregate Bn): U (1 - gamma_mu) forward, U^dag (1 + gamma_mu)
// backward, the stencil core of the dslash kernels
template <int MU, bool FWD>
__device__ __forceinline__ void mg_hop(const MGGeom &m, const GaugeView<GSOA64> &U, const float2 *nv, int par, int s,
                                       int n, int Bn, int tn, int k2, int ch2, double ph, Cpx<double> h[12]) {
  Cpx<double> psi[12], u[9];
#pragma unroll
  for (int comp = 0; comp < 12; comp++) {
    if (comp / 6 == ch2) {
      const float2 a = nv[nidx(m, k2, Bn, tn, comp)];
      psi[comp] = Cpx<double>(a.x, a.y);
    } else {
      psi[comp] = Cpx<double>(0, 0);
    }
  }
  link_load<GSOA64, double>(U, MU, FWD ? par : 1 - par, FWD ? s : n, u);
#pragma unroll
  for (int q = 0; q < 12; q++) h[q] = Cpx<double>(0, 0);
  hop<MU, FWD, MU == 3, double>(h, psi, u, ph);
}

// The coarse operator (yidx), column j = d nc + col, d = 0..7 the directions
// (Y_d), d = 8 the self block X; col = ch2 nvec + k2 (the vector acted on),
// row = ch nvec + k:
//   Y_d = -kappa sum_{x in B, x +- mu outside B} v_row(x)^dag [D_d v_col](x)
//   X   = sum_{x in B} v_row^dag A v_col - kappa sum_{x, x +- mu in B} v_row^dag [D_d v_col](x)
// One thread block per aggregate, one thread per site; sums by warp shuffles,
// then over the warps in shared memory.
__global__ void __launch_bounds__(MG_MAXBLOCK) k_mg_build(MGGeom m, GaugeView<GSOA64> U, CloverView<CSOA64> A0,
                                                        CloverView<CSOA64> A1, int clover, double t_bc,
                                                        double kappa, const float2 *nv, float2 *Y) {
  __shared__ double red[MG_MAXBLOCK / 32][MG_MAXVEC][8];
  __shared__ double2 xs[2 * MG_MAXVEC][2 * MG_MAXVEC];
  const int B = blockIdx.x;
  const int nc = m.nc, nvec = m.nvec;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int t = threadIdx.x;
  const SiteC c = mg_site(m, B, t);
  for (int i = threadIdx.x; i < nc * nc; i += blockDim.x) xs[i / nc][i % nc] = make_double2(0, 0);
  __syncthreads();
  for (int d = 0; d < 9; d++) {
    int n = 0, inblock = 1, Bn = B, tn = t;
    double ph = 1.0;
    if (d < 8) {
      const int mu = d >> 1;
      const bool fwd = !(d & 1);
      int y[4] = {c.x[0], c.x[1], c.x[2], c.x[3]};
      y[mu] = fwd ? (y[mu] + 1) % m.L[mu] : (y[mu] + m.L[mu] - 1) % m.L[mu];
      n = ((y[3] * m.L[2] + y[2]) * m.L[1] + y[1]) * (m.L[0] / 2) + (y[0] >> 1);
      Bn = mg_block_of(m, y);
      tn = mg_local(m, y);
      inblock = Bn == B;
      if (mu == 3 && ((fwd && c.x[3] == m.L[3] - 1) || (!fwd && c.x[3] == 0))) ph = t_bc;
    }
    for (int col = 0; col < nc; col++) {
      const int ch2 = col / nvec, k2 = col % nvec;
      Cpx<double> h[12];
      switch (d) {
        case 0: mg_hop<0, true>(m, U, nv, c.par, c.s, n, Bn, tn, k2, ch2, ph, h); break;
        case 1: mg_hop<0, false>(m, U, nv, c.par, c.s, n, Bn, tn, k2, ch2, ph, h); break;
        case 2: mg_hop<1, true>(m, U, nv, c.par, c.s, n, Bn, tn, k2, ch2, ph, h); break;
        case 3: mg_hop<1, false>(m, U, nv, c.par, c.s, n, Bn, tn, k2, ch2, ph, h); break;
        case 4: mg_hop<2, true>(m, U, nv, c.par, c.s, n, Bn, tn, k2, ch2, ph, h); break;
        case 5: mg_hop<2, false>(m, U, nv, c.par, c.s, n, Bn, tn, k2, ch2, ph, h); break;
        case 6: mg_hop<3, true>(m, U, nv, c.par, c.s, n, Bn, tn, k2, ch2, ph, h); break;
        case 7: mg_hop<3, false>(m, U, nv, c.par, c.s, n, Bn, tn, k2, ch2, ph, h); break;
        default:  // the local term A v_col (v_col itself without clover)
#pragma unroll
          for (int comp = 0; comp < 12; comp++) {
            if (comp / 6 == ch2) {
              const float2 a = nv[nidx(m, k2, B, t, comp)];
              h[comp] = Cpx<double>(a.x, a.y);
            } else {
              h[comp] = Cpx<double>(0, 0);
            }
          }
          if (clover) clover_apply_site<CSOA64, double>(c.par ? A1 : A0, c.s, h);
          break;
      }
      for (int k = 0; k < nvec; k++) {
        double p[4] = {0, 0, 0, 0};  // Re, Im of v_k^dag h on chirality 0, then 1
#pragma unroll
        for (int comp = 0; comp < 12; comp++) {
          const int ch = comp / 6;
          const float2 a = nv[nidx(m, k, B, t, comp)];
          p[2 * ch] += (double)a.x * h[comp].re + (double)a.y * h[comp].im;
          p[2 * ch + 1] += (double)a.x * h[comp].im - (double)a.y * h[comp].re;
        }
        double q[8];  // [0..3]: hops that stay in B (and the local term), [4..7]: hops that leave it
#pragma unroll
        for (int i = 0; i < 4; i++) {
          q[i] = inblock ? p[i] : 0.0;
          q[4 + i] = inblock ? 0.0 : p[i];
        }
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) q[i] += __shfl_xor_sync(0xffffffffu, q[i], o);
        if (lane == 0)
#pragma unroll
          for (int i = 0; i < 8; i++) red[w][k][i] = q[i];
      }
      __syncthreads();
      for (int i = threadIdx.x; i < 8 * nvec; i += blockDim.x) {
        const int k = i >> 3, j = i & 7;
        double tot = 0;
        for (int q = 0; q < nw; q++) tot += red[q][k][j];
        const int leaves = j >> 2, ch = (j >> 1) & 1, im = j & 1;
        const int row = ch * nvec + k;
        const double val = d == 8 ? tot : -kappa * tot;
        if (!leaves) {
          double *x = im ? &xs[col][row].y : &xs[col][row].x;
          *x += val;  // one writer per (row, Re/Im)
        } else if (d < 8) {
          float *y = reinterpret_cast<float *>(Y + yidx(m, B, d * nc + col, row));
          y[im] = (float)val;
        }
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < nc * nc; i += blockDim.x) {
    const double2 v = xs[i / nc][i % nc];
    Y[yidx(m, B, 8 * nc + i / nc, i % nc)] = make_float2((float)v.x, (float)v.y);
  }
}

// ---------------------------------------------------------------- coarse solve on the device
__device__ __forceinline__ double2 cmul2(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cdiv2(double2 a, double2 b) {
  const double d = b.x * b.x + b.y * b.y;
  return make_double2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}

constexpr int CAPPLY_WARPS = 8;

// the entries [jp0, jp1) column pairs of one row of A_c times x (xin: the nine
// blocks' inputs); Yb: the aggregate's matrix at this row (in shared memory when SHARED)
template <bool SHARED>
__device__ __forceinline__ float2 mg_row(const float4 *Yb, int nc, const float2 *xin, int jp0, int jp1) {
  float re0 = 0.f, im0 = 0.f, re1 = 0.f, im1 = 0.f;
#pragma unroll 4
  for (int jp = jp0; jp < jp1; jp++) {
    const float4 a = SHARED ? Yb[jp * nc] : __ldg(Yb + (size_t)jp * nc);  // (A[2 jp][row], A[2 jp + 1][row])
    const float2 x0 = xin[2 * jp], x1 = xin[2 * jp + 1];
    re0 = fmaf(a.x, x0.x, fmaf(-a.y, x0.y, re0));
    im0 = fmaf(a.x, x0.y, fmaf(a.y, x0.x, im0));
    re1 = fmaf(a.z, x1.x, fmaf(-a.w, x1.y, re1));
    im1 = fmaf(a.z, x1.y, fmaf(a.w, x1.x, im1));
  }
  return make_float2(re0 + re1, im0 + im1);
}

// the same from global memory with C loads of a lane in flight at a time: 7, as
// a warp of eight has 13 or 14 column pairs of 24 rows (14 at a time cost the
// registers of a quarter of the blocks)
template <int C>
__device__ __forceinline__ float2 mg_row_wide(const float4 *Yb, int nc, const float2 *xin, int jp0, int jp1) {
  float re0 = 0.f, im0 = 0.f, re1 = 0.f, im1 = 0.f;
  for (int jp = jp0; jp < jp1; jp += C) {
    float4 a[C];
#pragma unroll
    for (int c = 0; c < C; c++) a[c] = jp + c < jp1 ? __ldg(Yb + (size_t)(jp + c) * nc) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < C; c++) {
      if (jp + c >= jp1) break;
      const float2 x0 = xin[2 * (jp + c)], x1 = xin[2 * (jp + c) + 1];
      re0 = fmaf(a[c].x, x0.x, fmaf(-a[c].y, x0.y, re0));
      im0 = fmaf(a[c].x, x0.y, fmaf(a[c].y, x0.x, im0));
      re1 = fmaf(a[c].z, x1.x, fmaf(-a[c].w, x1.y, re1));
      im1 = fmaf(a[c].z, x1.y, fmaf(a[c].w, x1.x, im1));
    }
  }
  return make_float2(re0 + re1, im0 + im1);
}

// out = A_c in, one warp per aggregate, lane = row; the neighbours' inputs
// staged in shared memory (the set-up check; the solve is k_mg_coarse)
__global__ void __launch_bounds__(32 * CAPPLY_WARPS) k_mg_capply(MGGeom m, const float4 *Y, const float2 *in,
                                                               float2 *out) {
  __shared__ float2 xin[CAPPLY_WARPS][9 * 2 * MG_MAXVEC];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int B = blockIdx.x * CAPPLY_WARPS + wib;
  const int nc = m.nc, J = 9 * nc;
  if (B >= m.nblocks) return;
  for (int i = lane; i < J; i += 32) {
    const int d = i / nc;
    xin[wib][i] = in[(size_t)mg_cnbr(m, B, d) * nc + (i - d * nc)];
  }
  __syncwarp();
  if (lane < nc) out[(size_t)B * nc + lane] = mg_row<false>(Y + (size_t)B * (J / 2) * nc + lane, nc, xin[wib], 0, J / 2);
}

struct CState {
  int status;          // of the last solve that ended
  long long total_it;  // iterations summed over the solves since the last reset
  GridRed red;         // its partials, at the end, stay on the device
};
struct CoarseArgs {
  MGGeom m;
  const float4 *Y;
  const float2 *b;
  float2 *x, *r0, *r1, *p0, *p1, *v0, *v1, *t;
  CState *st;
  double tol2;
  int maxit;
  int apb;  // aggregates a block works on at a time, a power of two
};

// x ~ A_c^-1 b by BiCGSTAB (FP32 vectors, FP64 scalars) from zero, to
// |r|^2 <= tol2 |b|^2 or maxit iterations, as one cooperative kernel.  Two grid
// barriers an iteration, after each application of A_c: a block forms the
// vectors it needs at its aggregates' neighbours itself, from the vectors
// before the update (which therefore alternate between two buffers) and the
// scalars, instead of waiting for another block to store them; and <rt, r> and
// |r|^2 of the new residual r = s - omega t follow from the products of s, t
// and rt that the second application's reduction carries,
//   <rt, r> = <rt, s> - omega <rt, t>,   |r|^2 = |s|^2 - |<t, s>|^2 / |t|^2.
// The 32 warps of a block share the columns of one or more aggregates (lane =
// row).  Bound by the latency of its barriers and of A_c's entries from L2
// (where every block's part fits, it stays in shared memory).  16^3 x 32, 4^4
// aggregates, 24 rows: 12.8 us an iteration, 4.3 of them the barriers, where
// nine kernels an iteration took 49 us.
// A_c larger than MGC_STREAM is read from HBM, and the chain from an aggregate's
// neighbours to its inputs to its product has to be covered: four blocks of 256
// threads an SM, each at its own place in the chain, and the next aggregate's
// matrix asked for ahead.  32^3 x 64 (340 MB): 165 us an
// iteration, against 226 with one block of 1024 (211 with four blocks but nothing
// asked for ahead) and 181 with nine kernels; 24^3 x 48 (108 MB): 70, 89 and 91.
// Aggregates with few rows are many and their matrices small: a block takes as
// many at a time as have the threads for their inputs (mgc_threads), and where a
// warp or two are left to each, the lanes share a row's columns as well (SPLIT).
// us an iteration, aggregates x rows: nine kernels / four (one when streamed) a
// block, lane = row / as now:
//   4096 x 4 (5 MB)     35 /  41 / 15        20736 x 8 (96 MB)    122 / 215 /  89
//   4096 x 8 (19 MB)    39 /  44 / 26        65536 x 4 (75 MB)    190 / 512 / 124
//   8192 x 8 (38 MB)    56 /  80 / 42         8192 x 16 (151 MB)  130 / 133 /  97
// (With a whole block an aggregate the shares are too many to sum: 128 x 8 11.0 ->
// 21.4 us, so SPLIT only comes with the fewest threads; with 24 rows one lane a
// row and 256 threads an aggregate are faster: 1296 x 24 34.7 us, 42.9 split and
// 37.5 with 128; 2592 x 24, streamed, 69, 76 and 74.)
constexpr int MGC_THREADS = 1024;
// below it the one large block is as fast (24^4, 54 MB: 35 us against 37; 16^2 x
// 24 x 32: 27 against 30), as the matrices stay in L2
constexpr size_t MGC_STREAM = (size_t)64 << 20;
constexpr int MGC_SMEM = 180 * 1024;  // the most a block's matrices may take of its shared memory
// the fewest threads an aggregate of nc rows takes: two of its 9 nc inputs each
int mgc_threads(int nc) {
  if (nc > 16) return 256;
  int t = 32;
  while (2 * t < 9 * nc) t *= 2;
  return t;
}
template <bool CACHED, int T, bool SPLIT>
__global__ void __launch_bounds__(T, MGC_THREADS / T) k_mg_coarse(CoarseArgs a) {
  constexpr bool STREAM = T < MGC_THREADS;
  extern __shared__ float4 ysm[];  // CACHED: the entries of the block's aggregates
  __shared__ float2 xin_all[2 * T];  // [aggregate][J]: at most two inputs a thread
  __shared__ float2 psum[T / 32][32];
  __shared__ int nb[T / 32][9];
  __shared__ GridRedShared red;
  __shared__ double tot[8];
  __shared__ double2 sc[5];  // alpha, omega, beta, beta omega, rho
  __shared__ int done;
  const int nc = a.m.nc, J = 9 * nc, P = J / 2;
  const int tpa = T / a.apb, wpa = tpa / 32;
  const int al = threadIdx.x / tpa, lt = threadIdx.x % tpa, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2 *const xin = xin_all + al * J;
  const int first = blockIdx.x * a.apb, stride = gridDim.x * a.apb;
  if (grid_red_failed(&a.st->red)) return;
  // SPLIT: lane = row + nc * (its share of the warp's columns); else lane = row
  const int groups = SPLIT ? 32 / nc : 1, grp = SPLIT ? lane / nc : 0, row = SPLIT ? lane - grp * nc : lane;
  const int parts = wpa * groups, share = (lt >> 5) * groups + grp;
  const int jp0 = share * P / parts, jp1 = (share + 1) * P / parts;
  // the (at most two, as J <= 2 tpa) inputs this thread stages: block d, row
  const int d0 = lt / nc, row0 = lt - d0 * nc, d1 = (lt + tpa) / nc, row1 = lt + tpa - d1 * nc;
  const unsigned count0 = a.st->red.base;
  unsigned epoch = 0;

  // A_c times the staged inputs at row lt < nc of aggregate B (every thread calls it)
  auto apply = [&](int B, bool mine) -> float2 {
    __syncthreads();
    if (mine && (SPLIT ? grp < groups : lane < nc))
      psum[warp][lane] = CACHED ? mg_row<true>(ysm + (size_t)al * P * nc + row, nc, xin, jp0, jp1)
                       : STREAM ? mg_row_wide<7>(a.Y + (size_t)B * P * nc + row, nc, xin, jp0, jp1)
                                : mg_row<false>(a.Y + (size_t)B * P * nc + row, nc, xin, jp0, jp1);
    __syncthreads();
    float2 o = make_float2(0.f, 0.f);
    if (mine && lt < nc)
      for (int w = 0; w < wpa; w++) {
        if constexpr (SPLIT) {
          for (int k = lt; k < groups * nc; k += nc)
            o = make_float2(o.x + psum[al * wpa + w][k].x, o.y + psum[al * wpa + w][k].y);
        } else {
          o = make_float2(o.x + psum[al * wpa + w][lt].x, o.y + psum[al * wpa + w][lt].y);
        }
      }
    return o;
  };
  auto neighbours = [&](int B) {
    if (B < a.m.nblocks && lt < 9) nb[al][lt] = mg_cnbr(a.m, B, lt);
  };
  // STREAM: has the matrix of the aggregate after B (of the next application,
  // after the last) fetched into L2 while B's inputs are formed and used
  auto prefetch = [&](int B) {
    const int Bn = B + stride < a.m.nblocks ? B + stride : first + al;
    if (STREAM && lt == tpa - 1 && Bn < a.m.nblocks)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.Y + (size_t)Bn * P * nc), "r"(P * nc * 16) : "memory");
  };

  double v1[1] = {0.0}, v2[2], v8[8];
  for (int base = first; base < a.m.nblocks; base += stride) {
    const int B = base + al;
    if (B < a.m.nblocks && lt < nc) {
      const float2 q = a.b[(size_t)B * nc + lt];
      a.x[(size_t)B * nc + lt] = make_float2(0.f, 0.f);
      v1[0] += (double)q.x * q.x + (double)q.y * q.y;
    }
  }
  if constexpr (CACHED) {
    const int n = min(a.apb, a.m.nblocks - first) * P * nc;
    for (int i = threadIdx.x; i < n; i += T) ysm[i] = __ldg(a.Y + (size_t)first * P * nc + i);
    neighbours(first + al);
  }
  bool ok = grid_allreduce<1>(&a.st->red, count0, ++epoch, v1, wpa, tot, red);
  if (!ok) return;
  const double bb = tot[0];
  int status = bb > 0 ? ST_RUNNING : ST_CONVERGED, it = 0;
  if (threadIdx.x == 0) {
    sc[0] = sc[1] = sc[2] = sc[3] = make_double2(0, 0);
    sc[4] = make_double2(bb, 0.0);  // <rt, r> with rt = r = b
  }
  for (; status == ST_RUNNING; it++) {
    const int cur = it & 1;
    float2 *rc = cur ? a.r1 : a.r0, *pc = cur ? a.p1 : a.p0, *vc = cur ? a.v1 : a.v0;
    const float2 *ro = cur ? a.r0 : a.r1, *po = cur ? a.p0 : a.p1, *vo = cur ? a.v0 : a.v1;
    __syncthreads();
    float ar = (float)sc[0].x, ai = (float)sc[0].y, wr = (float)sc[1].x, wi = (float)sc[1].y;
    const float br = (float)sc[2].x, bi = (float)sc[2].y, gr = (float)sc[3].x, gi = (float)sc[3].y;
    // p = r + beta (p - omega v), r the new residual s - omega t; v = A_c p; <rt, v>
    v2[0] = v2[1] = 0.0;
    for (int base = first; base < a.m.nblocks; base += stride) {
      const int B = base + al;
      const bool mine = B < a.m.nblocks;
      if constexpr (!CACHED) {
        __syncthreads();
        neighbours(B);
        prefetch(B);
        __syncthreads();
      }
      auto stage = [&](int i, int d, int row) {
        const size_t e = (size_t)nb[al][d] * nc + row;
        float2 rn, pn;
        if (it == 0) {
          rn = pn = a.b[e];
        } else {
          const float2 r = __ldcg(ro + e), q = __ldcg(vo + e), t = __ldcg(a.t + e), p = __ldcg(po + e);
          const float2 s = make_float2(r.x - ar * q.x + ai * q.y, r.y - ar * q.y - ai * q.x);
          rn = make_float2(s.x - wr * t.x + wi * t.y, s.y - wr * t.y - wi * t.x);
          pn = make_float2(rn.x + br * p.x - bi * p.y - gr * q.x + gi * q.y,
                           rn.y + br * p.y + bi * p.x - gr * q.y - gi * q.x);
          if (d == 8) {
            const float2 x = a.x[e];
            a.x[e] = make_float2(x.x + ar * p.x - ai * p.y + wr * s.x - wi * s.y,
                                 x.y + ar * p.y + ai * p.x + wr * s.y + wi * s.x);
          }
        }
        xin[i] = pn;
        if (d == 8) {
          rc[e] = rn;
          pc[e] = pn;
        }
      };
      if (mine && lt < J) stage(lt, d0, row0);
      if (mine && lt + tpa < J) stage(lt + tpa, d1, row1);
      const float2 o = apply(B, mine);
      if (mine && lt < nc) {
        const size_t e = (size_t)B * nc + lt;
        vc[e] = o;
        const float2 q = a.b[e];
        v2[0] += (double)q.x * o.x + (double)q.y * o.y;
        v2[1] += (double)q.x * o.y - (double)q.y * o.x;
      }
    }
    ok = grid_allreduce<2>(&a.st->red, count0, ++epoch, v2, wpa, tot, red);
    if (!ok) return;
    const double2 rtv = make_double2(tot[0], tot[1]);
    if (!(rtv.x * rtv.x + rtv.y * rtv.y > 0)) {
      status = ST_BREAKDOWN;
      break;
    }
    if (threadIdx.x == 0) sc[0] = cdiv2(sc[4], rtv);
    __syncthreads();
    ar = (float)sc[0].x, ai = (float)sc[0].y;
    // s = r - alpha v; t = A_c s; the products of t, s and rt
#pragma unroll
    for (int k = 0; k < 8; k++) v8[k] = 0.0;
    for (int base = first; base < a.m.nblocks; base += stride) {
      const int B = base + al;
      const bool mine = B < a.m.nblocks;
      if constexpr (!CACHED) {
        __syncthreads();
        neighbours(B);
        prefetch(B);
        __syncthreads();
      }
      auto stage = [&](int i, int d, int row) {
        const size_t e = (size_t)nb[al][d] * nc + row;
        const float2 r = __ldcg(rc + e), q = __ldcg(vc + e);
        xin[i] = make_float2(r.x - ar * q.x + ai * q.y, r.y - ar * q.y - ai * q.x);
      };
      if (mine && lt < J) stage(lt, d0, row0);
      if (mine && lt + tpa < J) stage(lt + tpa, d1, row1);
      const float2 o = apply(B, mine);
      if (mine && lt < nc) {
        const size_t e = (size_t)B * nc + lt;
        a.t[e] = o;
        const float2 s = xin[8 * nc + lt], q = a.b[e];
        v8[0] += (double)o.x * s.x + (double)o.y * s.y;  // <t, s>
        v8[1] += (double)o.x * s.y - (double)o.y * s.x;
        v8[2] += (double)o.x * o.x + (double)o.y * o.y;  // |t|^2
        v8[3] += (double)q.x * s.x + (double)q.y * s.y;  // <rt, s>
        v8[4] += (double)q.x * s.y - (double)q.y * s.x;
        v8[5] += (double)q.x * o.x + (double)q.y * o.y;  // <rt, t>
        v8[6] += (double)q.x * o.y - (double)q.y * o.x;
        v8[7] += (double)s.x * s.x + (double)s.y * s.y;  // |s|^2
      }
    }
    ok = grid_allreduce<8>(&a.st->red, count0, ++epoch, v8, wpa, tot, red);
    if (!ok) return;
    if (threadIdx.x == 0) {  // omega = 0 when t = 0 (then s = 0 too)
      const double it2 = tot[2] > 0 ? 1.0 / tot[2] : 0.0;
      const double2 w = make_double2(tot[0] * it2, tot[1] * it2);
      const double2 wt = cmul2(w, make_double2(tot[5], tot[6]));
      const double2 next = make_double2(tot[3] - wt.x, tot[4] - wt.y);
      const double rr = fmax(tot[7] - (tot[0] * tot[0] + tot[1] * tot[1]) * it2, 0.0);
      const double2 beta = cdiv2(cmul2(next, sc[0]), cmul2(sc[4], w));
      sc[1] = w;
      sc[2] = beta;
      sc[3] = cmul2(beta, w);
      sc[4] = next;
      done = !(tot[7] == tot[7]) || !(tot[2] == tot[2]) ? ST_NAN
             : rr <= a.tol2 * bb                         ? ST_CONVERGED
             : it + 1 >= a.maxit                         ? ST_MAXITER
             : !(next.x * next.x + next.y * next.y > 0) || !(w.x * w.x + w.y * w.y > 0) ? ST_BREAKDOWN
                                                                                        : ST_RUNNING;
    }
    __syncthreads();
    status = done;
    if (status != ST_RUNNING) {  // the last x += alpha p + omega s
      wr = (float)sc[1].x, wi = (float)sc[1].y;
      for (int base = first; base < a.m.nblocks; base += stride) {
        const int B = base + al;
        if (B < a.m.nblocks && lt < nc) {
          const size_t e = (size_t)B * nc + lt;
          const float2 r = __ldcg(rc + e), q = __ldcg(vc + e), p = __ldcg(pc + e), x = a.x[e];
          const float2 s = make_float2(r.x - ar * q.x + ai * q.y, r.y - ar * q.y - ai * q.x);
          a.x[e] = make_float2(x.x + ar * p.x - ai * p.y + wr * s.x - wi * s.y,
                               x.y + ar * p.y + ai * p.x + wr * s.y + wi * s.x);
        }
      }
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.st->status = status;
    a.st->total_it += it;
    grid_red_end(&a.st->red, count0, epoch);
  }
}

// ---------------------------------------------------------------- vector kernels
// out = a x + b y + c z (complex scalars; y, z may be null), n complex numbers
template <typename V>
__global__ void k_mg_lin3(int64_t n, V *out, double2 a, const V *x, double2 b, const V *y, double2 c, const V *z) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double xr = x[i].x, xi = x[i].y;
    double re = a.x * xr - a.y * xi, im = a.x * xi + a.y * xr;
    if (y) {
      const double yr = y[i].x, yi = y[i].y;
      re += b.x * yr - b.y * yi;
      im += b.x * yi + b.y * yr;
    }
    if (z) {
      const double zr = z[i].x, zi = z[i].y;
      re += c.x * zr - c.y * zi;
      im += c.x * zi + c.y * zr;
    }
    out[i].x = re;
    out[i].y = im;
  }
}
// per-block partials of Re<a,b>, Im<a,b>, |a|^2 (<a,b> = sum conj(a) b); behind
// them, whether a barrier of the coarse solves so far gave up
template <typename V>
__global__ void __launch_bounds__(MG_RED) k_mg_dots(int64_t n, const V *a, const V *b, const CState *cs, double *part) {
  __shared__ double sh[(MG_RED / 32) * 3];
  double v[3] = {0, 0, 0};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double ax = a[i].x, ay = a[i].y, bx = b[i].x, by = b[i].y;
    v[0] += ax * bx + ay * by;
    v[1] += ax * by - ay * bx;
    v[2] += ax * ax + ay * ay;
  }
  mg_block_sum<3>(v, sh);
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; k++) part[blockIdx.x * 3 + k] = v[k];
  if (blockIdx.x == 0 && threadIdx.x == 0) part[gridDim.x * 3] = cs->red.failed;
}
// the sums onto the solver state's sums (in block order, no host in between)
__global__ void __launch_bounds__(MG_RED) k_mg_dots_dev(int64_t n, const double2 *a, const double2 *b, SolverState *st,
                                                       double *partials) {
  double v[3] = {0, 0, 0};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 x = a[i], y = b[i];
    v[0] += x.x * y.x + x.y * y.y;
    v[1] += x.x * y.y - x.y * y.x;
    v[2] += x.x * x.x + x.y * x.y;
  }
  grid_reduce<3, MG_RED>(v, RedCtx{st, partials, FIN_STORE});
}
// an MR step with its multiple from the sums <q, s>, |q|^2: x += a s; s -= a q
// (nothing when q = 0, as s is then)
__global__ void k_mg_mr(int64_t n, double2 *x, double2 *s, const double2 *q, const SolverState *st) {
  const double qq = st->sums[2];
  if (!(qq > 0)) return;
  const double2 a = make_double2(st->sums[0] / qq, st->sums[1] / qq);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 ss = s[i], ww = q[i], xx = x[i];
    x[i] = make_double2(xx.x + a.x * ss.x - a.y * ss.y, xx.y + a.x * ss.y + a.y * ss.x);
    s[i] = make_double2(ss.x - a.x * ww.x + a.y * ww.y, ss.y - a.x * ww.y - a.y * ww.x);
  }
}
// x += a y; r -= a w (the GCR update in one pass)
__global__ void k_mg_axpy2(int64_t n, double2 *x, const double2 *y, double2 *r, const double2 *w, double2 a) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 yy = y[i], ww = w[i], xx = x[i], rr = r[i];
    x[i] = make_double2(xx.x + a.x * yy.x - a.y * yy.y, xx.y + a.x * yy.y + a.y * yy.x);
    r[i] = make_double2(rr.x - a.x * ww.x + a.y * ww.y, rr.y - a.x * ww.y - a.y * ww.x);
  }
}
// flexible GCR orthogonalisation, up to MG_CHUNK earlier directions per pass
constexpr int MG_CHUNK = 8;
struct Dirs {
  const double2 *p[MG_CHUNK];
  double2 c[MG_CHUNK];
};
// block partials of <W_i, w>, i < cnt: part[block * 2 MG_CHUNK + 2 i + (0 Re, 1 Im)]
__global__ void __launch_bounds__(MG_RED) k_mg_multidot(int64_t n, Dirs W, int cnt, const double2 *w, double *part) {
  __shared__ double sh[(MG_RED / 32) * 2 * MG_CHUNK];
  double v[2 * MG_CHUNK];
#pragma unroll
  for (int i = 0; i < 2 * MG_CHUNK; i++) v[i] = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const double2 b = w[e];
#pragma unroll
    for (int i = 0; i < MG_CHUNK; i++) {
      if (i < cnt) {
        const double2 a = W.p[i][e];
        v[2 * i] += a.x * b.x + a.y * b.y;
        v[2 * i + 1] += a.x * b.y - a.y * b.x;
      }
    }
  }
  mg_block_sum<2 * MG_CHUNK>(v, sh);
  if (threadIdx.x == 0)
    for (int i = 0; i < 2 * MG_CHUNK; i++) part[(size_t)blockIdx.x * 2 * MG_CHUNK + i] = v[i];
}
// out -= sum_{i < cnt} c_i W_i
__global__ void k_mg_multiaxpy(int64_t n, double2 *out, Dirs W, int cnt) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    double2 o = out[e];
#pragma unroll
    for (int i = 0; i < MG_CHUNK; i++) {
      if (i < cnt) {
        const double2 a = W.p[i][e], c = W.c[i];
        o.x -= c.x * a.x - c.y * a.y;
        o.y -= c.x * a.y + c.y * a.x;
      }
    }
    out[e] = o;
  }
}

// one parity (SOA64 half spinors, the Vh real sites only): block partials of
// <a, b>, |a|^2, and the same flag behind them
__global__ void __launch_bounds__(MG_RED) k_mg_half_dots(int Vh, const double2 *a, const double2 *b, const CState *cs,
                                                        double *part) {
  __shared__ double sh[(MG_RED / 32) * 3];
  double v[3] = {0, 0, 0};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (int64_t)Vh * 12;
       i += (int64_t)gridDim.x * blockDim.x) {
    const size_t k = hidx((int)(i / 12), (int)(i % 12));
    const double2 x = a[k], y = b[k];
    v[0] += x.x * y.x + x.y * y.y;
    v[1] += x.x * y.y - x.y * y.x;
    v[2] += x.x * x.x + x.y * x.y;
  }
  mg_block_sum<3>(v, sh);
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; k++) part[blockIdx.x * 3 + k] = v[k];
  if (blockIdx.x == 0 && threadIdx.x == 0) part[gridDim.x * 3] = cs->red.failed;
}
// z *= alpha; q = r - alpha q (one parity)
__global__ void k_mg_half_mr(int Vh, double2 *z, double2 *q, const double2 *r, double2 al) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (int64_t)Vh * 12;
       i += (int64_t)gridDim.x * blockDim.x) {
    const size_t k = hidx((int)(i / 12), (int)(i % 12));
    const double2 zz = z[k], qq = q[k], rr = r[k];
    z[k] = make_double2(al.x * zz.x - al.y * zz.y, al.x * zz.y + al.y * zz.x);
    q[k] = make_double2(rr.x - (al.x * qq.x - al.y * qq.y), rr.y - (al.x * qq.y + al.y * qq.x));
  }
}
// near-null vector k (FP32, aggregate-major) from a full FP64 vector
__global__ void __launch_bounds__(MG_MAXBLOCK) k_mg_store_nv(MGGeom m, int k, const double2 *v, float2 *nv) {
  const int B = blockIdx.x, t = threadIdx.x;
  const SiteC c = mg_site(m, B, t);
#pragma unroll
  for (int comp = 0; comp < 12; comp++) {
    const double2 a = v[fidx(m, c.par, c.s, comp)];
    nv[nidx(m, k, B, t, comp)] = make_float2((float)a.x, (float)a.y);
  }
}

int mg_grid(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + MG_RED - 1) / MG_RED, MG_RED_GRID));
}

}  // namespace

// ---------------------------------------------------------------- host
struct MG {
  GaugeHandle *G = nullptr;
  double kappa = 0;
  MGParams p;
  MGGeom m;
  int device = 0;
  DevBuf nv, Y;  // near-null vectors (FP32 full vectors), coarse operator (FP32)
  DevBuf part;   // reduction partials
  std::vector<double> part_h;
  // FP64 full vectors: b, x, r; s, q (the smoother); e1 (scratch of mg_check); tmp (one parity, A in)
  DevBuf b, x, r, e1, s, q, tmp;
  std::vector<std::unique_ptr<DevBuf>> Z, W;  // flexible GCR directions
  // coarse FP32 vectors
  DevBuf cb, cx, cr, cr2, cp, cp2, cv, cv2, ct;
  DevBuf cstate;                        // CState of the coarse solve
  double setup_seconds = 0;

  int64_t nfull() const { return (int64_t)2 * m.Vp * 12; }
  int64_t ncoarse() const { return (int64_t)m.nblocks * m.nc; }
};

namespace {

using C = Cpx<double>;
double2 *f64(DevBuf &d) { return d.as<double2>(); }
float2 *f32(DevBuf &d) { return d.as<float2>(); }
// the parity slabs of a full vector
FineVec slabs(const MG &mg, const double2 *v) {
  double2 *p = const_cast<double2 *>(v);
  return FineVec{{p, p + (size_t)mg.m.Vp * 12}};
}

// the sums of gr blocks' three partials, on the host; throws when the flag
// behind them says that a barrier gave up: nothing of the cycle is used then
void read_sums(MG &mg, cudaStream_t st, int gr, double out[3]) {
  QCU_CUDA(cudaMemcpyAsync(mg.part_h.data(), mg.part.p, ((size_t)gr * 3 + 1) * sizeof(double), cudaMemcpyDeviceToHost, st));
  QCU_CUDA(cudaStreamSynchronize(st));
  if (mg.part_h[(size_t)gr * 3] != 0.0) throw Error(2, "mg: a barrier of the coarse solve timed out");
  out[0] = out[1] = out[2] = 0;
  for (int i = 0; i < gr; i++)
    for (int k = 0; k < 3; k++) out[k] += mg.part_h[(size_t)i * 3 + k];
}
template <typename V>
void dots(MG &mg, cudaStream_t st, int64_t n, const V *a, const V *b, double out[3]) {
  const int gr = mg_grid(n);
  k_mg_dots<V><<<gr, MG_RED, 0, st>>>(n, a, b, mg.cstate.as<CState>(), mg.part.as<double>());
  QCU_CHECK_LAUNCH();
  read_sums(mg, st, gr, out);
}

template <typename V>
void lin3(cudaStream_t st, int64_t n, V *out, C a, const V *x, C b = C(0, 0), const V *y = nullptr, C c = C(0, 0),
          const V *z = nullptr) {
  k_mg_lin3<V><<<mg_grid(n), MG_RED, 0, st>>>(n, out, make_double2(a.re, a.im), x, make_double2(b.re, b.im), y,
                                             make_double2(c.re, c.im), z);
  QCU_CHECK_LAUNCH();
}

// out = M in on full FP64 vectors: out_p = A_p in_p - kappa D_{p <- 1-p} in_{1-p};
// dots: also <out, in> and |out|^2 in the solver state's sums[0..2] (from the
// two hops themselves without a clover term, whose epilogue holds both vectors:
// 16^3 x 32, an MR step 62 us without a word to the host; dots of their own took
// 59 us of kernels and the round trip between them)
void mat(MG &mg, Context &ctx, const double2 *in, double2 *out, bool dots = false) {
  const GaugeHandle &G = *mg.G;
  const size_t half = (size_t)mg.m.Vp * 12;
  for (int p = 0; p < 2; p++) {
    DslashArgs d;
    d.gauge = G.g64.p;
    d.t_bc = G.t_bc;
    d.a = -mg.kappa;
    d.b1 = 1.0;
    d.in = in + (1 - p) * half;
    d.out = out + p * half;
    d.parity = p;
    if (G.has_clover) {
      launch_clover_apply(SOA64, G.g.Vh, G.A64[p].p, in + p * half, mg.tmp.p, ctx.stream);
      d.x1 = mg.tmp.p;
    } else {
      d.x1 = in + p * half;
      if (dots) {
        d.red = RED_TS_TT;
        d.fin = p ? FIN_ADD : FIN_STORE;
      }
    }
    launch_dslash(SOA64, GSOA64, CSOA64, G.g, d, ctx, ctx.stream);
  }
  if (dots && G.has_clover) {
    k_mg_dots_dev<<<mg_grid(mg.nfull()), MG_RED, 0, ctx.stream>>>(mg.nfull(), out, in, ctx.st, ctx.partials);
    QCU_CHECK_LAUNCH();
  }
}

int capply_grid(const MG &mg) { return (mg.m.nblocks + CAPPLY_WARPS - 1) / CAPPLY_WARPS; }

// out = b - M e on full FP64 vectors in one dslash pass per parity:
// out_p = kappa D_{p <- 1-p} e_{1-p} + b_p - A_p e_p
void residual(MG &mg, Context &ctx, const double2 *e, const double2 *b, double2 *out) {
  const GaugeHandle &G = *mg.G;
  const size_t half = (size_t)mg.m.Vp * 12;
  for (int p = 0; p < 2; p++) {
    DslashArgs d;
    d.gauge = G.g64.p;
    d.t_bc = G.t_bc;
    d.a = mg.kappa;
    d.in = e + (1 - p) * half;
    d.out = out + p * half;
    d.parity = p;
    d.x1 = b + p * half;
    d.b1 = 1.0;
    if (G.has_clover) {
      launch_clover_apply(SOA64, G.g.Vh, G.A64[p].p, e + p * half, mg.tmp.p, ctx.stream);
      d.x2 = mg.tmp.p;
    } else {
      d.x2 = e + p * half;
    }
    d.b2 = -1.0;
    launch_dslash(SOA64, GSOA64, CSOA64, G.g, d, ctx, ctx.stream);
  }
}

// out = A_c in
void capply(MG &mg, cudaStream_t st, const float2 *in, float2 *out) {
  k_mg_capply<<<capply_grid(mg), 32 * CAPPLY_WARPS, 0, st>>>(mg.m, mg.Y.as<float4>(), in, out);
  QCU_CHECK_LAUNCH();
}

// cx ~ A_c^-1 cb on the device
void coarse_solve(MG &mg, Context &ctx) {
  CoarseArgs a;
  a.m = mg.m;
  a.Y = mg.Y.as<float4>();
  a.b = f32(mg.cb);
  a.x = f32(mg.cx);
  a.r0 = f32(mg.cr);
  a.r1 = f32(mg.cr2);
  a.p0 = f32(mg.cp);
  a.p1 = f32(mg.cp2);
  a.v0 = f32(mg.cv);
  a.v1 = f32(mg.cv2);
  a.t = f32(mg.ct);
  a.st = mg.cstate.as<CState>();
  a.tol2 = mg.p.coarse_tol * mg.p.coarse_tol;
  a.maxit = mg.p.coarse_maxiter;
  const size_t part = (size_t)(9 * a.m.nc / 2) * a.m.nc * sizeof(float4);  // of A_c, an aggregate's
  const bool stream = part * mg.m.nblocks > MGC_STREAM;
  const int T = stream ? 256 : MGC_THREADS, per = MGC_THREADS / T, fewest = mgc_threads(a.m.nc);
  // spread the aggregates over the SMs before a block takes several at a time
  a.apb = stream ? T / fewest : 1;
  while (!stream && a.apb * ctx.sms < mg.m.nblocks && T / (2 * a.apb) >= fewest) a.apb *= 2;
  const bool split = T / a.apb == fewest && a.m.nc <= 16;
  const int grid = std::min(std::min(per * ctx.sms, GRID_RED_BLOCKS), (mg.m.nblocks + a.apb - 1) / a.apb);
  // A_c stays in shared memory where every block has one set of aggregates that fits
  const size_t smem = a.apb * part;
  const bool cached = !stream && smem <= MGC_SMEM && (int64_t)grid * a.apb >= a.m.nblocks;
  auto pick = [&](auto plain, auto shared_out) {
    return split ? reinterpret_cast<const void *>(shared_out) : reinterpret_cast<const void *>(plain);
  };
  const void *k = stream   ? pick(k_mg_coarse<false, 256, false>, k_mg_coarse<false, 256, true>)
                  : cached ? pick(k_mg_coarse<true, MGC_THREADS, false>, k_mg_coarse<true, MGC_THREADS, true>)
                           : pick(k_mg_coarse<false, MGC_THREADS, false>, k_mg_coarse<false, MGC_THREADS, true>);
  if (cached) QCU_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, MGC_SMEM));
  void *args[] = {&a};
  QCU_CUDA(grid_red_inject(&a.st->red, "coarse", ctx.stream));
  QCU_CUDA(cudaLaunchCooperativeKernel(k, dim3(grid), dim3(T), args, cached ? smem : 0, ctx.stream));
  note_launch(1);
}

constexpr size_t CSTATE_HEAD = offsetof(CState, red) + offsetof(GridRed, part);

// the iterations of the coarse solves since the last reset, on the host
long long coarse_iterations(MG &mg, cudaStream_t st) {
  CState cs;
  QCU_CUDA(cudaMemcpyAsync(&cs, mg.cstate.p, CSTATE_HEAD, cudaMemcpyDeviceToHost, st));
  QCU_CUDA(cudaStreamSynchronize(st));
  return cs.total_it;
}

void axpy2(cudaStream_t st, int64_t n, double2 *x, const double2 *y, double2 *r, const double2 *w, C a) {
  k_mg_axpy2<<<mg_grid(n), MG_RED, 0, st>>>(n, x, y, r, w, make_double2(a.re, a.im));
  QCU_CHECK_LAUNCH();
}

// steps MR iterations on M e = r from e (start: s = r - M e, or s = r when
// e = 0); s = r - M e on return
void smooth(MG &mg, Context &ctx, const double2 *r, double2 *e, int steps, bool e_zero) {
  cudaStream_t st = ctx.stream;
  const int64_t n = mg.nfull();
  double2 *s = f64(mg.s), *q = f64(mg.q);
  if (e_zero) {
    QCU_CUDA(cudaMemsetAsync(e, 0, (size_t)n * sizeof(double2), st));
    QCU_CUDA(cudaMemcpyAsync(s, r, (size_t)n * sizeof(double2), cudaMemcpyDeviceToDevice, st));
  } else {
    residual(mg, ctx, e, r, s);
  }
  for (int k = 0; k < steps; k++) {
    mat(mg, ctx, s, q, true);  // with <M s, s>, |M s|^2
    k_mg_mr<<<mg_grid(n), MG_RED, 0, st>>>(n, e, s, q, ctx.st);
    QCU_CHECK_LAUNCH();
  }
}

// e = K r: nu_pre MR steps, the coarse correction, nu_post MR steps
void cycle(MG &mg, Context &ctx, const double2 *r, double2 *e) {
  cudaStream_t st = ctx.stream;
  const MGGeom &m = mg.m;
  const int64_t n = mg.nfull();
  const float2 *nv = mg.nv.as<float2>();
  const double2 *rc = r;  // the residual the coarse grid sees
  if (mg.p.nu_pre > 0) {
    smooth(mg, ctx, r, e, mg.p.nu_pre, true);
    rc = f64(mg.s);  // r - M e
  }
  k_mg_restrict<<<m.nblocks, m.bsites, 0, st>>>(m, nv, slabs(mg, rc), f32(mg.cb));
  QCU_CHECK_LAUNCH();
  coarse_solve(mg, ctx);
  k_mg_prolong<<<m.nblocks, m.bsites, 0, st>>>(m, nv, f32(mg.cx), slabs(mg, e), mg.p.nu_pre > 0 ? 1 : 0);
  QCU_CHECK_LAUNCH();
  if (mg.p.nu_post > 0) smooth(mg, ctx, r, e, mg.p.nu_post, false);
}

}  // namespace

MG *mg_create(GaugeHandle &G, double kappa, const MGParams &p) {
  const auto t0 = std::chrono::steady_clock::now();
  require(kappa > 0, "mg: kappa must be positive");
  require(p.n_vec >= 1 && p.n_vec <= MG_MAXVEC, "mg: n_vec must be 1.." + std::to_string(MG_MAXVEC));
  require(p.gcr_k >= 1 && p.gcr_k <= 32, "mg: gcr_k must be 1..32");
  require(p.nu_pre >= 0 && p.nu_post >= 0 && p.coarse_maxiter >= 1 && p.setup_maxiter >= 1 && p.coarse_tol > 0,
          "mg: nu_pre, nu_post >= 0, coarse_maxiter, setup_maxiter >= 1 and coarse_tol > 0 are required");
  auto mg = std::make_unique<MG>();
  mg->G = &G;
  mg->kappa = kappa;
  mg->p = p;
  MGGeom &m = mg->m;
  for (int d = 0; d < 4; d++) {
    m.L[d] = G.latt[d];
    m.b[d] = p.geo_block_size[d];
    require(m.b[d] >= 1 && m.L[d] % m.b[d] == 0, "mg: every block extent must divide the lattice extent");
    m.nb[d] = m.L[d] / m.b[d];
  }
  require(m.b[0] % 2 == 0, "mg: the x block extent must be even");
  m.nblocks = m.nb[0] * m.nb[1] * m.nb[2] * m.nb[3];
  m.bsites = m.b[0] * m.b[1] * m.b[2] * m.b[3];
  require(m.bsites % 32 == 0 && m.bsites <= MG_MAXBLOCK,
          "mg: sites per block must be a multiple of 32 and at most " + std::to_string(MG_MAXBLOCK));
  m.Vh = G.g.Vh;
  m.Vp = pad_sites(G.g.Vh);
  m.nvec = p.n_vec;
  m.nc = 2 * p.n_vec;
  const int Vh = m.Vh;
  const int clov = G.has_clover ? 1 : 0;
  Context &ctx = context();
  mg->device = ctx.device;
  {
    std::lock_guard<std::mutex> lk(ctx.mu);
    const size_t full = (size_t)mg->nfull() * sizeof(double2);
    const size_t cfull = (size_t)mg->ncoarse() * sizeof(float2);
    mg->nv.ensure((size_t)m.nvec * mg->nfull() * sizeof(float2));
    mg->Y.ensure((size_t)m.nblocks * 9 * m.nc * m.nc * sizeof(float2));
    mg->part.ensure((size_t)MG_RED_GRID * 2 * MG_CHUNK * sizeof(double));
    mg->cstate.ensure(sizeof(CState));
    QCU_CUDA(cudaMemsetAsync(mg->cstate.p, 0, sizeof(CState), ctx.stream));
    mg->part_h.resize((size_t)MG_RED_GRID * 2 * MG_CHUNK);
    for (DevBuf *d : {&mg->b, &mg->x, &mg->r, &mg->e1, &mg->s, &mg->q}) d->ensure(full);
    mg->tmp.ensure(full / 2);
    for (int k = 0; k < p.gcr_k; k++) {
      mg->Z.emplace_back(new DevBuf);
      mg->W.emplace_back(new DevBuf);
      mg->Z.back()->ensure(full);
      mg->W.back()->ensure(full);
    }
    for (DevBuf *d : {&mg->cb, &mg->cx, &mg->cr, &mg->cr2, &mg->cp, &mg->cp2, &mg->cv, &mg->cv2, &mg->ct})
      d->ensure(cfull);
    // the padding sites of the full vectors stay zero throughout
    for (DevBuf *d : {&mg->b, &mg->x, &mg->r, &mg->e1, &mg->s, &mg->q}) QCU_CUDA(cudaMemsetAsync(d->p, 0, full, ctx.stream));
    for (int k = 0; k < p.gcr_k; k++) {
      QCU_CUDA(cudaMemsetAsync(mg->Z[k]->p, 0, full, ctx.stream));
      QCU_CUDA(cudaMemsetAsync(mg->W[k]->p, 0, full, ctx.stream));
    }
    QCU_CUDA(cudaMemsetAsync(mg->nv.p, 0, mg->nv.n, ctx.stream));
    QCU_CUDA(cudaStreamSynchronize(ctx.stream));
  }
  // near-null vectors: v = v0 - y, y a short solve of M y = M v0 (PyQuda-layout buffers)
  {
    const size_t half_pyq = spinor_bytes(AOS64, Vh);
    DevBuf v0, bq, yq;
    {
      std::lock_guard<std::mutex> lk(ctx.mu);
      v0.ensure(2 * half_pyq);
      bq.ensure(2 * half_pyq);
      yq.ensure(2 * half_pyq);
    }
    SolveParams sp;
    sp.kappa = kappa;
    sp.tol = 1e-30;  // never met: the solve stops after setup_maxiter iterations
    sp.maxiter = p.setup_maxiter;
    sp.precision = 32;
    sp.solver = 0;
    sp.use_clover = clov;
    for (int k = 0; k < m.nvec; k++) {
      {
        std::lock_guard<std::mutex> lk(ctx.mu);
        launch_fermion_random(v0.p, (int64_t)Vh * 24, 0, 0x6d670000ULL + 7919ULL * (k + 1), ctx.stream);
        QCU_CUDA(cudaStreamSynchronize(ctx.stream));
      }
      handle_mat(G, bq.p, v0.p, kappa, clov);
      solve(G, yq.p, bq.p, sp);
      std::lock_guard<std::mutex> lk(ctx.mu);
      cudaStream_t st = ctx.stream;
      double2 *vf = f64(mg->b), *yf = f64(mg->x);
      const size_t half = (size_t)m.Vp * 12;
      for (int par = 0; par < 2; par++) {
        launch_convert(AOS64, SOA64, Vh, static_cast<char *>(v0.p) + par * half_pyq, nullptr, vf + par * half,
                       nullptr, st);
        launch_convert(AOS64, SOA64, Vh, static_cast<char *>(yq.p) + par * half_pyq, nullptr, yf + par * half,
                       nullptr, st);
      }
      const int64_t n = mg->nfull();
      lin3(st, n, vf, C(1, 0), vf, C(-1, 0), yf);
      k_mg_store_nv<<<m.nblocks, m.bsites, 0, st>>>(m, k, vf, mg->nv.as<float2>());
      QCU_CHECK_LAUNCH();
      QCU_CUDA(cudaStreamSynchronize(st));
    }
  }
  std::lock_guard<std::mutex> lk(ctx.mu);
  cudaStream_t st = ctx.stream;
  k_mg_orth<<<m.nblocks, m.bsites, 0, st>>>(m, mg->nv.as<float2>());
  QCU_CHECK_LAUNCH();
  const CloverView<CSOA64> A0{clov ? G.A64[0].p : nullptr, Vh}, A1{clov ? G.A64[1].p : nullptr, Vh};
  k_mg_build<<<m.nblocks, m.bsites, 0, st>>>(m, GaugeView<GSOA64>{G.g64.p, m.Vp}, A0, A1, clov, G.t_bc, kappa,
                                             mg->nv.as<float2>(), mg->Y.as<float2>());
  QCU_CHECK_LAUNCH();
  QCU_CUDA(cudaStreamSynchronize(st));
  mg->setup_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  return mg.release();
}

void mg_free(MG *mg) { delete mg; }

void mg_require_compatible(const MG &mg, const GaugeHandle &G, double kappa, int use_clover) {
  require(mg.G == &G, "mg: the multigrid was built on another gauge handle");
  require(mg.kappa == kappa, "mg: the multigrid was built for another kappa");
  require((use_clover != 0) == G.has_clover,
          "mg: the multigrid's operator includes the handle's clover term exactly when it has one");
  require(context().device == mg.device, "mg: the multigrid was set up on another device");
}

void mg_coarse_odd(MG &mg, Context &ctx, const void *r_odd, void *z_odd) {
  cudaStream_t st = ctx.stream;
  const MGGeom &m = mg.m;
  const GaugeHandle &G = *mg.G;
  const double2 *src = static_cast<const double2 *>(r_odd);
  if (G.has_clover) {  // M_pc = A_o^-1 S: S^-1 acts on A_o r
    launch_clover_apply(SOA64, G.g.Vh, G.A64[1].p, r_odd, mg.tmp.p, st);
    src = mg.tmp.as<double2>();
  }
  const float2 *nv = mg.nv.as<float2>();
  k_mg_restrict<<<m.nblocks, m.bsites, 0, st>>>(m, nv, FineVec{{nullptr, const_cast<double2 *>(src)}},
                                                f32(mg.cb));
  QCU_CHECK_LAUNCH();
  coarse_solve(mg, ctx);
  k_mg_prolong<<<m.nblocks, m.bsites, 0, st>>>(m, nv, f32(mg.cx), FineVec{{nullptr, static_cast<double2 *>(z_odd)}},
                                               0);
  QCU_CHECK_LAUNCH();
}

double2 mg_minres_scale(MG &mg, Context &ctx, void *z, void *q, const void *r) {
  cudaStream_t st = ctx.stream;
  const int Vh = mg.m.Vh;
  const int gr = mg_grid((int64_t)Vh * 12);
  k_mg_half_dots<<<gr, MG_RED, 0, st>>>(Vh, static_cast<const double2 *>(q), static_cast<const double2 *>(r),
                                        mg.cstate.as<CState>(), mg.part.as<double>());
  QCU_CHECK_LAUNCH();
  double d[3];
  read_sums(mg, st, gr, d);
  const double2 al = d[2] > 0 ? make_double2(d[0] / d[2], d[1] / d[2]) : make_double2(0, 0);
  k_mg_half_mr<<<gr, MG_RED, 0, st>>>(Vh, static_cast<double2 *>(z), static_cast<double2 *>(q),
                                      static_cast<const double2 *>(r), al);
  QCU_CHECK_LAUNCH();
  return al;
}

void mg_reset_coarse(MG &mg, Context &ctx) { QCU_CUDA(cudaMemsetAsync(mg.cstate.p, 0, CSTATE_HEAD, ctx.stream)); }

double mg_setup_seconds(const MG &mg) { return mg.setup_seconds; }

MGInfo mg_solve(MG &mg, void *x_pyq, const void *b_pyq, double tol, int maxiter) {
  require(x_pyq != nullptr && b_pyq != nullptr, "mg: null spinor pointer");
  require(tol > 0 && maxiter > 0, "mg: tol and maxiter must be positive");
  const auto t0 = std::chrono::steady_clock::now();
  Context &ctx = context();
  require(ctx.device == mg.device, "mg: the multigrid was set up on another device");
  std::lock_guard<std::mutex> lk(ctx.mu);
  QCU_CUDA(cudaDeviceSynchronize());  // inputs written on any stream are complete
  cudaStream_t st = ctx.stream;
  const MGGeom &m = mg.m;
  const int Vh = m.Vh;
  const size_t half = (size_t)m.Vp * 12, half_pyq = spinor_bytes(AOS64, Vh);
  const int64_t n = mg.nfull();
  double2 *b = f64(mg.b), *x = f64(mg.x), *r = f64(mg.r);
  for (int par = 0; par < 2; par++)
    launch_convert(AOS64, SOA64, Vh, static_cast<const char *>(b_pyq) + par * half_pyq, nullptr, b + par * half,
                   nullptr, st);
  QCU_CUDA(cudaMemsetAsync(x, 0, (size_t)n * sizeof(double2), st));
  QCU_CUDA(cudaMemcpyAsync(r, b, (size_t)n * sizeof(double2), cudaMemcpyDeviceToDevice, st));
  MGInfo info;
  mg_reset_coarse(mg, ctx);
  double d[3];
  dots(mg, st, n, b, b, d);
  const double bb = d[2];
  if (bb == 0.0) {
    QCU_CUDA(cudaMemsetAsync(x_pyq, 0, 2 * half_pyq, st));
    QCU_CUDA(cudaStreamSynchronize(st));
    info.status = ST_CONVERGED;
    return info;
  }
  const double target = tol * tol * bb;
  double rr = bb;
  std::vector<double> nw(mg.p.gcr_k);  // |w_j|^2
  info.status = ST_MAXITER;
  while (info.outer < maxiter) {
    for (int j = 0; j < mg.p.gcr_k && info.outer < maxiter; j++) {
      double2 *z = f64(*mg.Z[j]), *w = f64(*mg.W[j]);
      cycle(mg, ctx, r, z);
      mat(mg, ctx, z, w);
      // w_j -= sum_i <w_i, w_j> / |w_i|^2 w_i, z_j likewise; in chunks of
      // MG_CHUNK directions (Gram-Schmidt by blocks)
      for (int i0 = 0; i0 < j; i0 += MG_CHUNK) {
        const int cnt = std::min(MG_CHUNK, j - i0);
        Dirs Wd{}, Zd{};
        for (int i = 0; i < cnt; i++) {
          Wd.p[i] = f64(*mg.W[i0 + i]);
          Zd.p[i] = f64(*mg.Z[i0 + i]);
        }
        const int gr = mg_grid(n);
        k_mg_multidot<<<gr, MG_RED, 0, st>>>(n, Wd, cnt, w, mg.part.as<double>());
        QCU_CHECK_LAUNCH();
        QCU_CUDA(cudaMemcpyAsync(mg.part_h.data(), mg.part.p, (size_t)gr * 2 * MG_CHUNK * sizeof(double),
                                 cudaMemcpyDeviceToHost, st));
        QCU_CUDA(cudaStreamSynchronize(st));
        for (int i = 0; i < cnt; i++) {
          double re = 0, im = 0;
          for (int b = 0; b < gr; b++) {
            re += mg.part_h[(size_t)b * 2 * MG_CHUNK + 2 * i];
            im += mg.part_h[(size_t)b * 2 * MG_CHUNK + 2 * i + 1];
          }
          Wd.c[i] = Zd.c[i] = make_double2(re / nw[i0 + i], im / nw[i0 + i]);
        }
        k_mg_multiaxpy<<<mg_grid(n), MG_RED, 0, st>>>(n, w, Wd, cnt);
        QCU_CHECK_LAUNCH();
        k_mg_multiaxpy<<<mg_grid(n), MG_RED, 0, st>>>(n, z, Zd, cnt);
        QCU_CHECK_LAUNCH();
      }
      dots(mg, st, n, w, r, d);  // <w, r>, |w|^2
      if (!(d[2] > 0) || !(d[0] == d[0]) || !(d[1] == d[1])) {
        info.status = d[2] == d[2] ? ST_BREAKDOWN : ST_NAN;
        break;
      }
      nw[j] = d[2];
      axpy2(st, n, x, z, r, w, C(d[0] / d[2], d[1] / d[2]));  // alpha = <w, r> / |w|^2
      info.outer++;
      rr = std::max(0.0, rr - (d[0] * d[0] + d[1] * d[1]) / d[2]);  // |r - alpha w|^2; the restart recomputes it
      if (rr <= target) break;
    }
    if (info.status == ST_BREAKDOWN || info.status == ST_NAN) break;
    // restart from the FP64 true residual
    residual(mg, ctx, x, b, r);
    dots(mg, st, n, r, r, d);
    rr = d[2];
    if (rr <= target) {
      info.status = ST_CONVERGED;
      break;
    }
  }
  if (info.status == ST_BREAKDOWN || info.status == ST_NAN) {
    residual(mg, ctx, x, b, r);
    dots(mg, st, n, r, r, d);
    rr = d[2];
  }
  info.true_residual = std::sqrt(rr / bb);
  info.coarse_iters = (int)std::min<long long>(coarse_iterations(mg, st), 0x7fffffff);
  for (int par = 0; par < 2; par++)
    launch_convert(SOA64, AOS64, Vh, x + par * half, nullptr, static_cast<char *>(x_pyq) + par * half_pyq, nullptr,
                   st);
  QCU_CUDA(cudaStreamSynchronize(st));
  info.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  return info;
}

void mg_check(MG &mg, double *orth_err, double *galerkin_err) {
  Context &ctx = context();
  require(ctx.device == mg.device, "mg: the multigrid was set up on another device");
  std::lock_guard<std::mutex> lk(ctx.mu);
  cudaStream_t st = ctx.stream;
  mg_reset_coarse(mg, ctx);
  const MGGeom &m = mg.m;
  const int64_t nc = mg.ncoarse();
  // a seeded coarse vector, uniform in [-1, 1) (xorshift64)
  std::vector<float2> hc((size_t)nc);
  uint64_t z = 0x9e3779b97f4a7c15ULL;
  auto next = [&z]() {
    z ^= z << 13;
    z ^= z >> 7;
    z ^= z << 17;
    return (float)((double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0);
  };
  for (auto &v : hc) {
    v.x = next();
    v.y = next();
  }
  float2 *c0 = f32(mg.cb), *c1 = f32(mg.cx), *c2 = f32(mg.cr);
  QCU_CUDA(cudaMemcpyAsync(c0, hc.data(), (size_t)nc * sizeof(float2), cudaMemcpyHostToDevice, st));
  double2 *e = f64(mg.e1), *q = f64(mg.q);
  const float2 *nv = mg.nv.as<float2>();
  double d[3], d0[3];
  // P^dag P c against c
  k_mg_prolong<<<m.nblocks, m.bsites, 0, st>>>(m, nv, c0, slabs(mg, e), 0);
  QCU_CHECK_LAUNCH();
  k_mg_restrict<<<m.nblocks, m.bsites, 0, st>>>(m, nv, slabs(mg, e), c1);
  QCU_CHECK_LAUNCH();
  lin3(st, nc, c1, C(1, 0), c1, C(-1, 0), c0);
  dots(mg, st, nc, c1, c1, d);
  dots(mg, st, nc, c0, c0, d0);
  *orth_err = std::sqrt(d[2] / d0[2]);
  // A_c c against P^dag M P c
  mat(mg, ctx, e, q);
  k_mg_restrict<<<m.nblocks, m.bsites, 0, st>>>(m, nv, slabs(mg, q), c1);
  QCU_CHECK_LAUNCH();
  capply(mg, st, c0, c2);
  dots(mg, st, nc, c1, c1, d0);
  lin3(st, nc, c2, C(1, 0), c2, C(-1, 0), c1);
  dots(mg, st, nc, c2, c2, d);
  *galerkin_err = std::sqrt(d[2] / d0[2]);
}

}  // namespace qcu
