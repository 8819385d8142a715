// The GCR's inner solve (BiCGSTAB on 16-bit spinors and links) on a small
// lattice, as one cooperative kernel.
//
// With a few thousand sites per parity every kernel of an iteration takes its
// minimum of 2-7 us, and ten of them, with the gaps between, took 51 us at
// 8^3 x 16 for little memory traffic: the time is latency, of launches and of
// the eight hops that one thread takes one after the other.  Here
//   * a block takes 32 sites with eight warps, a hop each (lane = site, so
//     every access stays contiguous); two of them then sum the hops from shared
//     memory, one per chirality, apply that chirality's clover block and store;
//   * the blocks stay, with a grid barrier where neighbours exchange, four an
//     iteration:
//       tmp = A_e^-1 D p | v = p - k^2 A_o^-1 D tmp, <rt, v> |
//       tmp = A_e^-1 D s | t = s - k^2 A_o^-1 D tmp and its products |
//     p and s are never waited for: a hop forms its neighbour's
//       s = r - alpha v,   p = r - (alpha + beta omega) v - omega t + beta p
//     from the vectors before the update (r and p therefore alternate between
//     two buffers), while two other warps update the block's own x, r and p;
//   * <rt, r> = <rt, s> - omega <rt, t> and |r|^2 = |s|^2 - |<t, s>|^2 / |t|^2
//     of the new residual come with the second product's sums: FP64 sums of FP64
//     products with t as it is stored, since the differences round relative to
//     |s|^2 and not to |r|^2.  They hold where one iteration takes |s|^2 down by
//     less than about 1e15 (beyond, fmax makes |r|^2 zero and the solve ends); the
//     rounding of t to 16 bits alone leaves |r|^2 at some 1e-11 |s|^2.
// Vectors are stored in 16 bits and computed in FP32, sums in FP64, as in the
// kernels of dslash.cu and blas.cu.  A whole solve's time per inner iteration,
// outer steps included, 24 systems each, with the graph of kernels -> with this one:
//                with the clover term      without
//   8^3 x 16     57.4 -> 34.4 us           55.0 -> 33.3 us
//   12^2 x 8 x 16  57.7 -> 43.4            55.5 -> 41.8
//   12^3 x 16    59.4 -> 53.0              57.0 -> 50.1    (three tiles an SM)
// at 16^4 it would rise from 66 to 91 us, seven tiles a block one after the other,
// so the graph of kernels keeps more than three tiles an SM.  (FP32 products in the
// sums: 33.9 us at 8^3 x 16 with the clover term.)
#include <algorithm>

#include "gridbar.cuh"
#include "internal.h"

namespace qcu {
namespace {

constexpr int IS_THREADS = 256;
using CF = Cpx<float>;
constexpr float F16 = 1.0f / FIX16_SCALE;

// the 12 words of a site, or the 6 of one chirality, and its norm, from L2 (written by this kernel)
struct Raw12 {
  unsigned w[12];
  float n;
};
__device__ __forceinline__ void raw12(const void *p, const float *n, int s, Raw12 &o) {
  const char *b = static_cast<const char *>(p);
  const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(b + s16_w8(s))), y = __ldcg(reinterpret_cast<const uint4 *>(b + s16_w8(s)) + 1),
              z = __ldcg(reinterpret_cast<const uint4 *>(b + s16_w4(s)));
  o.w[0] = x.x, o.w[1] = x.y, o.w[2] = x.z, o.w[3] = x.w, o.w[4] = y.x, o.w[5] = y.y, o.w[6] = y.z, o.w[7] = y.w;
  o.w[8] = z.x, o.w[9] = z.y, o.w[10] = z.z, o.w[11] = z.w;
  o.n = __ldcg(n + s) * F16;
}
struct Raw6 {
  unsigned w[6];
  float n;
};
__device__ __forceinline__ void raw6(const void *p, const float *n, int s, int q, Raw6 &o) {
  const char *b = static_cast<const char *>(p);
  const uint2 u = __ldcg(reinterpret_cast<const uint2 *>(b + s16_w8(s) + (q ? 24 : 16)));
  const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(b + (q ? s16_w4(s) : s16_w8(s))));
  if (q) o.w[0] = u.x, o.w[1] = u.y, o.w[2] = x.x, o.w[3] = x.y, o.w[4] = x.z, o.w[5] = x.w;
  else o.w[0] = x.x, o.w[1] = x.y, o.w[2] = x.z, o.w[3] = x.w, o.w[4] = u.x, o.w[5] = u.y;
  o.n = __ldcg(n + s) * F16;
}
// component spin * 3 + colour (of the chirality) from words 2 * colour + (re, im)
template <int N, typename R>
__device__ __forceinline__ void decode(const R &r, CF (&v)[N]) {
#pragma unroll
  for (int q = 0; q < N / 6; q++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float2 re = fix16_unpack(r.w[6 * q + 2 * c]), im = fix16_unpack(r.w[6 * q + 2 * c + 1]);
      v[6 * q + c] = CF(re.x * r.n, im.x * r.n);
      v[6 * q + 3 + c] = CF(re.y * r.n, im.y * r.n);
    }
}
// v += a r
template <int N, typename R>
__device__ __forceinline__ void add_scaled(CF (&v)[N], CF a, const R &r) {
  CF f[N];
  decode(r, f);
#pragma unroll
  for (int k = 0; k < N; k++) {
    v[k].re = fmaf(a.re, f[k].re, fmaf(-a.im, f[k].im, v[k].re));
    v[k].im = fmaf(a.re, f[k].im, fmaf(a.im, f[k].re, v[k].im));
  }
}

// 16-bit store of one site by two warps (q = chirality): the site's largest
// component over both goes through mx; bar names a barrier of the two.  STORED:
// v becomes what a load of the stored site gives.
template <bool STORED = false>
__device__ __forceinline__ void store6(void *p, float *n, int s, bool active, int q, CF (&v)[6], float (*mx)[32],
                                       int bar) {
  const int lane = threadIdx.x & 31;
  float m = 0.f;
#pragma unroll
  for (int k = 0; k < 6; k++) m = fmaxf(m, fmaxf(fabsf(v[k].re), fabsf(v[k].im)));
  mx[q][lane] = m;
  asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
  m = fmaxf(m, mx[1 - q][lane]);
  asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");  // mx may be written again
  const float k = m > 0.f ? FIX16_SCALE / m : 0.f;
  Raw6 r;
  r.n = m * F16;
  unsigned(&w)[6] = r.w;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    w[2 * c] = fix16_pack_k(v[c].re, v[3 + c].re, k);
    w[2 * c + 1] = fix16_pack_k(v[c].im, v[3 + c].im, k);
  }
  if constexpr (STORED) decode(r, v);
  if (!active) return;
  char *b = static_cast<char *>(p);
  if (q) {
    *reinterpret_cast<uint2 *>(b + s16_w8(s) + 24) = make_uint2(w[0], w[1]);
    *reinterpret_cast<uint4 *>(b + s16_w4(s)) = make_uint4(w[2], w[3], w[4], w[5]);
  } else {
    *reinterpret_cast<uint4 *>(b + s16_w8(s)) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint2 *>(b + s16_w8(s) + 16) = make_uint2(w[4], w[5]);
    n[s] = m;
  }
}

// products and sums in FP64: <rt, r> and |r|^2 of a new residual are differences of these
__device__ __forceinline__ void dot6(const CF (&a)[6], const CF (&b)[6], double &re, double &im) {
#pragma unroll
  for (int c = 0; c < 6; c++) {
    re = fma((double)a[c].re, (double)b[c].re, fma((double)a[c].im, (double)b[c].im, re));
    im = fma((double)a[c].re, (double)b[c].im, fma(-(double)a[c].im, (double)b[c].re, im));
  }
}
__device__ __forceinline__ void norm6(const CF (&a)[6], double &n2) {
#pragma unroll
  for (int c = 0; c < 6; c++) n2 = fma((double)a[c].re, (double)a[c].re, fma((double)a[c].im, (double)a[c].im, n2));
}

// This warp's hop (h = 2 mu + (0 forward, 1 backward)): what its projector
// multiplies the lower spins by, S g(mu, 0) and S g(mu, 1).
struct HopOfWarp {
  int h;
  CF a0, a1;
};
__device__ __forceinline__ HopOfWarp hop_of_warp(int h) {
  HopOfWarp o;
  o.h = h;
  const float S = h & 1 ? 1.f : -1.f;
  switch (h >> 1) {
    case 0: o.a0 = CF(S * gre(0, 0), S * gim(0, 0)), o.a1 = CF(S * gre(0, 1), S * gim(0, 1)); break;
    case 1: o.a0 = CF(S * gre(1, 0), S * gim(1, 0)), o.a1 = CF(S * gre(1, 1), S * gim(1, 1)); break;
    case 2: o.a0 = CF(S * gre(2, 0), S * gim(2, 0)), o.a1 = CF(S * gre(2, 1), S * gim(2, 1)); break;
    default: o.a0 = CF(S * gre(3, 0), S * gim(3, 0)), o.a1 = CF(S * gre(3, 1), S * gim(3, 1)); break;
  }
  return o;
}

// neighbour of site s (parity par) along the warp's hop, and the t-boundary phase
__device__ __forceinline__ int hop_neighbour(const InnerArgs &a, int s, int par, int h, float &ph) {
  const Geom &g = a.g;
  int xh, y, z, t;
  site_coords(g, s, xh, y, z, t);
  const int xodd = (y + z + t + par) & 1;
  ph = 1.f;
  switch (h) {
    case 0: return xodd ? (xh == g.Lxh - 1 ? s - xh : s + 1) : s;
    case 1: return xodd ? s : (xh == 0 ? s + g.Lxh - 1 : s - 1);
    case 2: return y == g.Ly - 1 ? s - (g.Ly - 1) * g.sy : s + g.sy;
    case 3: return y == 0 ? s + (g.Ly - 1) * g.sy : s - g.sy;
    case 4: return z == g.Lz - 1 ? s - (g.Lz - 1) * g.sz : s + g.sz;
    case 5: return z == 0 ? s + (g.Lz - 1) * g.sz : s - g.sz;
    case 6:
      if (t == g.Lt - 1) ph = (float)a.t_bc;
      return t == g.Lt - 1 ? s - (g.Lt - 1) * g.st : s + g.st;
    default:
      if (t == 0) ph = (float)a.t_bc;
      return t == 0 ? s + (g.Lt - 1) * g.st : s - g.st;
  }
}

// U h or U^dag h of the projected spinor psi, both spins, into ex[12][32]
__device__ __forceinline__ void hop_warp(const HopOfWarp &o, const unsigned (&lw)[6], float ph, const CF (&psi)[12],
                                         float (*ex)[32]) {
  const bool cross = o.h < 4, back = o.h & 1;  // x, y: spin 0 with 3 and 1 with 2; z, t: 0 with 2 and 1 with 3
  CF u[9], h[2][3];
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const float2 f = fix16_unpack(lw[k]);
    u[k] = CF(f.x * F16, f.y * F16);
  }
  su3_row2(u);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const CF q0 = cross ? psi[9 + c] : psi[6 + c], q1 = cross ? psi[6 + c] : psi[9 + c];
    h[0][c].re = fmaf(o.a0.re, q0.re, fmaf(-o.a0.im, q0.im, psi[c].re));
    h[0][c].im = fmaf(o.a0.re, q0.im, fmaf(o.a0.im, q0.re, psi[c].im));
    h[1][c].re = fmaf(o.a1.re, q1.re, fmaf(-o.a1.im, q1.im, psi[3 + c].re));
    h[1][c].im = fmaf(o.a1.re, q1.im, fmaf(o.a1.im, q1.re, psi[3 + c].im));
  }
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < 3; r++) {
    CF m[3];
#pragma unroll
    for (int c = 0; c < 3; c++) m[c] = back ? u[c * 3 + r].conj() : u[r * 3 + c];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      float re = 0.f, im = 0.f;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        re = fmaf(m[c].re, h[k][c].re, fmaf(-m[c].im, h[k][c].im, re));
        im = fmaf(m[c].re, h[k][c].im, fmaf(m[c].im, h[k][c].re, im));
      }
      ex[(k * 3 + r) * 2][lane] = re * ph;
      ex[(k * 3 + r) * 2 + 1][lane] = im * ph;
    }
  }
}

// one hop's share of chirality Q's components (spins 2Q, 2Q + 1) from its two stored spins
template <int MU, bool FWD, int Q>
__device__ __forceinline__ void add_hop(const float (*ex)[32], int lane, CF (&w)[6]) {
  constexpr int S = FWD ? -1 : 1;
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int r = 0; r < 3; r++) {
      constexpr int C0 = Q ? gcol(MU, 2) : 0, C1 = Q ? gcol(MU, 3) : 1;
      const int e = ((k ? C1 : C0) * 3 + r) * 2;
      const CF v(ex[e][lane], ex[e + 1][lane]);
      if constexpr (Q == 0) w[k * 3 + r] += v;
      else if (k == 0) w[r] += unit_mul<S * gre(MU, 2), S * gim(MU, 2)>(v);
      else w[3 + r] += unit_mul<S * gre(MU, 3), S * gim(MU, 3)>(v);
    }
}
template <int Q>
__device__ __forceinline__ void sum_hops(const float (*ex)[12][32], int lane, CF (&w)[6]) {
#pragma unroll
  for (int k = 0; k < 6; k++) w[k] = CF(0.f, 0.f);
  add_hop<0, true, Q>(ex[0], lane, w);
  add_hop<0, false, Q>(ex[1], lane, w);
  add_hop<1, true, Q>(ex[2], lane, w);
  add_hop<1, false, Q>(ex[3], lane, w);
  add_hop<2, true, Q>(ex[4], lane, w);
  add_hop<2, false, Q>(ex[5], lane, w);
  add_hop<3, true, Q>(ex[6], lane, w);
  add_hop<3, false, Q>(ex[7], lane, w);
}
__device__ __forceinline__ void clover6(const float (&d)[6], const CF (&L)[15], CF (&w)[6]) {
  CF y[6];
#pragma unroll
  for (int i = 0; i < 6; i++) y[i] = w[i] * d[i];
#pragma unroll
  for (int i = 1; i < 6; i++)
#pragma unroll
    for (int j = 0; j < i; j++) {
      const CF l = L[i * (i - 1) / 2 + j];
      y[i] += l * w[j];
      y[j] += cdotmul(l, w[i]);
    }
#pragma unroll
  for (int i = 0; i < 6; i++) w[i] = y[i];
}

// x += al p + om s of one chirality's components (x: SOA32, written by this thread only)
__device__ __forceinline__ void add_x(float4 *x, int s, bool active, int q, CF al, const CF (&p)[6], CF om, const CF (&sv)[6]) {
  if (!active) return;
  float4 *xs = x + blk_base<6>(s) + 3 * q * SB;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const float4 v = __ldcg(xs + c * SB);
    const CF d0 = p[c] * al + sv[c] * om, d1 = p[3 + c] * al + sv[3 + c] * om;
    xs[c * SB] = make_float4(v.x + d0.re, v.y + d1.re, v.z + d0.im, v.w + d1.im);
  }
}

template <bool CLOV>
__global__ void __launch_bounds__(IS_THREADS, 1) k_inner_small(InnerArgs a) {
  __shared__ GridRedShared sh;
  __shared__ float ex[8][12][32];
  __shared__ float mx[4][2][32];  // of the tmp/v/t stores, and of the own r and p
  __shared__ double tot[8];
  __shared__ Cpx<double> sc[4];  // alpha, omega, beta, <rt, r>
  __shared__ double rrs;
  __shared__ int state, next;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int Vh = a.g.Vh, ntile = (Vh + 31) / 32;
  if (grid_red_failed(a.red)) {
    if (threadIdx.x == 0) a.st->gave_up = 1;
    return;
  }
  const unsigned base = a.red->base;
  unsigned epoch = 0;
  const HopOfWarp hw = hop_of_warp(warp);
  const VecSet &vs = a.vs;
  float4 *x = static_cast<float4 *>(vs.x);
  // the two buffers of r and p: selected, not indexed (no local memory)
  auto rbuf = [&](int i) { return i ? vs.s : vs.r; };
  auto rnorm = [&](int i) { return i ? vs.sn : vs.rn; };
  auto pbuf = [&](int i) { return i ? a.p2 : vs.p; };
  auto pnorm = [&](int i) { return i ? a.p2n : vs.pn; };
  const float k2 = (float)-a.k2;

  // the link of this warp's hop onto site s of parity par (n: its neighbour)
  auto link = [&](int par, int s, int n, unsigned(&lw)[6]) {
    const int lpar = warp & 1 ? 1 - par : par;
    g16_load_words(a.gauge, (size_t)((warp >> 1) * 2 + lpar) * pad_sites(Vh), warp & 1 ? n : s, lw);
  };

  // r = rt = p = r64 in 16 bits, x = 0: warps 0 and 1, a chirality each
  double v2[2] = {0.0, 0.0};
  for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int s = min(tile * 32 + lane, Vh - 1);
    const bool active = tile * 32 + lane < Vh;
    if (warp < 2) {
      CF f[6];
      const double2 *p = static_cast<const double2 *>(vs.r64) + blk_base<12>(s) + 6 * warp * SB;
#pragma unroll
      for (int c = 0; c < 6; c++) {
        const double2 d = __ldg(p + c * SB);
        f[c] = CF((float)d.x, (float)d.y);
        if (active) {
          v2[0] += (double)f[c].re * f[c].re + (double)f[c].im * f[c].im;
          v2[1] += d.x * d.x + d.y * d.y;
        }
      }
      store6(rbuf(0), rnorm(0), s, active, warp, f, mx[0], 1);
      store6(vs.rt, vs.rtn, s, active, warp, f, mx[0], 1);
      store6(pbuf(0), pnorm(0), s, active, warp, f, mx[0], 1);
      if (active)
#pragma unroll
        for (int c = 0; c < 3; c++) x[blk_base<6>(s) + (3 * warp + c) * SB] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  bool ok = grid_allreduce<2>(a.red, base, ++epoch, v2, 1, tot, sh);
  const double rr0 = tot[1], tol2 = a.rel2 * rr0;
  double rr = rr0;
  int status = !ok ? ST_RUNNING : bad_number(rr0) ? ST_NAN : rr0 <= tol2 ? ST_CONVERGED : ST_RUNNING, it = 0;
  if (threadIdx.x == 0) sc[3] = Cpx<double>(tot[0], 0.0);
  CF al(0.f, 0.f), om(0.f, 0.f), be(0.f, 0.f);  // of the previous iteration, until its own are known
  while (ok && status == ST_RUNNING) {
    const int cur = it & 1, old = cur ^ 1;
    // The four products of an iteration share one copy of the code: four copies
    // (100 KB) did not stay in the instruction cache and took twice as long.
#pragma unroll 1
    for (int part = 0; part < 4; part++) {
      // the product's source, src[0] + c1 v + c2 t + c3 p at the neighbour
      // (nsrc of them), and what is added to it, x1 (- alpha v)
      const int par = part & 1;
      const bool fresh = part == 0 && it > 0;  // p is new: formed here
      const int rs = fresh ? old : (part == 0 ? 0 : cur);
      const void *src = par ? a.tmp : rbuf(rs);
      const float *srcn = par ? a.tmpn : rnorm(rs);
      const int nsrc = fresh ? 4 : (part == 2 ? 2 : 1);
      const CF bo = be * om;
      const CF c1 = fresh ? CF(-(al.re + bo.re), -(al.im + bo.im)) : CF(-al.re, -al.im);
      const void *x1 = part == 1 ? pbuf(cur) : rbuf(cur);
      const float *x1n = part == 1 ? pnorm(cur) : rnorm(cur);
      void *dst = par == 0 ? a.tmp : (part == 1 ? vs.v : vs.t);
      float *dstn = par == 0 ? a.tmpn : (part == 1 ? vs.vn : vs.tn);
      double v8[8];
#pragma unroll
      for (int k = 0; k < 8; k++) v8[k] = 0.0;
#pragma unroll 1
      for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int s = min(tile * 32 + lane, Vh - 1);
        const bool active = tile * 32 + lane < Vh;
        float ph;
        const int n = hop_neighbour(a, s, par, warp, ph);
        unsigned lw[6];
        link(par, s, n, lw);
        Raw12 R, V, T, P;
        raw12(src, srcn, n, R);
        if (nsrc > 1) raw12(vs.v, vs.vn, n, V);
        if (nsrc > 2) {
          raw12(vs.t, vs.tn, n, T);
          raw12(pbuf(old), pnorm(old), n, P);
        }
        CF psi[12];
        decode(R, psi);
        if (nsrc > 1) add_scaled(psi, c1, V);
        if (nsrc > 2) {
          add_scaled(psi, CF(-om.re, -om.im), T);
          add_scaled(psi, be, P);
        }
        Raw6 X, W, Z;  // of the epilogue: under way while the hops are computed
        if (par && warp < 2) {
          raw6(x1, x1n, s, warp, X);
          raw6(vs.rt, vs.rtn, s, warp, Z);
          if (part == 3) raw6(vs.v, vs.vn, s, warp, W);
        }
        float cd[6];
        CF cL[15];
        if (CLOV && warp < 2) clover_block_load<CSOA32, float>(CloverView<CSOA32>{par ? a.c1 : a.c0, Vh}, warp, s, cd, cL);
        __syncthreads();  // the previous tile's hops are summed
        hop_warp(hw, lw, ph, psi, ex[warp]);
        __syncthreads();
        if (warp < 2) {
          CF w[6], q[6], z[6];
          if (warp) sum_hops<1>(ex, lane, w);
          else sum_hops<0>(ex, lane, w);
          if constexpr (CLOV) clover6(cd, cL, w);
          if (par) {
            decode(X, q);
            if (part == 3) add_scaled(q, CF(-al.re, -al.im), W);
#pragma unroll
            for (int k = 0; k < 6; k++) w[k] = w[k] * k2 + q[k];
          }
          store6<true>(dst, dstn, s, active, warp, w, mx[0], 1);
          if (par && active) {
            decode(Z, z);
            dot6(z, w, v8[0], v8[1]);  // <rt, v> or <rt, t>
            if (part == 3) {
              dot6(w, q, v8[2], v8[3]);  // <t, s>
              norm6(w, v8[4]);           // |t|^2
              dot6(z, q, v8[5], v8[6]);  // <rt, s>
              norm6(q, v8[7]);           // |s|^2
            }
          }
        } else if (warp < 4 && fresh) {
          // the own x += alpha p + omega s; r, p <- new, into the other buffers
          const int q = warp - 2;
          Raw6 r6, v6, t6, p6;
          raw6(rbuf(old), rnorm(old), s, q, r6);
          raw6(vs.v, vs.vn, s, q, v6);
          raw6(vs.t, vs.tn, s, q, t6);
          raw6(pbuf(old), pnorm(old), s, q, p6);
          CF sv[6], pv[6];
          decode(r6, sv);
          add_scaled(sv, CF(-al.re, -al.im), v6);
          decode(p6, pv);
          add_x(x, s, active, q, al, pv, om, sv);
          add_scaled(sv, CF(-om.re, -om.im), t6);  // the new r
          add_scaled(pv, CF(-om.re, -om.im), v6);
#pragma unroll
          for (int k = 0; k < 6; k++) pv[k] = sv[k] + pv[k] * be;
          store6(rbuf(cur), rnorm(cur), s, active, q, sv, mx[2], 2);
          store6(pbuf(cur), pnorm(cur), s, active, q, pv, mx[3], 2);
        }
      }
      if (par == 0) {
        ok = grid_barrier(a.red, base, ++epoch, sh);
        if (!ok) break;
        continue;
      }
      ok = grid_allreduce<8>(a.red, base, ++epoch, v8, 1, tot, sh);
      if (!ok) break;
      if (threadIdx.x == 0) {
        if (part == 1) {
          const Cpx<double> den(tot[0], tot[1]);
          state = den.norm2() == 0.0 || bad_number(tot[0]) || bad_number(tot[1]) ? ST_BREAKDOWN : ST_RUNNING;
          sc[0] = sc[3] * den.conj() * (1.0 / den.norm2());  // one division, not two: they are slow and serial
        } else if (tot[4] == 0.0 || bad_number(tot[4])) {
          state = bad_number(tot[4]) ? ST_NAN : ST_BREAKDOWN;
        } else {
          const double inv = 1.0 / tot[4];
          const Cpx<double> w(tot[2] * inv, tot[3] * inv);
          const Cpx<double> rho = Cpx<double>(tot[5], tot[6]) - w * Cpx<double>(tot[0], tot[1]);
          const Cpx<double> den = sc[3] * w;
          sc[2] = rho * sc[0] * den.conj() * (1.0 / den.norm2());
          sc[1] = w;
          sc[3] = rho;
          rrs = fmax(tot[7] - (tot[2] * tot[2] + tot[3] * tot[3]) * inv, 0.0);
          next = bad_number(tot[7])               ? ST_NAN
                 : rrs <= tol2                    ? ST_CONVERGED
                 : rho.re == 0.0 && rho.im == 0.0 ? ST_BREAKDOWN
                 : it + 1 >= a.maxiter            ? ST_MAXITER
                                                  : ST_RUNNING;
        }
      }
      __syncthreads();
      if (state != ST_RUNNING) {
        status = state;
        break;
      }
      if (part == 1) al = CF((float)sc[0].re, (float)sc[0].im);
    }
    if (!ok || status != ST_RUNNING) break;
    status = next;
    rr = rrs;
    om = CF((float)sc[1].re, (float)sc[1].im);
    be = CF((float)sc[2].re, (float)sc[2].im);
    it++;
    if (status != ST_RUNNING && status != ST_NAN && warp >= 2 && warp < 4) {  // the last x update (buffers as they are now)
      for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int s = min(tile * 32 + lane, Vh - 1);
        const int q = warp - 2;
        Raw6 R, V, P;
        raw6(rbuf(cur), rnorm(cur), s, q, R);
        raw6(vs.v, vs.vn, s, q, V);
        raw6(pbuf(cur), pnorm(cur), s, q, P);
        CF sv[6], pv[6];
        decode(R, sv);
        add_scaled(sv, CF(-al.re, -al.im), V);
        decode(P, pv);
        add_x(x, s, tile * 32 + lane < Vh, q, al, pv, om, sv);
      }
    }
  }
  __syncthreads();
  if (!ok) {
    if (threadIdx.x == 0) a.st->gave_up = 1;
    return;
  }
  // the result in FP64 (warp 2 and 3 own x)
  if (warp >= 2 && warp < 4)
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
      const int s = tile * 32 + lane, q = warp - 2;
      if (s >= Vh) continue;
      double2 *z = static_cast<double2 *>(a.z) + blk_base<12>(s) + 6 * q * SB;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const float4 d = __ldcg(x + blk_base<6>(s) + (3 * q + c) * SB);
        z[c * SB] = make_double2(d.x, d.z);
        z[(c + 3) * SB] = make_double2(d.y, d.w);
      }
    }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.st->iter = it;
    a.st->rr = rr;
    a.st->status = status;
    a.st->done = 1;
    grid_red_end(a.red, base, epoch);
  }
}

}  // namespace

// three 32-site tiles an SM: beyond, the graph of kernels overtakes it
bool inner_small_fits(int Vh, int sms) { return Vh <= 3 * 32 * sms; }

void launch_inner_small(const InnerArgs &a, int sms, cudaStream_t s) {
  const int grid = std::min(std::min(GRID_RED_BLOCKS, sms), (a.g.Vh + 31) / 32);  // one block an SM
  const void *k = a.c0 ? reinterpret_cast<const void *>(k_inner_small<true>) : reinterpret_cast<const void *>(k_inner_small<false>);
  InnerArgs arg = a;
  void *args[] = {&arg};
  QCU_CUDA(grid_red_inject(a.red, "inner", s));
  QCU_CUDA(cudaLaunchCooperativeKernel(k, dim3(grid), dim3(IS_THREADS), args, 0, s));
  note_launch(1);
}

}  // namespace qcu
