// One training step's loss and gradient of the parallel-transport network.
//
// The network is linear in its input, so the gradient needs neither the hidden
// field nor its adjoint.  With the features of an even site y (h = 1..8)
//   v_{hb}(y) = (T_h r_b)(y)            the transported inputs,
//   u_{ha}(y) = (T_h^dag delta_a)(y)    the output error, brought back along hop h,
// and with c summed over colours,
//   R_{ha,h'b} = sum_y,c u_ha conj(v_h'b)    (32 x 32),
//   S_{ab}     = sum_x,c delta_a conj(r_b)   (4 x 4, odd sites),
// the gradients of both layers follow from R and S by products with the weights:
//   dL/dW2[h]_ak = sum_j R_{ha,j} conj(W1_{k,j}),   dL/dW1[h']_kb = sum_i conj(W2_{i,k}) R_{i,h'b}
// (h = 0: the same with S).  A step is
//   k_tr_load   complex128 batches -> FP32 fields, |e|^2
//   k_tr_even   hidden = sum_h W1[h] v_h on the even sites, kept in registers;
//               z_h = W2[h] hidden, what hop h of the one odd site that reaches
//               y by it will transport: mixing before transporting moves 4
//               colour vectors where transporting the hidden field moves 16
//   k_tr_odd    out = sum_h T_h z_h + W2[0] W1[0] r, the loss, delta, S
//   k_tr_outer  R, as a GEMM over (site, colour) in shared memory
//   k_tr_reduce, k_tr_grads
// FP32 arithmetic on paired instructions; a block's sums of R, S and the loss
// over its tiles are FP32, the sums across blocks FP64, all in a fixed order (the
// gradient is reproducible to the bit).  16^4, batch 16: 1.00 ms a step (load 45
// us, even 335, odd 144, outer 409), where layer by layer gradients with warp
// reductions and atomics took 8.2 ms.  Error of the gradient against 64 bits, 16^4
// batch 16, 16^3 x 32 batch 32 and 32^3 x 64 batch 4 (55, 221 and 443 tiles a
// block): 3.1e-8, 2.9e-8 and 2.8e-8, where it was 9e-7, 1.9e-6 and 2.7e-6.
#include <algorithm>

#include "hop32.cuh"
#include "nn.h"

namespace qcu {
namespace {

constexpr int TR_BLOCK = 128;

// site-blocked FP32 field of NC float4 (two complex numbers each) per site
template <int NC>
__device__ __forceinline__ size_t tr_at(int nblk, int b, int s) {
  return ((size_t)b * nblk + (s >> 5)) * NC * 32 + (s & 31);
}

// i z
__device__ __forceinline__ float2 times_i(float2 z) { return make_float2(-z.y, z.x); }
// acc += w z
__device__ __forceinline__ void cmad2(float2 &acc, float2 wre, float2 wim, float2 z, float2 iz) {
  acc = fma2(wre, z, acc);
  acc = fma2(wim, iz, acc);
}

// A hop from site s of parity par: the site it reads (of the other parity) and
// the matrix it multiplies by, boundary phase included.
struct TrHop {
  int n;
  Cpx<float> m[9];
};
__device__ __forceinline__ void tr_hop(const Geom &g, const void *gauge, float t_bc, int s, const int c[4], int par,
                                       int mu, bool fwd, TrHop &o) {
  const int xodd = (c[1] + c[2] + c[3] + par) & 1;
  float ph = 1.f;
  if (mu == 0) o.n = fwd ? (xodd ? (c[0] == g.Lxh - 1 ? s - c[0] : s + 1) : s) : (xodd ? s : (c[0] == 0 ? s + g.Lxh - 1 : s - 1));
  else if (mu == 1) o.n = fwd ? (c[1] == g.Ly - 1 ? s - (g.Ly - 1) * g.sy : s + g.sy) : (c[1] == 0 ? s + (g.Ly - 1) * g.sy : s - g.sy);
  else if (mu == 2) o.n = fwd ? (c[2] == g.Lz - 1 ? s - (g.Lz - 1) * g.sz : s + g.sz) : (c[2] == 0 ? s + (g.Lz - 1) * g.sz : s - g.sz);
  else {
    o.n = fwd ? (c[3] == g.Lt - 1 ? s - (g.Lt - 1) * g.st : s + g.st) : (c[3] == 0 ? s + (g.Lt - 1) * g.st : s - g.st);
    if (fwd ? c[3] == g.Lt - 1 : c[3] == 0) ph = t_bc;
  }
  Cpx<float> u[9];
  link_load<GSOA32, float>(GaugeView<GSOA32>{gauge, pad_sites(g.Vh)}, mu, fwd ? par : 1 - par, fwd ? s : o.n, u);
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int k = 0; k < 3; k++) o.m[r * 3 + k] = (fwd ? u[r * 3 + k] : u[k * 3 + r].conj()) * ph;
}

// v[a][r] = (or +=) sum_c m_rc q[a][c] for the four colour vectors (6 float4) at p
template <bool ADD>
__device__ __forceinline__ void tr_transport(const Cpx<float> m[9], const float4 *p, float2 v[4][3]) {
  float2 q[12];
#pragma unroll
  for (int j = 0; j < 6; j++) {
    const float4 d = __ldg(p + j * 32);
    q[2 * j] = make_float2(d.x, d.y);
    q[2 * j + 1] = make_float2(d.z, d.w);
  }
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int r = 0; r < 3; r++) {
      float2 t = ADD ? v[a][r] : make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < 3; c++)
        cmad2(t, bc2(m[r * 3 + c].re), bc2(m[r * 3 + c].im), q[a * 3 + c], times_i(q[a * 3 + c]));
      v[a][r] = t;
    }
}

// complex128 half spinors r, e [B][Vh][12] -> site-blocked FP32, and the block
// sums of |e|^2; a warp moves its 32 records contiguously (as k_convert_aos)
__global__ void __launch_bounds__(TR_BLOCK) k_tr_load(int Vh, int nb, const double2 *r, const double2 *e, float4 *fr, float4 *fe,
                                                     double *norms) {
  __shared__ double2 rec[TR_BLOCK / 32][32 * 13];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nblk = (Vh + 31) / 32;
  const int b = blockIdx.x / nb, s0 = (blockIdx.x % nb * (TR_BLOCK / 32) + warp) * 32, s = s0 + lane;
  const int n = min(32, Vh - s0) * 12;
  double2 *w = rec[warp];
  double e2[1] = {0.0};
#pragma unroll
  for (int which = 0; which < 2; which++) {
    const double2 *p = (which ? e : r) + ((size_t)b * Vh + s0) * 12;
#pragma unroll
    for (int k = 0; k < 12; k++) {
      const int i = k * 32 + lane;
      if (i < n) w[i / 12 * 13 + i % 12] = __ldcs(p + i);
    }
    __syncwarp();
    if (s < Vh) {
      float4 *o = (which ? fe : fr) + tr_at<6>(nblk, b, s);
#pragma unroll
      for (int j = 0; j < 6; j++) {
        const double2 x = w[lane * 13 + 2 * j], y = w[lane * 13 + 2 * j + 1];
        o[j * 32] = make_float4((float)x.x, (float)x.y, (float)y.x, (float)y.y);
        if (which) e2[0] += x.x * x.x + x.y * x.y + y.x * y.x + y.y * y.y;
      }
    }
    __syncwarp();
  }
  double tot[1];
  block_sum<1, TR_BLOCK>(e2, tot);
  if (threadIdx.x == 0) norms[blockIdx.x] = tot[0];
}

__global__ void __launch_bounds__(TR_BLOCK) k_tr_norms(int n, const double *norms, float *enorm) {
  double v[1] = {0.0}, tot[1];
  for (int i = threadIdx.x; i < n; i += TR_BLOCK) v[0] += norms[(size_t)blockIdx.x * n + i];
  block_sum<1, TR_BLOCK>(v, tot);
  if (threadIdx.x == 0) enorm[blockIdx.x] = (float)tot[0];
}

// complex weights as the broadcast pairs of the paired instructions
__device__ __forceinline__ float4 dup(float2 w) { return make_float4(w.x, w.x, w.y, w.y); }

// z_h = W2[h] sum_h' W1[h'] T_h' r on the even sites, h = 1..8.  Bound by FP32
// arithmetic: 13.4 kFMA a site, against 0.9 KB written.
__global__ void __launch_bounds__(TR_BLOCK, 3) k_tr_even(Geom g, TrainArgs a, int nb) {
  __shared__ float4 W1[8 * 64], W2[8 * 64];  // [h][k][b], [h][a][k]
  for (int i = threadIdx.x; i < 8 * 64; i += TR_BLOCK) {
    W1[i] = dup(a.w1[64 + i]);
    W2[i] = dup(a.w2[64 + i]);
  }
  __syncthreads();
  const int b = blockIdx.x / nb, s = blockIdx.x % nb * TR_BLOCK + threadIdx.x, nblk = (g.Vh + 31) / 32;
  if (s >= g.Vh) return;
  int c[4];
  site_coords(g, s, c[0], c[1], c[2], c[3]);
  float2 hid[16][3];
#pragma unroll
  for (int k = 0; k < 16; k++)
#pragma unroll
    for (int r = 0; r < 3; r++) hid[k][r] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int h = 0; h < 8; h++) {
    TrHop t;
    tr_hop(g, a.gauge, a.t_bc, s, c, 0, h >> 1, (h & 1) == 0, t);
    float2 v[4][3];
    tr_transport<false>(t.m, a.r + tr_at<6>(nblk, b, t.n), v);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float2 i0 = times_i(v[q][0]), i1 = times_i(v[q][1]), i2 = times_i(v[q][2]);
#pragma unroll
      for (int k = 0; k < 16; k++) {
        const float4 w = W1[h * 64 + k * 4 + q];
        const float2 re = make_float2(w.x, w.y), im = make_float2(w.z, w.w);
        cmad2(hid[k][0], re, im, v[q][0], i0);
        cmad2(hid[k][1], re, im, v[q][1], i1);
        cmad2(hid[k][2], re, im, v[q][2], i2);
      }
    }
  }
  float4 *z = a.z + tr_at<48>(nblk, b, s);
#pragma unroll 1
  for (int h = 0; h < 8; h++) {
#pragma unroll 1
    for (int q = 0; q < 4; q += 2) {  // two output channels at a time: 3 float4
      float2 re[6], im[6];            // sums of Re w times hid and of Im w times hid
#pragma unroll
      for (int i = 0; i < 6; i++) re[i] = im[i] = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 16; k++) {
#pragma unroll
        for (int d = 0; d < 2; d++) {
          const float4 w = W2[h * 64 + (q + d) * 16 + k];
#pragma unroll
          for (int r = 0; r < 3; r++) {
            re[d * 3 + r] = fma2(make_float2(w.x, w.y), hid[k][r], re[d * 3 + r]);
            im[d * 3 + r] = fma2(make_float2(w.z, w.w), hid[k][r], im[d * 3 + r]);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 3; j++)
        z[(h * 6 + (q >> 1) * 3 + j) * 32] = make_float4(re[2 * j].x - im[2 * j].y, re[2 * j].y + im[2 * j].x,
                                                        re[2 * j + 1].x - im[2 * j + 1].y, re[2 * j + 1].y + im[2 * j + 1].x);
    }
  }
}

// The odd sites: out, delta = (out - e) / (|e|^2 B), and this block's share of
// the loss and of S.  Bound by memory: every z_h is read once.
constexpr int TR_NS = 33;  // Re, Im of S[a][b], then the loss
__global__ void __launch_bounds__(TR_BLOCK, 3) k_tr_odd(Geom g, TrainArgs a, int nb) {
  __shared__ float4 W0[16];  // (W2[0] W1[0])[a][b]
  __shared__ float part[TR_BLOCK / 32][TR_NS];
  if (threadIdx.x < 16) {
    const int o = threadIdx.x >> 2, i = threadIdx.x & 3;
    double re = 0, im = 0;
    for (int k = 0; k < 16; k++) {
      const float2 x = a.w2[o * 16 + k], y = a.w1[k * 4 + i];
      re += (double)x.x * y.x - (double)x.y * y.y;
      im += (double)x.x * y.y + (double)x.y * y.x;
    }
    W0[threadIdx.x] = dup(make_float2((float)re, (float)im));
  }
  __syncthreads();
  const int b = blockIdx.x / nb, nblk = (g.Vh + 31) / 32;
  const float inv = 1.f / a.enorm[b];
  float2 S[16];
#pragma unroll
  for (int k = 0; k < 16; k++) S[k] = make_float2(0.f, 0.f);
  float loss = 0.f;
  for (int s = blockIdx.x % nb * TR_BLOCK + threadIdx.x; s < g.Vh; s += nb * TR_BLOCK) {
    int c[4];
    site_coords(g, s, c[0], c[1], c[2], c[3]);
    float2 out[4][3];
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
      for (int r = 0; r < 3; r++) out[o][r] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int h = 0; h < 8; h++) {
      TrHop t;
      tr_hop(g, a.gauge, a.t_bc, s, c, 1, h >> 1, (h & 1) == 0, t);
      tr_transport<true>(t.m, a.z + tr_at<48>(nblk, b, t.n) + h * 6 * 32, out);
    }
    float2 r[4][3];
    const float4 *pr = a.r + tr_at<6>(nblk, b, s), *pe = a.e + tr_at<6>(nblk, b, s);
    float4 *pd = a.delta + tr_at<6>(nblk, b, s);
#pragma unroll
    for (int j = 0; j < 6; j++) {
      const float4 d = __ldg(pr + j * 32);
      r[2 * j / 3][2 * j % 3] = make_float2(d.x, d.y);
      r[(2 * j + 1) / 3][(2 * j + 1) % 3] = make_float2(d.z, d.w);
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const float2 ir = times_i(r[q][k]);
#pragma unroll
        for (int o = 0; o < 4; o++) {
          const float4 w = W0[o * 4 + q];
          cmad2(out[o][k], make_float2(w.x, w.y), make_float2(w.z, w.w), r[q][k], ir);
        }
      }
    float l = 0.f;
#pragma unroll
    for (int j = 0; j < 6; j++) {
      const float4 e = __ldg(pe + j * 32);
      float2 &x = out[2 * j / 3][2 * j % 3], &y = out[(2 * j + 1) / 3][(2 * j + 1) % 3];
      x = make_float2(x.x - e.x, x.y - e.y);
      y = make_float2(y.x - e.z, y.y - e.w);
      l += x.x * x.x + x.y * x.y + y.x * y.x + y.y * y.y;
      x = make_float2(x.x * inv / a.B, x.y * inv / a.B);
      y = make_float2(y.x * inv / a.B, y.y * inv / a.B);
      pd[j * 32] = make_float4(x.x, x.y, y.x, y.y);
    }
    loss += l * inv;
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int k = 0; k < 3; k++) {  // delta conj(r) = Re r delta - i Im r delta
          float2 &acc = S[o * 4 + q];
          acc = fma2(bc2(r[q][k].x), out[o][k], acc);
          acc = fma2(bc2(r[q][k].y), make_float2(out[o][k].y, -out[o][k].x), acc);
        }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < TR_NS; k++) {
    float v = k == 32 ? loss : (k & 1 ? S[k >> 1 & 15].y : S[k >> 1 & 15].x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) part[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < TR_NS) {
    double v = 0.0;
    for (int w = 0; w < TR_BLOCK / 32; w++) v += (double)part[w][threadIdx.x];
    a.part_s[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = v;
  }
}

// R = sum over the even sites and colours of u conj(v).  A tile is 32 sites:
// warp w (lane = site) forms the features of the neighbour in direction w / 2
// -- one matrix transports r for hop h and delta for the hop back, h ^ 1 --
// and the block then accumulates the 32 x 32 outer products over the tile's 96
// (site, colour) rows: 64 threads of 4 x 4 outputs for each quarter of the
// rows.  v lies planar and u as broadcast pairs, so that every multiply-add is
// a paired one on values as they are loaded: 6 16-byte shared loads for 32
// paired multiply-adds.  Bound by FP32 arithmetic: 12.3 + 2.3 kFMA a site.
// Row pitches are odd numbers of 16-byte units: a column of 32 sites is
// written without conflicts.
constexpr int TO_THREADS = 256, TO_ROWS = 96;
constexpr int TO_UP = 33;  // float4 per row of u: 32 features and the pad
constexpr int TO_VP = 9;   // float4 per row of Re v and of Im v: 32 floats and the pad
constexpr int TO_SMEM = TO_ROWS * (TO_UP + 2 * TO_VP) * 16;
static_assert(TO_SMEM >= 4 * 2048 * 4, "the final sum over the quarters reuses the tile");

__global__ void __launch_bounds__(TO_THREADS, 2) k_tr_outer(Geom g, TrainArgs a) {
  extern __shared__ __align__(16) float4 to_smem[];
  float4 *U = to_smem, *VR = U + TO_ROWS * TO_UP, *VI = VR + TO_ROWS * TO_VP;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nblk = (g.Vh + 31) / 32;
  const int ig = lane & 7, jg = (lane >> 3) + 4 * (warp & 1), quarter = warp >> 1;
  float2 R[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) R[i][j] = make_float2(0.f, 0.f);
  for (long long tile = blockIdx.x; tile < (long long)nblk * a.B; tile += gridDim.x) {
    const int b = (int)(tile / nblk), s = (int)(tile % nblk) * 32 + lane;
    __syncthreads();  // the previous tile is consumed
    float2 u[4][3], v[4][3];
    if (s < g.Vh) {
      int c[4];
      site_coords(g, s, c[0], c[1], c[2], c[3]);
      TrHop t;
      tr_hop(g, a.gauge, a.t_bc, s, c, 0, warp >> 1, (warp & 1) == 0, t);
      const size_t at = tr_at<6>(nblk, b, t.n);
      tr_transport<false>(t.m, a.r + at, v);
      tr_transport<false>(t.m, a.delta + at, u);
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int r = 0; r < 3; r++) u[q][r] = v[q][r] = make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const int row = lane * 3 + r;
      VR[row * TO_VP + warp] = make_float4(v[0][r].x, v[1][r].x, v[2][r].x, v[3][r].x);
      VI[row * TO_VP + warp] = make_float4(v[0][r].y, v[1][r].y, v[2][r].y, v[3][r].y);
#pragma unroll
      for (int q = 0; q < 4; q++) U[row * TO_UP + (warp ^ 1) * 4 + q] = dup(u[q][r]);
    }
    __syncthreads();
    float2 re[4][2], p[4][2], q[4][2];  // Ur Vr + Ui Vi, Ui Vr, Ur Vi, for j in pairs
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) re[i][j] = p[i][j] = q[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < TO_ROWS / 4; k++) {
      const int row = quarter * (TO_ROWS / 4) + k;
      const float4 xr = VR[row * TO_VP + jg], xi = VI[row * TO_VP + jg];
      const float2 vr[2] = {make_float2(xr.x, xr.y), make_float2(xr.z, xr.w)};
      const float2 vi[2] = {make_float2(xi.x, xi.y), make_float2(xi.z, xi.w)};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float4 w = U[row * TO_UP + ig + 8 * i];
        const float2 ur = make_float2(w.x, w.y), ui = make_float2(w.z, w.w);
#pragma unroll
        for (int j = 0; j < 2; j++) {
          re[i][j] = fma2(ur, vr[j], re[i][j]);
          re[i][j] = fma2(ui, vi[j], re[i][j]);
          p[i][j] = fma2(ui, vr[j], p[i][j]);
          q[i][j] = fma2(ur, vi[j], q[i][j]);
        }
      }
    }
    // the tile's sums (72 terms) onto the block's
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        R[i][2 * j] = add2(R[i][2 * j], make_float2(re[i][j].x, p[i][j].x - q[i][j].x));
        R[i][2 * j + 1] = add2(R[i][2 * j + 1], make_float2(re[i][j].y, p[i][j].y - q[i][j].y));
      }
  }
  __syncthreads();
  float2 *sum = reinterpret_cast<float2 *>(to_smem);  // [quarter][i][j]
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) sum[quarter * 1024 + (ig + 8 * i) * 32 + jg * 4 + j] = R[i][j];
  __syncthreads();
  const float *f = reinterpret_cast<const float *>(to_smem);
  for (int k = threadIdx.x; k < 2048; k += TO_THREADS)
    a.part_r[(size_t)blockIdx.x * 2048 + k] = ((double)f[k] + f[2048 + k]) + ((double)f[4096 + k] + f[6144 + k]);
}

// block partials -> sums[0..2047] = R, sums[2048..2080] = S and the loss
constexpr int TRR_BLOCK = 256;
__global__ void __launch_bounds__(TRR_BLOCK) k_tr_reduce(const double *part_r, int nr, const double *part_s, int ns,
                                                        double *sums) {
  if (blockIdx.x < 64) {  // 32 values of R each, 8 slices of the partials
    __shared__ double sh[8][32];
    const int k = blockIdx.x * 32 + (threadIdx.x & 31), slice = threadIdx.x >> 5;
    double v = 0.0;
    for (int i = slice; i < nr; i += 8) v += part_r[(size_t)i * 2048 + k];
    sh[slice][threadIdx.x & 31] = v;
    __syncthreads();
    if (slice == 0) {
      for (int i = 1; i < 8; i++) v += sh[i][threadIdx.x];
      sums[k] = v;
    }
  } else {
    const int k = blockIdx.x - 64;
    double v[1] = {0.0}, tot[1];
    for (int i = threadIdx.x; i < ns; i += TRR_BLOCK) v[0] += part_s[(size_t)k * ns + i];
    block_sum<1, TRR_BLOCK>(v, tot);
    if (threadIdx.x == 0) sums[2048 + k] = tot[0];
  }
}

// dL/dW1 [9][16][4], dL/dW2 [9][4][16] from R and S; a thread per weight of each
__global__ void __launch_bounds__(NN_HOPS * 64) k_tr_grads(const float2 *w1, const float2 *w2, const double *sums,
                                                         float2 *grad) {
  const int t = threadIdx.x, h = t / 64;
  const int n = h == 0 ? 4 : 32;  // terms: the channels of the other layer's outer side
  auto outer = [&](int i, int j) {  // R (h >= 1) or S
    const double *p = sums + (h == 0 ? 2048 + 2 * (i * 4 + j) : 2 * (i * 32 + j));
    return Cpx<double>(p[0], p[1]);
  };
  auto weight = [](float2 w) { return Cpx<double>((double)w.x, (double)w.y); };
  {
    const int k = (t % 64) / 4, b = t % 4;
    Cpx<double> v(0, 0);
    for (int i = 0; i < n; i++) {
      const int hi = h == 0 ? 0 : 1 + i / 4;
      v += cdotmul(weight(w2[(hi * 4 + i % 4) * 16 + k]), outer(i, h == 0 ? b : (h - 1) * 4 + b));
    }
    grad[t] = make_float2((float)v.re, (float)v.im);
  }
  {
    const int o = (t % 64) / 16, k = t % 16;
    Cpx<double> v(0, 0);
    for (int j = 0; j < n; j++) {
      const int hj = h == 0 ? 0 : 1 + j / 4;
      v += cdotmul(weight(w1[(hj * 16 + k) * 4 + j % 4]), outer(h == 0 ? o : (h - 1) * 4 + o, j));
    }
    grad[NN_HOPS * 64 + t] = make_float2((float)v.re, (float)v.im);
  }
}

}  // namespace

static int tr_blocks(int Vh) { return (Vh + TR_BLOCK - 1) / TR_BLOCK; }
// odd-site blocks per sample: a few waves of the whole batch, so that the
// 33-value block sums are shared by several sites a thread
static int tr_odd_blocks(int Vh, int B, int sms) { return std::min(tr_blocks(Vh), std::max(1, 6 * sms / B)); }
static int tr_outer_blocks(int Vh, int B, int sms) { return (int)std::min<int64_t>((int64_t)((Vh + 31) / 32) * B, 2 * sms); }

size_t train_field_bytes(int Vh, int B) { return (size_t)B * pad_sites(Vh) * 96; }
size_t train_part_bytes(int Vh, int B, int sms) {
  const size_t norms = (size_t)B * tr_blocks(Vh), s = (size_t)TR_NS * B * tr_odd_blocks(Vh, B, sms);
  return sizeof(double) * (2048 + TR_NS + norms + s + (size_t)2048 * tr_outer_blocks(Vh, B, sms));
}

void launch_train(const Geom &g, TrainArgs a, const void *r, const void *e, float4 *fr, float4 *fe, double *work,
                  float *enorm, float2 *grad, int sms, cudaStream_t s) {
  const int nb = tr_blocks(g.Vh), no = tr_odd_blocks(g.Vh, a.B, sms), nr = tr_outer_blocks(g.Vh, a.B, sms);
  double *sums = work, *norms = sums + 2048 + TR_NS;
  a.r = fr;
  a.e = fe;
  a.enorm = enorm;
  a.part_s = norms + (size_t)a.B * nb;
  a.part_r = a.part_s + (size_t)TR_NS * a.B * no;
  k_tr_load<<<nb * a.B, TR_BLOCK, 0, s>>>(g.Vh, nb, static_cast<const double2 *>(r), static_cast<const double2 *>(e), fr,
                                         fe, norms);
  QCU_CHECK_LAUNCH();
  k_tr_norms<<<a.B, TR_BLOCK, 0, s>>>(nb, norms, enorm);
  QCU_CHECK_LAUNCH();
  k_tr_even<<<nb * a.B, TR_BLOCK, 0, s>>>(g, a, nb);
  QCU_CHECK_LAUNCH();
  k_tr_odd<<<no * a.B, TR_BLOCK, 0, s>>>(g, a, no);
  QCU_CHECK_LAUNCH();
  QCU_CUDA(cudaFuncSetAttribute(k_tr_outer, cudaFuncAttributeMaxDynamicSharedMemorySize, TO_SMEM));
  k_tr_outer<<<nr, TO_THREADS, TO_SMEM, s>>>(g, a);
  QCU_CHECK_LAUNCH();
  k_tr_reduce<<<64 + TR_NS, TRR_BLOCK, 0, s>>>(a.part_r, nr, a.part_s, no * a.B, sums);
  QCU_CHECK_LAUNCH();
  k_tr_grads<<<1, NN_HOPS * 64, 0, s>>>(a.w1, a.w2, sums, grad);
  QCU_CHECK_LAUNCH();
}

}  // namespace qcu
