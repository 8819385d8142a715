// Clover term: build, pack, invert, apply.
//
// qcu's make_clover (src/clover_dslash.cu:5-837) forms, for each plane mu<nu,
// the four plaquette leaves Q_munu around x, F = Q - Q^dag, adds F into the
// 12x12 site matrix with the spin pattern of gamma_mu gamma_nu, and returns
// A = 1 - 1/8 sum (:826-835); inverse_clover (:839-855) then runs an
// unpivoted 12x12 Gauss-Jordan per site with a 288-entry local array, and
// give_clover (:857-882) multiplies densely.
//
// Here A is kept as what it is in the DeGrand-Rossi (chiral) basis: two
// Hermitian 6x6 blocks (spins {0,1} and {2,3}), 36 reals each -- 72 reals per
// site instead of 144 complex.  The inverse is an LDL^H factorisation per
// block (real pivots, no square roots, valid whenever the leading minors are
// non-zero, which is also what the unpivoted Gauss-Jordan requires), written
// back in the same packed form, and the apply is fused into the dslash
// epilogue (fields.cuh: clover_apply_site).  `coeff` scales the field-strength
// term: 1 reproduces qcu, kappa*csw gives the Sheikholeslami-Wohlert term.
#include "internal.h"

namespace qcu {

using C = Cpx<double>;

// acc += a b, acc += conj(a) b: four fused multiply-adds each
__device__ __forceinline__ void cmad(C &acc, const C &a, const C &b) {
  acc.re = fma(-a.im, b.im, fma(a.re, b.re, acc.re));
  acc.im = fma(a.im, b.re, fma(a.re, b.im, acc.im));
}
__device__ __forceinline__ void cmadc(C &acc, const C &a, const C &b) {
  acc.re = fma(a.im, b.im, fma(a.re, b.re, acc.re));
  acc.im = fma(-a.im, b.re, fma(a.re, b.im, acc.im));
}

// a <- a b and a <- a b^dag, row by row in place
__device__ __forceinline__ void mul_nn(C *a, const C *b) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const C u = a[r * 3], v = a[r * 3 + 1], w = a[r * 3 + 2];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      C t = u * b[k];
      cmad(t, v, b[3 + k]);
      cmad(t, w, b[6 + k]);
      a[r * 3 + k] = t;
    }
  }
}
__device__ __forceinline__ void mul_nd(C *a, const C *b) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const C u = a[r * 3], v = a[r * 3 + 1], w = a[r * 3 + 2];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      C t = cdotmul(b[k * 3], u);
      cmadc(t, b[k * 3 + 1], v);
      cmadc(t, b[k * 3 + 2], w);
      a[r * 3 + k] = t;
    }
  }
}
// d -= a^dag b
__device__ __forceinline__ void sub_dn(C *d, const C *a, const C *b) {
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const C m(-a[c * 3 + r].re, -a[c * 3 + r].im);
#pragma unroll
      for (int k = 0; k < 3; k++) cmadc(d[r * 3 + k], m, b[c * 3 + k]);
    }
}
// f += w - w^dag: the imaginary parts of the diagonal, then the entries (1,0), (2,0), (2,1)
__device__ __forceinline__ void add_antiherm(double f[9], const C *w) {
#pragma unroll
  for (int k = 0; k < 3; k++) f[k] += 2.0 * w[4 * k].im;
  f[3] += w[3].re - w[1].re;
  f[4] += w[3].im + w[1].im;
  f[5] += w[6].re - w[2].re;
  f[6] += w[6].im + w[2].im;
  f[7] += w[7].re - w[5].re;
  f[8] += w[7].im + w[5].im;
}

// a site by its full coordinates, and its neighbour one step (st = +1 or -1) along d, periodic
struct Pos {
  int x, y, z, t;
};
__device__ __forceinline__ int wrap_step(int v, int L, int st) {
  v += st;
  return v == L ? 0 : (v < 0 ? L - 1 : v);
}
__device__ __forceinline__ Pos step(const Geom &g, Pos c, int d, int st) {
  if (d == 0) c.x = wrap_step(c.x, 2 * g.Lxh, st);
  else if (d == 1) c.y = wrap_step(c.y, g.Ly, st);
  else if (d == 2) c.z = wrap_step(c.z, g.Lz, st);
  else c.t = wrap_step(c.t, g.Lt, st);
  return c;
}

// Links staged ahead of their use: a warp copies the rows 0 and 1 of its 32
// sites' links into its slots of shared memory (cp.async, 16 bytes a lane) and
// reads them back when their turn comes, two links later: no block barrier, and
// no registers held by loads in flight.  Packed links are contiguous over the
// sites, so every thread copies its own.  Of PyQuda's records (144 bytes apart)
// a request for one element of 32 sites would touch 32 lines: there the lanes
// take consecutive pieces of sixteen records at a time, and each reads its own
// record afterwards (96 bytes apart, rotated by one piece in every second four
// records against bank conflicts).  dslashCloverQcu needs no packed copy of the
// links for that: 24^3 x 48 540 us a call, against 629 with a thread per record
// and 547 when the links were packed first, into 768 B a site more of scratch.
constexpr int CL_SLOTS = 3;
constexpr int CL_SLOT_BYTES = 6 * 16 * 32;  // one warp's links
template <int G>
struct LinkStage {
  GaugeView<G> U;
  Geom g;
  unsigned slot0;  // the warp's slot 0
  const double2 *slot0p;
  int lane;
  // 16-byte unit of piece p in record r
  static __device__ __forceinline__ int unit(int r, int p) {
    p += (r >> 2) & 1;
    return r * 6 + (p >= 6 ? p - 6 : p);
  }
  static __device__ __forceinline__ void copy16(unsigned d, const double2 *p) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(p) : "memory");
  }
  // every lane calls it
  __device__ __forceinline__ void fetch(int i, const Pos &c, int mu) const {
    const int s = ((c.t * g.Lz + c.z) * g.Ly + c.y) * g.Lxh + (c.x >> 1);
    const int slab = mu * 2 + ((c.x + c.y + c.z + c.t) & 1);
    const unsigned d = slot0 + (i % CL_SLOTS) * CL_SLOT_BYTES;
    if constexpr (G == GAOS64) {
      const unsigned l = (unsigned)slab * (unsigned)U.stride + (unsigned)s;  // < 8 * 2^28
      __syncwarp();  // the link that lay here has been read
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const int j = (k % 3) * 32 + lane, r = j / 6, p = j % 6;
        copy16(d + (k / 3) * 16 * 96 + unit(r, p) * 16,
               static_cast<const double2 *>(U.p) + (size_t)__shfl_sync(0xffffffffu, l, 16 * (k / 3) + r) * 9 + p);
      }
    } else {
      const double2 *p = static_cast<const double2 *>(U.p) + (size_t)slab * U.stride * 6 + blk_base<6>(s);
#pragma unroll
      for (int k = 0; k < 6; k++) copy16(d + k * 512 + lane * 16, p + k * SB);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // link i, once at most `pending` later fetches are still in flight
  template <int PENDING>
  __device__ __forceinline__ void take(int i, C *m) const {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
    if constexpr (G == GAOS64) __syncwarp();  // the other lanes' pieces as well
    const double2 *p = slot0p + (i % CL_SLOTS) * (CL_SLOT_BYTES / 16);
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const double2 v = p[G == GAOS64 ? unit(lane, k) : k * 32 + lane];
      m[k] = C(v.x, v.y);
    }
    m[6] = row2(m[1], m[5], m[2], m[4]);
    m[7] = row2(m[2], m[3], m[0], m[5]);
    m[8] = row2(m[0], m[4], m[1], m[3]);
  }
  // conj(a b - c d), the cross product's component, in fused multiply-adds
  static __device__ __forceinline__ C row2(const C &a, const C &b, const C &c, const C &d) {
    C v = a * b;
    cmad(v, C(-c.re, -c.im), d);
    return v.conj();
  }
};

// Q - Q^dag of the plane (mu, nu) at c, Q the sum of the four plaquette
// leaves.  Two leaves begin with U_mu(x), two end with U_mu(x - mu), and a leaf
// may be replaced by minus its adjoint, so
//   W = U_mu(x) (S1 - S2) + (S3 - S4) U_mu(x - mu),   Q - Q^dag = W - W^dag
// with the staples
//   S1 = U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+         S3 = U_nu(x) U_mu(x-mu+nu)^+ U_nu(x-mu)^+
//   S2 = (U_mu(x-nu) U_nu(x+mu-nu))^+ U_nu(x-nu)   S4 = (U_mu(x-mu-nu) U_nu(x-nu))^+ U_nu(x-mu-nu)
// : ten 3x3 products a plane where the leaves one by one take twelve.
// The products run in place (three matrices live at a time).
template <int G>
__device__ __forceinline__ void clover_plane(const LinkStage<G> &S, const Pos &c, int mu, int nu, double f[9]) {
  const Geom &g = S.g;
  C a[9], b[9], d[9];
#pragma unroll
  for (int k = 0; k < 9; k++) f[k] = 0.0;
  const Pos xm = step(g, c, mu, -1), xn = step(g, c, nu, -1), xmn = step(g, xm, nu, -1);
  S.fetch(0, step(g, c, mu, 1), nu);
  S.fetch(1, step(g, c, nu, 1), mu);
  S.fetch(2, c, nu);
  S.template take<2>(0, d);
  S.template take<1>(1, b);
  mul_nd(d, b);
  S.fetch(3, xn, mu);
  S.fetch(4, step(g, xn, mu, 1), nu);
  S.template take<2>(2, b);
  mul_nd(d, b);
  S.fetch(5, xn, nu);
  S.template take<2>(3, a);
  S.template take<1>(4, b);
  mul_nn(a, b);
  S.fetch(6, c, mu);
  S.fetch(7, c, nu);
  S.template take<2>(5, b);
  sub_dn(d, a, b);
  S.fetch(8, step(g, xm, nu, 1), mu);
  S.template take<2>(6, a);
  mul_nn(a, d);
  add_antiherm(f, a);
  S.fetch(9, xm, nu);
  S.template take<2>(7, d);
  S.template take<1>(8, b);
  mul_nd(d, b);
  S.fetch(10, xmn, mu);
  S.fetch(11, xn, nu);
  S.template take<2>(9, b);
  mul_nd(d, b);
  S.fetch(12, xmn, nu);
  S.template take<2>(10, a);
  S.template take<1>(11, b);
  mul_nn(a, b);
  S.fetch(13, xm, mu);
  S.template take<1>(12, b);
  sub_dn(d, a, b);
  S.template take<0>(13, a);
  mul_nn(d, a);
  add_antiherm(f, d);
}

// packed lower triangle of a Hermitian 6x6 block: diagonal d, (i, j), i > j, at tri(i, j)
__host__ __device__ constexpr int tri(int i, int j) { return i * (i - 1) / 2 + j; }

// Chiral block B (spins 2B, 2B+1) of A = 1 + scale sum_{mu<nu} gamma_mu
// gamma_nu F_munu from the six planes' F of one site (F[9 * plane + e] at
// stride SB); only the lower triangle is formed.
template <int B>
__device__ __forceinline__ void clover_block(const double *F, double scale, double d[6], C L[15]) {
#pragma unroll
  for (int k = 0; k < 6; k++) d[k] = 0.0;
#pragma unroll
  for (int k = 0; k < 15; k++) L[k] = C(0, 0);
  int plane = 0;
#pragma unroll
  for (int mu = 0; mu < 4; mu++)
#pragma unroll
    for (int nu = mu + 1; nu < 4; nu++, plane++) {
      double f[9];
#pragma unroll
      for (int e = 0; e < 9; e++) f[e] = F[(plane * 9 + e) * SB];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int s0 = 2 * B + h;
        const int j = gcol(mu, s0), s1 = gcol(nu, j);
        const int vr = gre(mu, s0) * gre(nu, j) - gim(mu, s0) * gim(nu, j);
        const int vi = gre(mu, s0) * gim(nu, j) + gim(mu, s0) * gre(nu, j);
        const int r0 = h * 3, c0 = (s1 & 1) * 3;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int k = 0; k < 3; k++) {
            if (r0 + i < c0 + k) continue;
            const int e = i > k ? 3 + 2 * tri(i, k) : 3 + 2 * tri(k, i);
            const C v = i == k ? C(0.0, f[i]) : (i > k ? C(f[e], f[e + 1]) : C(-f[e], f[e + 1]));
            // times vr + i vi, one of 1, -1, i, -i (known when unrolled)
            const C u = vr == 1 ? v : (vr == -1 ? -v : (vi == 1 ? C(-v.im, v.re) : C(v.im, -v.re)));
            if (r0 + i == c0 + k) d[r0 + i] += u.re;
            else L[tri(r0 + i, c0 + k)] += u;
          }
      }
    }
#pragma unroll
  for (int k = 0; k < 6; k++) d[k] = 1.0 + d[k] * scale;
#pragma unroll
  for (int k = 0; k < 15; k++) L[k] = L[k] * scale;
}

// In place: the block A (d, L) -> M = L^-1 of A = L D L^H and 1 / D, so that
// A^-1 = M^H D^-1 M.  False on a zero or undefined pivot.
__device__ __forceinline__ bool ldl6(double d[6], C L[15]) {
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 6; j++) {
#pragma unroll
    for (int k = 0; k < j; k++) d[j] -= L[tri(j, k)].norm2() * d[k];
    ok = ok && d[j] != 0.0 && d[j] == d[j];
    const double inv = 1.0 / d[j];
#pragma unroll
    for (int i = j + 1; i < 6; i++) {
      C v = L[tri(i, j)];
#pragma unroll
      for (int k = 0; k < j; k++) v -= L[tri(i, k)] * L[tri(j, k)].conj() * d[k];
      L[tri(i, j)] = v * inv;
    }
  }
  // M_ij = -(L_ij + sum_{j<k<i} L_ik M_kj): row by row, columns upwards, so
  // that every L_ik (k > j) is read before it is overwritten
#pragma unroll
  for (int i = 1; i < 6; i++)
#pragma unroll
    for (int j = 0; j < i; j++) {
      C v = L[tri(i, j)];
#pragma unroll
      for (int k = j + 1; k < i; k++) v += L[tri(i, k)] * L[tri(k, j)];
      L[tri(i, j)] = -v;
    }
#pragma unroll
  for (int k = 0; k < 6; k++) d[k] = 1.0 / d[k];
  return ok;
}

// entry (i, j), i >= j, of M^H D^-1 M
__device__ __forceinline__ C inv6_entry(const double d[6], const C L[15], int i, int j) {
  C v(0, 0);
#pragma unroll
  for (int k = i; k < 6; k++) {
    const C a = k == i ? C(d[k], 0.0) : L[tri(k, i)].conj() * d[k];
    if (k == j) v += a;
    else v += a * L[tri(k, j)];
  }
  return v;
}

// Writes one block in the packed form (18 double2: the diagonal in pairs, then
// the lower triangle row by row), also as 9 float4 where o32 is given; entry(k)
// returns double2 k.
template <typename F>
__device__ __forceinline__ void block_write(double2 *o64, float4 *o32, F entry) {
#pragma unroll
  for (int k = 0; k < 18; k += 2) {
    const double2 u = entry(k), w = entry(k + 1);
    o64[k * SB] = u;
    o64[(k + 1) * SB] = w;
    if (o32) o32[(k / 2) * SB] = make_float4((float)u.x, (float)u.y, (float)w.x, (float)w.y);
  }
}

template <int B>
__device__ __forceinline__ void clover_finish(const double *F, double scale, int s, const CloverOut &o, int q) {
  double d[6];
  C L[15];
  clover_block<B>(F, scale, d, L);
  constexpr int row[15] = {1, 2, 2, 3, 3, 3, 4, 4, 4, 4, 5, 5, 5, 5, 5};
  constexpr int col[15] = {0, 0, 1, 0, 1, 2, 0, 1, 2, 3, 0, 1, 2, 3, 4};
  // selected, not indexed: a run-time index would copy the parameters to local memory
  void *const A64 = q ? o.A64[1] : o.A64[0], *const Ainv64 = q ? o.Ainv64[1] : o.Ainv64[0],
       *const Ainv32 = q ? o.Ainv32[1] : o.Ainv32[0];
  if (A64)
    block_write(static_cast<double2 *>(A64) + blk_base<36>(s) + B * 18 * SB, nullptr, [&](int k) {
      return k < 3 ? make_double2(d[2 * k], d[2 * k + 1]) : make_double2(L[k - 3].re, L[k - 3].im);
    });
  if (!Ainv64) return;
  const bool ok = ldl6(d, L);
  if (!ok) atomicAdd(o.bad, 1);
  float4 *o32 = Ainv32 ? static_cast<float4 *>(Ainv32) + blk_base<18>(s) + B * 9 * SB : nullptr;
  block_write(static_cast<double2 *>(Ainv64) + blk_base<36>(s) + B * 18 * SB, o32, [&](int k) {
    if (!ok) return make_double2(0.0, 0.0);
    if (k < 3) return make_double2(inv6_entry(d, L, 2 * k, 2 * k).re, inv6_entry(d, L, 2 * k + 1, 2 * k + 1).re);
    const C v = inv6_entry(d, L, row[k - 3], col[k - 3]);
    return make_double2(v.re, v.im);
  });
}

// The clover term and its inverse, 32 sites of one parity at a time: warp p
// forms plane p's F for the sites (lane = site, so the loads of the
// site-blocked links are contiguous and nothing diverges).  After `groups`
// (1 or 3) such rounds a warp per 32 sites and chiral block assembles,
// factorises and writes it: with three rounds all six warps have one.  Bound
// by FP64 arithmetic (10 products and 14 link reconstructions a plane, 1.4
// kFMA, and ~1.4 kFMA a chiral block) at the latency of its link loads; a
// thread per site and plane keeps the working set (three 3x3 matrices and a
// sum) in registers, where one thread for all planes held the 72-entry blocks
// as well and its leaves went through a call with local arrays (24^3 x 48,
// one parity: 1158 -> 341 us on packed links, FP64 pipe 58 % busy; 387 us on
// PyQuda's records, 48 %).
constexpr int CB_THREADS = 192;
constexpr int CB_GROUPS = 3;
constexpr int CB_SMEM = (CB_THREADS / 32) * CL_SLOTS * CL_SLOT_BYTES + CB_GROUPS * 6 * 9 * SB * (int)sizeof(double);
template <int G>
__global__ void __launch_bounds__(CB_THREADS, 2) k_clover_build(Geom g, GaugeView<G> U, double scale, CloverOut o,
                                                               int groups) {
  extern __shared__ __align__(16) unsigned char cb_smem[];
  double *F = reinterpret_cast<double *>(cb_smem + (CB_THREADS / 32) * CL_SLOTS * CL_SLOT_BYTES);  // [group][9 plane + e][site]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s0 = blockIdx.x * groups * SB, q = blockIdx.y;
  const int mu = warp < 3 ? 0 : (warp < 5 ? 1 : 2), nu = warp < 3 ? warp + 1 : (warp < 5 ? warp - 1 : 3);
  unsigned char *slot = cb_smem + warp * CL_SLOTS * CL_SLOT_BYTES;
  const LinkStage<G> S{U, g, (unsigned)__cvta_generic_to_shared(slot), reinterpret_cast<const double2 *>(slot), lane};
  for (int k = 0; k < groups; k++) {
    if (s0 + k * SB >= g.Vh) break;
    const int s = min(s0 + k * SB + lane, g.Vh - 1);  // lanes past the end copy for the others
    Pos c;
    int xh;
    site_coords(g, s, xh, c.y, c.z, c.t);
    c.x = 2 * xh + ((c.y + c.z + c.t + o.par0 + q) & 1);
    double f[9];
    clover_plane<G>(S, c, mu, nu, f);
#pragma unroll
    for (int e = 0; e < 9; e++) F[((k * 6 + warp) * 9 + e) * SB + lane] = f[e];
  }
  __syncthreads();
  const int k = warp >> 1, s = s0 + k * SB + lane;
  if (k >= groups || s >= g.Vh) return;
  const double *Fk = F + k * 6 * 9 * SB + lane;
  if (warp & 1) clover_finish<1>(Fk, scale, s, o, q);
  else clover_finish<0>(Fk, scale, s, o, q);
}

template <int K>
__global__ void k_clover_apply(int Vh, CloverView<CSOA64> cv, const void *in, void *out) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < Vh; s += gridDim.x * blockDim.x) {
    Cpx<double> v[12];
    spinor_load<K, double>(SpinorView<K>{const_cast<void *>(in), nullptr, Vh}, s, v);
    clover_apply_site<CSOA64, double>(cv, s, v);
    spinor_store<K, double>(SpinorView<K>{out, nullptr, Vh}, s, v);
  }
}

size_t clover_bytes(int ckind, int Vh) { return (size_t)2 * (ckind == CSOA64 ? 18 * 16 : 9 * 16) * pad_sites(Vh); }

void launch_clover_build(int gkind, const Geom &g, const void *gauge, int nparities, double coeff, const CloverOut &o,
                         int sms, cudaStream_t s) {
  // three rounds a block once that still fills every SM with its two blocks
  // twice (below, the shorter blocks finish sooner than the balance of the last
  // phase gains)
  const int blocks = (g.Vh + SB - 1) / SB;
  const int groups = (int64_t)blocks * nparities >= (int64_t)sms * 2 * CB_GROUPS * 2 ? CB_GROUPS : 1;
  const dim3 grid((blocks + groups - 1) / groups, nparities);
  auto run = [&](auto kernel, auto view) {
    QCU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CB_SMEM));
    kernel<<<grid, CB_THREADS, CB_SMEM, s>>>(g, view, -0.125 * coeff, o, groups);
  };
  if (gkind == GSOA64) run(k_clover_build<GSOA64>, GaugeView<GSOA64>{gauge, pad_sites(g.Vh)});
  else if (gkind == GAOS64) run(k_clover_build<GAOS64>, GaugeView<GAOS64>{gauge, g.Vh});
  else throw Error(1, "clover build: unsupported gauge kind");
  QCU_CHECK_LAUNCH();
}

void launch_clover_apply(int kind, int Vh, const void *c64, const void *in, void *out, cudaStream_t s) {
  const CloverView<CSOA64> cv{c64, Vh};
  if (kind == AOS64) k_clover_apply<AOS64><<<blas_grid(Vh), BLAS_BLOCK, 0, s>>>(Vh, cv, in, out);
  else if (kind == SOA64) k_clover_apply<SOA64><<<blas_grid(Vh), BLAS_BLOCK, 0, s>>>(Vh, cv, in, out);
  else throw Error(1, "clover apply: unsupported spinor kind");
  QCU_CHECK_LAUNCH();
}

}  // namespace qcu
