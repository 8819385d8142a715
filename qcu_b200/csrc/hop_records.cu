// The FP64 hopping term on PyQuda-layout fields (dslashQcu's path): spinor
// records of 192 bytes, link records of 144 (rows 0 and 1 are read).
//
// A thread that reads its own records touches 32 lines with every request of
// its warp: at 32^3 x 64 the L1 was 92 % busy with those lookups and DRAM 60 %.
// Here a warp copies the 32 records that its sites need for one hop with
// cp.async, lanes on consecutive 16-byte pieces (5 to 8 lines a request), into
// one of two stages of shared memory, two hops ahead of their use; each lane
// then takes its own record from there (the records' pieces are rotated by the
// record's number, spin_unit and link_unit, so that a column of records is read
// without bank conflicts; padding the records to odd pitches measured 282 us).
// The copies hold no registers, need no block barrier, and follow the neighbour
// index of any lattice, wraps included.  The result leaves through the same
// stage.  Bound by DRAM, which reads the links' records whole (1.43 + 0.19 GB at
// 32^3 x 64, 250 us): 278 us, 5.8 TB/s, against 303 us for a thread per record.
// Two blocks an SM: with three the stages leave no L1, and neighbours' records
// come from L2 again (389 us).
#include "internal.h"

namespace qcu {
namespace {

constexpr int HR_WARPS = 4;
constexpr int HR_SPIN = 12 * 16, HR_LINK = 6 * 16;  // bytes of a staged record
constexpr int HR_STAGE = 32 * (HR_SPIN + HR_LINK);
constexpr int HR_SMEM = HR_WARPS * 2 * HR_STAGE;

struct HopArgs {
  const double2 *in, *gauge;
  double2 *out;
  int par;
  double t_bc;
};

__device__ __forceinline__ void cp16(unsigned dst, const double2 *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// hop I: direction I / 2, forward when even (the order of wilson_hop_site)
template <int I>
__device__ __forceinline__ int hop_site(const Geom &g, int s, int xh, int y, int z, int t, int xodd) {
  if constexpr (I == 0) return xodd ? (xh == g.Lxh - 1 ? s - xh : s + 1) : s;
  else if constexpr (I == 1) return xodd ? s : (xh == 0 ? s + g.Lxh - 1 : s - 1);
  else if constexpr (I == 2) return y == g.Ly - 1 ? s - (g.Ly - 1) * g.sy : s + g.sy;
  else if constexpr (I == 3) return y == 0 ? s + (g.Ly - 1) * g.sy : s - g.sy;
  else if constexpr (I == 4) return z == g.Lz - 1 ? s - (g.Lz - 1) * g.sz : s + g.sz;
  else if constexpr (I == 5) return z == 0 ? s + (g.Lz - 1) * g.sz : s - g.sz;
  else if constexpr (I == 6) return t == g.Lt - 1 ? s - (g.Lt - 1) * g.st : s + g.st;
  else return t == 0 ? s + (g.Lt - 1) * g.st : s - g.st;
}

// 16-byte unit of piece p in record r
__device__ __forceinline__ int spin_unit(int r, int p) {
  p += (r >> 1) & 3;
  return r * 12 + (p >= 12 ? p - 12 : p);
}
__device__ __forceinline__ int link_unit(int r, int p) {
  p += (r >> 2) & 1;
  return r * 6 + (p >= 6 ? p - 6 : p);
}

struct HopWarp {
  Geom g;
  HopArgs a;
  unsigned stage;           // shared address of the warp's stages
  const unsigned char *sp;  // the same as a pointer
  int lane, s, xh, y, z, t, xodd;
  int rs[3], ps[3], rl[3], pl[3];  // record and piece of this lane's share, spinors and links
  int us[3], ul[3];                // their units (8 spinor or 16 link records on: the same rotation)

  template <int I>
  __device__ __forceinline__ void fetch() const {
    if constexpr (I < 8) {
      const int n = hop_site<I>(g, s, xh, y, z, t, xodd);
      const unsigned d = stage + (I & 1) * HR_STAGE;
#pragma unroll
      for (int k = 0; k < 12; k++) {  // 12 pieces a record: three requests cover eight records
        const int r = 8 * (k / 3) + rs[k % 3];
        cp16(d + (k / 3 * 8 * 12 + us[k % 3]) * 16, a.in + (size_t)__shfl_sync(0xffffffffu, n, r) * 12 + ps[k % 3]);
      }
      const int l = (I & 1) ? n : s;  // the link lives on the site the hop starts from, or comes from
      const size_t slab = (size_t)((I >> 1) * 2 + ((I & 1) ? 1 - a.par : a.par)) * g.Vh;
#pragma unroll
      for (int k = 0; k < 6; k++) {  // 6 pieces a record: three requests cover sixteen records
        const int r = 16 * (k / 3) + rl[k % 3];
        cp16(d + 32 * HR_SPIN + (k / 3 * 16 * 6 + ul[k % 3]) * 16,
             a.gauge + (slab + __shfl_sync(0xffffffffu, l, r)) * 9 + pl[k % 3]);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  template <int I>
  __device__ __forceinline__ void take(Cpx<double> acc[12]) const {
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // all but the newest group: hop I's has landed
    __syncwarp();
    const double2 *p = reinterpret_cast<const double2 *>(sp + (I & 1) * HR_STAGE);
    const double2 *q = reinterpret_cast<const double2 *>(sp + (I & 1) * HR_STAGE + 32 * HR_SPIN);
    Cpx<double> psi[12], u[9];
#pragma unroll
    for (int k = 0; k < 12; k++) {
      const double2 v = p[spin_unit(lane, k)];
      psi[k] = Cpx<double>(v.x, v.y);
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const double2 v = q[link_unit(lane, k)];
      u[k] = Cpx<double>(v.x, v.y);
    }
    __syncwarp();  // the stage is read: hop I + 2 may have it
    fetch<I + 2>();
    u[6] = (u[1] * u[5] - u[2] * u[4]).conj();
    u[7] = (u[2] * u[3] - u[0] * u[5]).conj();
    u[8] = (u[0] * u[4] - u[1] * u[3]).conj();
    const double ph = (I == 6 && t == g.Lt - 1) || (I == 7 && t == 0) ? a.t_bc : 1.0;
    hop<(I >> 1), (I & 1) == 0, (I >> 1) == 3, double>(acc, psi, u, ph);
  }
};

__global__ void __launch_bounds__(HR_WARPS * 32, 2) k_hop_records(Geom g, HopArgs a) {
  extern __shared__ __align__(16) unsigned char hr_smem[];
  HopWarp w;
  w.g = g;
  w.a = a;
  w.lane = threadIdx.x & 31;
  const int s0 = (blockIdx.x * HR_WARPS + (threadIdx.x >> 5)) * 32;
  if (s0 >= g.Vh) return;
  w.s = min(s0 + w.lane, g.Vh - 1);  // lanes past the end repeat the last site and store nothing
  unsigned char *sp = hr_smem + (threadIdx.x >> 5) * 2 * HR_STAGE;
  w.sp = sp;
  w.stage = (unsigned)__cvta_generic_to_shared(sp);
  site_coords(g, w.s, w.xh, w.y, w.z, w.t);
  w.xodd = (w.y + w.z + w.t + a.par) & 1;
#pragma unroll
  for (int b = 0; b < 3; b++) {
    w.rs[b] = (32 * b + w.lane) / 12;
    w.ps[b] = (32 * b + w.lane) % 12;
    w.rl[b] = (32 * b + w.lane) / 6;
    w.pl[b] = (32 * b + w.lane) % 6;
    w.us[b] = spin_unit(w.rs[b], w.ps[b]);
    w.ul[b] = link_unit(w.rl[b], w.pl[b]);
  }
  Cpx<double> acc[12];
#pragma unroll
  for (int k = 0; k < 12; k++) acc[k] = Cpx<double>(0, 0);
  w.fetch<0>();
  w.fetch<1>();
  w.take<0>(acc);
  w.take<1>(acc);
  w.take<2>(acc);
  w.take<3>(acc);
  w.take<4>(acc);
  w.take<5>(acc);
  w.take<6>(acc);
  w.take<7>(acc);
  __syncwarp();
  double2 *o = reinterpret_cast<double2 *>(sp);
#pragma unroll
  for (int k = 0; k < 12; k++) o[spin_unit(w.lane, k)] = make_double2(acc[k].re, acc[k].im);
  __syncwarp();
  const int n = min(32, g.Vh - s0) * 12;
#pragma unroll
  for (int k = 0; k < 12; k++) {
    const int r = 8 * (k / 3) + w.rs[k % 3], p = w.ps[k % 3];
    if (r * 12 + p < n) a.out[(size_t)s0 * 12 + r * 12 + p] = o[k / 3 * 8 * 12 + w.us[k % 3]];
  }
}

}  // namespace

void launch_hop_records(const Geom &g, const void *in, void *out, const void *gauge, int par, double t_bc,
                        Context &ctx, cudaStream_t s) {
  const HopArgs a{static_cast<const double2 *>(in), static_cast<const double2 *>(gauge), static_cast<double2 *>(out), par,
                  t_bc};
  if (!ctx.hop_records_smem) {  // once, not per call: 0.3 us of the 20 us of a call at 8^4
    QCU_CUDA(cudaFuncSetAttribute(k_hop_records, cudaFuncAttributeMaxDynamicSharedMemorySize, HR_SMEM));
    ctx.hop_records_smem = true;
  }
  k_hop_records<<<(g.Vh + HR_WARPS * 32 - 1) / (HR_WARPS * 32), HR_WARPS * 32, HR_SMEM, s>>>(g, a);
  QCU_CHECK_LAUNCH();
}

}  // namespace qcu
