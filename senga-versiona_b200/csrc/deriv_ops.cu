// Operator-level derivative family (DFBYDX..D2FDYZ) of one field: the
// reference's call surfaces FUNCTN -> FDERIV (src/dfbydx.f:36-37, 53-238;
// src/d2fdx2.f:54-270; src/d2fdxy.f:55-1937), on interior arrays (BIG =
// false; periodic neighbours folded into the domain) or on halo-extended
// ones (BIG = true; five points per side, read as the caller filled them).
//
// What bounds them: the latency of the neighbours' loads (6 to 10 warps wait for
// one per issue, at half the warp slots; L1 31 to 62% busy, DRAM 8 to 12%). The
// floor is 16 bytes a point, 9 us for a 192 x 160 x 120 field at 6.5 TB/s. So
// what has to go is everything else: one thread marches over the z planes of
// its (x, y), with the in-plane neighbour offsets folded once into registers,
// and the z operators slide a register window so that every value is loaded
// (ZB + 10) / ZB times. One thread per point with a 64-bit index decode and
// a fold per neighbour took 543 us of device time for the nine operators on
// that field; this form takes 243 us (64^3: 57 and 45, 47x153x61: 85 and 59).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "senga_internal.h"
#include "stencil.cuh"

namespace senga {
namespace {

constexpr int H = 5;
constexpr int kThreads = 256;
constexpr int kMaxZB = 16;

// element strides of the operand: the interior array, or the halo-extended
// one with its origin at the first interior point
struct InLay {
  int64_t base;  // offset of interior point (0, 0, 0)
  int sy;        // row stride
  int64_t sz;    // plane stride
};

// The block covers blockDim.x x blockDim.y points of a plane, and blockDim.z
// marches of zb planes each.
struct Where {
  int x, y;
  bool in;
};
__device__ __forceinline__ Where where(const Geo& g, int ntx) {
  const int bx = (int)(blockIdx.x % (unsigned)ntx), by = (int)(blockIdx.x / (unsigned)ntx);
  Where w;
  w.x = bx * (int)blockDim.x + (int)threadIdx.x;
  w.y = by * (int)blockDim.y + (int)threadIdx.y;
  w.in = w.x < g.nx && w.y < g.ny;
  return w;
}
// first march of this thread, and the distance to its next one, in marches
__device__ __forceinline__ int64_t first_march() { return (int64_t)blockIdx.y * blockDim.z + threadIdx.z; }
__device__ __forceinline__ int64_t march_step() { return (int64_t)gridDim.y * blockDim.z; }

// distance in elements to the point m steps away along a direction of extent
// n: folded (any extent, also shorter than the stencil), or as it is
template <bool BIG>
__device__ __forceinline__ int fold_off(int c, int m, int n, int st) {
  int cm = c + m;
  if (!BIG) {
    if (n > H) {
      cm = cm < 0 ? cm + n : cm >= n ? cm - n : cm;
    } else {
      cm %= n;
      if (cm < 0) cm += n;
    }
  }
  return (cm - c) * st;
}

// x and y operators: ORD 1 or 2 along D (0 or 1). At four blocks an SM and one
// plane a turn: two planes a turn took 76 registers, three blocks, and the
// second y derivative 9.4 instead of 7.0 us on 80^3, 40 instead of 26 on
// 192x160x120.
template <bool BIG, int D, int ORD>
__global__ void __launch_bounds__(kThreads, 4) k_plane_op(Geo g, InLay il, int ntx, int zb, const double* __restrict__ in,
                                                       double* __restrict__ out) {
  const Where w = where(g, ntx);
  if (!w.in) return;
  const int c = D == 0 ? w.x : w.y, n = D == 0 ? g.nx : g.ny, st = D == 0 ? 1 : il.sy;
  const int64_t plane = (int64_t)g.nx * g.ny;
  const double* const p0 = in + il.base + w.x + (int64_t)w.y * il.sy;
  double* const o0 = out + w.x + (int64_t)w.y * g.nx;
  const double sc = ORD == 1 ? g.ovd[D] : g.ovd2[D];
  int off[2 * H + 1];
#pragma unroll
  for (int m = -H; m <= H; ++m) off[m + H] = fold_off<BIG>(c, m, n, st);
  for (int64_t z0 = first_march() * zb; z0 < g.nz; z0 += march_step() * zb) {
    const int z1 = (int)(z0 + zb < g.nz ? z0 + zb : g.nz);
    if (g.per[D]) {
#pragma unroll 1
      for (int z = (int)z0; z < z1; ++z) {
        const double* const p = p0 + z * il.sz;
        auto v = [&](int m) { return __ldg(p + off[m + H]); };
        o0[z * plane] = (ORD == 1 ? d1core(v, c, n, 1) : d2core(v, c, n, 1)) * sc;
      }
    } else {  // the closures read inward only: no fold
      for (int z = (int)z0; z < z1; ++z) {
        const double* const p = p0 + z * il.sz;
        auto v = [&](int m) { return __ldg(p + m * st); };
        o0[z * plane] = (ORD == 1 ? d1core(v, c, n, 0) : d2core(v, c, n, 0)) * sc;
      }
    }
  }
}

// z operators: a window of ZB + 10 values of the thread's column
template <bool BIG, int ORD, int ZB>
__global__ void __launch_bounds__(kThreads) k_z_op(Geo g, InLay il, int ntx, const double* __restrict__ in,
                                                   double* __restrict__ out) {
  const Where w = where(g, ntx);
  if (!w.in) return;
  const int64_t plane = (int64_t)g.nx * g.ny;
  const double* const p0 = in + il.base + w.x + (int64_t)w.y * il.sy;
  double* const o0 = out + w.x + (int64_t)w.y * g.nx;
  const double sc = ORD == 1 ? g.ovd[2] : g.ovd2[2];
  for (int64_t z0 = first_march() * ZB; z0 < g.nz; z0 += march_step() * ZB) {
    if (g.per[2]) {
      double c[ZB + 2 * H];
#pragma unroll
      for (int k = 0; k < ZB + 2 * H; ++k) {
        int z = (int)z0 + k - H;
        if (BIG) {  // past the last point's halo: unused
          z = z < g.nz + H ? z : g.nz + H - 1;
        } else if (g.nz >= ZB + H) {  // one fold reaches every plane of the window
          z = z < 0 ? z + g.nz : z >= g.nz ? z - g.nz : z;
        } else {
          z %= g.nz;
          if (z < 0) z += g.nz;
        }
        c[k] = __ldg(p0 + z * il.sz);
      }
#pragma unroll
      for (int k = 0; k < ZB; ++k) {
        if (z0 + k >= g.nz) break;
        auto v = [&](int m) { return c[k + m + H]; };
        o0[(z0 + k) * plane] = (ORD == 1 ? d1core(v, 0, g.nz, 1) : d2core(v, 0, g.nz, 1)) * sc;
      }
    } else {
      for (int k = 0; k < ZB && z0 + k < g.nz; ++k) {
        const int z = (int)z0 + k;
        const double* const p = p0 + z * il.sz;
        auto v = [&](int m) { return __ldg(p + m * il.sz); };
        o0[z * plane] = (ORD == 1 ? d1core(v, z, g.nz, 0) : d2core(v, z, g.nz, 0)) * sc;
      }
    }
  }
}

// mixed operators of two periodic directions (DA < DB)
template <bool BIG, int DA, int DB>
__global__ void __launch_bounds__(kThreads) k_mixed_op(Geo g, InLay il, int ntx, int zb, const double* __restrict__ in,
                                                       double* __restrict__ out) {
  // plane offsets of the block's z windows, one row per march (DB = z)
  extern __shared__ int64_t oz[];
  const Where w = where(g, ntx);
  const int64_t plane = (int64_t)g.nx * g.ny;
  const double* const p0 = in + il.base + w.x + (int64_t)w.y * il.sy;
  double* const o0 = out + w.x + (int64_t)w.y * g.nx;
  const double sa = g.ovd[DA], sb = g.ovd[DB];
  const int nw = zb + 2 * H;
  int oa[2 * H + 1], ob[2 * H + 1];
#pragma unroll
  for (int m = -H; m <= H; ++m) {
    oa[m + H] = w.in ? fold_off<BIG>(DA == 0 ? w.x : w.y, m, DA == 0 ? g.nx : g.ny, DA == 0 ? 1 : il.sy) : 0;
    if (DB == 1) ob[m + H] = w.in ? fold_off<BIG>(w.y, m, g.ny, il.sy) : 0;
  }
  // every thread of the block takes the same number of steps (barriers)
  for (int64_t m0 = (int64_t)blockIdx.y * blockDim.z; m0 * zb < g.nz; m0 += march_step()) {
    const int64_t z0 = (m0 + threadIdx.z) * zb;
    const int z1 = (int)(z0 + zb < g.nz ? z0 + zb : g.nz);
    if (DB == 2) {
      __syncthreads();
      const int nt = (int)(blockDim.x * blockDim.y * blockDim.z);
      for (int t = (int)(threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z)); t < nw * (int)blockDim.z;
           t += nt) {
        int64_t z = (m0 + t / nw) * zb + t % nw - H;
        if (BIG) {  // past the last point's halo: unused
          z = z < g.nz + H ? z : g.nz + H - 1;
        } else {
          z %= g.nz;
          if (z < 0) z += g.nz;
        }
        oz[t] = z * il.sz;
      }
      __syncthreads();
    }
    if (!w.in) continue;
    for (int z = (int)z0; z < z1; ++z) {
      double r;
      if (DB == 1) {
        const double* const p = p0 + z * il.sz;
        r = dmcore([&](int ma, int mb) { return __ldg(p + (oa[ma + H] + ob[mb + H])); });
      } else {
        const int64_t* const o = oz + (int)threadIdx.z * nw + (z - (int)z0) + H;
        r = dmcore([&](int ma, int mb) { return __ldg(p0 + o[mb] + oa[ma + H]); });
      }
      o0[z * plane] = r * sa * sb;
    }
  }
}

// mixed operators with a bounded direction (edge rows and corners)
template <bool BIG>
__global__ void __launch_bounds__(kThreads) k_mixed_ends(Geo g, InLay il, int kind, const double* __restrict__ in,
                                                         double* __restrict__ out) {
  const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (q >= g.n) return;
  const Pt pt = point_of(g, q);
  if (!BIG) {
    const Ld F{in};
    out[q] = kind == 6 ? DM<0, 1>(g, pt, F) : kind == 7 ? DM<0, 2>(g, pt, F) : DM<1, 2>(g, pt, F);
    return;
  }
  const double* const p = in + il.base + pt.i + (int64_t)pt.j * il.sy + pt.k * il.sz;
  const int64_t st[3] = {1, il.sy, il.sz};
  const int c3[3] = {pt.i, pt.j, pt.k};
  const int n3[3] = {g.nx, g.ny, g.nz};
  const int da = kind == 8 ? 1 : 0, db = kind == 6 ? 1 : 2;
  auto v = [&](int ma, int mb) { return __ldg(p + ma * st[da] + mb * st[db]); };
  double r;
  if (!g.per[db]) {
    constexpr int kFar = 1 << 20;
    const int ca = c3[da], cb = c3[db];
    const int la = g.per[da] ? kFar : ca, ra = g.per[da] ? kFar : n3[da] - 1 - ca;
    const int lb = cb, rb = n3[db] - 1 - cb;
    r = dmcore_ends(v, la < ra ? la : ra, ra < la, lb < rb ? lb : rb, rb < lb);
  } else {
    r = dmcore_b(v, c3[da], n3[da]);
  }
  out[q] = r * g.ovd[da] * g.ovd[db];
}

// n points in equal parts of at most `most`: the size of a part
int even_part(int n, int most) {
  const int parts = (n + most - 1) / most;
  return (n + parts - 1) / parts;
}

template <bool BIG>
void launch(const Geo& g, int kind, const double* in, double* out, cudaStream_t s) {
  InLay il{0, g.nx, (int64_t)g.nx * g.ny};
  if (BIG) {
    il.sy = g.nx + 2 * H;
    il.sz = (int64_t)il.sy * (g.ny + 2 * H);
    il.base = H + (int64_t)H * il.sy + H * il.sz;
  }
  const int da = kind == 8 ? 1 : 0, db = kind == 6 ? 1 : 2;
  if (kind >= 6 && !(g.per[da] && g.per[db])) {
    k_mixed_ends<BIG><<<(unsigned)((g.n + kThreads - 1) / kThreads), kThreads, 0, s>>>(g, il, kind, in, out);
    return;
  }
  // About 32 x 8 points of a plane per block (wider or taller on thin boxes),
  // in equal parts of the extents: a fixed 32 x 8 left a third of the threads
  // of a 47 x 153 plane without a point. 16 x 16 where that fits and 32 does
  // not: rows of whole warps (48^3: 30 us for the nine operators, 34 with 24
  // points a row).
  const int bx = even_part(g.nx, g.ny < 8 ? kThreads / g.ny : g.nx % 32 == 16 ? 16 : 32), by = even_part(g.ny, kThreads / bx);
  const int64_t ntx = (g.nx + bx - 1) / bx, nty = (g.ny + by - 1) / by;
  // Planes a thread marches over: as many as leave the chip 75 thousand
  // threads, a quarter of what it holds (148 SMs x 2048), twice that for the y
  // operators, whose eleven rows come from L2 more than the others' values. A
  // march of one plane spends its time on the folds: with marches that left
  // 300 thousand threads, and fixed blocks, 80^3 took 112 us, 120x100x90 152;
  // so 59 and 100 (one thread per point: 95 and 181).
  int zb = 1;
  const bool zop = kind == 2 || kind == 5;
  const int most = zop ? kMaxZB : 8;
  const int64_t fewest = kind == 1 || kind == 4 ? 150000 : 75000;
  while (zb < most && g.n / (2 * zb) >= fewest) zb *= 2;
  if (zop) zb = zb >= 16 ? 16 : zb >= 4 ? 4 : 1;
  // and several marches per block where the plane is smaller than a block
  const int64_t nzb = (g.nz + zb - 1) / zb;
  const int bz = (int)std::min<int64_t>({nzb, 64, kThreads / (bx * by)});
  const int64_t nzg = (nzb + bz - 1) / bz;
  const dim3 grid((unsigned)(ntx * nty), (unsigned)(nzg < 65535 ? nzg : 65535)), block(bx, by, bz);
  const size_t wb = (size_t)bz * (zb + 2 * H) * sizeof(int64_t);  // the z windows of a block
  const int nt = (int)ntx;
  switch (kind) {
    case 0: k_plane_op<BIG, 0, 1><<<grid, block, 0, s>>>(g, il, nt, zb, in, out); break;
    case 1: k_plane_op<BIG, 1, 1><<<grid, block, 0, s>>>(g, il, nt, zb, in, out); break;
    case 3: k_plane_op<BIG, 0, 2><<<grid, block, 0, s>>>(g, il, nt, zb, in, out); break;
    case 4: k_plane_op<BIG, 1, 2><<<grid, block, 0, s>>>(g, il, nt, zb, in, out); break;
    case 2:
      if (zb == 16) k_z_op<BIG, 1, 16><<<grid, block, 0, s>>>(g, il, nt, in, out);
      else if (zb == 4) k_z_op<BIG, 1, 4><<<grid, block, 0, s>>>(g, il, nt, in, out);
      else k_z_op<BIG, 1, 1><<<grid, block, 0, s>>>(g, il, nt, in, out);
      break;
    case 5:
      if (zb == 16) k_z_op<BIG, 2, 16><<<grid, block, 0, s>>>(g, il, nt, in, out);
      else if (zb == 4) k_z_op<BIG, 2, 4><<<grid, block, 0, s>>>(g, il, nt, in, out);
      else k_z_op<BIG, 2, 1><<<grid, block, 0, s>>>(g, il, nt, in, out);
      break;
    case 6: k_mixed_op<BIG, 0, 1><<<grid, block, 0, s>>>(g, il, nt, zb, in, out); break;
    case 7: k_mixed_op<BIG, 0, 2><<<grid, block, wb, s>>>(g, il, nt, zb, in, out); break;
    default: k_mixed_op<BIG, 1, 2><<<grid, block, wb, s>>>(g, il, nt, zb, in, out); break;
  }
}

}  // namespace

void launch_deriv(const Geo& g, int kind, const double* in, double* out, cudaStream_t s) {
  launch<false>(g, kind, in, out, s);
}

void launch_deriv_big(const Geo& g, int kind, const double* in, double* out, cudaStream_t s) {
  launch<true>(g, kind, in, out, s);
}

}  // namespace senga
