// Back-projection and forward projection of row-invariant geometries.
//
// A tilt is row-invariant when its detector column does not depend on the
// voxel row and its detector row is the voxel row plus a constant (a2 = 0,
// b1 = b3 = 0, b2 = 1: no XTILT, no in-plane rotation, any per-tilt shift),
// with steps |a1|, |a3| <= 1 and a1 >= 0.  Every row of the volume then
// interpolates at the same detector columns with the same weights, so the
// lanes of a warp run along the rows: the column walk is the same for the
// whole warp, its cost is shared by the lane's four rows, and no two lanes
// ever meet in a shared-memory bank.
//
// Stacks are kept transposed for this, [tilt][block of 128 rows][column][row]
// ("row stacks", with `margin` columns on each side of the detector's):
// blend_rows_kernel turns an image stack into voxel rows (the two detector
// rows of a voxel row blended with the tilt's constant y weights), so a
// window of columns x 128 rows is one contiguous piece, copied by a single
// bulk copy and used without staging by the threads; unblend_rows_kernel adds
// voxel-row sums back to detector rows.  (As boxes of a [tilt][column][row]
// tensor, the windows arrived at 8 bytes per clock and SM and the warps
// waited a third of the time for them.)
//
// The walk.  A warp owns a patch of 4 x 4 voxels in (x, z) and 128 rows, four
// per lane.  It visits the patch's 16 voxels on a snake path whose inner axis
// is the one with the smaller column step, so that successive voxels mostly
// share their two detector columns, which stay in registers: EV holds the
// even one of the two, OD the odd one.  Between the columns k and k + 1 at
// fraction f, OD's weight is f for even k and 1 - f for odd k, which is the
// magnitude of the coordinate modulo two columns taken as a signed Q1.31
// word.  A step crosses at most one column boundary (steps are at most one),
// where the register whose weight passes through zero is replaced.
//
// Coordinates, weights and crossings of a path are the same for all lanes, so
// the lanes compute them side by side -- lane i position i, two tilts at a
// time -- and leave them in shared memory as one 8-byte record per position,
// which a step reads as a broadcast.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "tr_device.cuh"
#include "tr_geom.h"
#include "tr_internal.cuh"

namespace trb {

namespace {

constexpr int kLaneRows = 4;
constexpr int kColBytes = kRowTile * (int)sizeof(float);  // one window column

// Shared bookkeeping of one tilt for one tile: coordinate of the tile's first
// voxel relative to kmin and the steps along x and z, Q32.32.
struct RowTilt {
  long long u0, sx, sz;
  int kmin;   // detector column of window column 0
  int flags;  // bit 0: x is the inner axis; bit 1: the window lies outside the stack
};

// FP64 setup of tilt g for the tile whose first voxel is (xc, zc) and whose
// extents minus one are (ex, ez).
__device__ __forceinline__ RowTilt row_tilt(const TiltGeo &g, int xc, int zc, float ox, float oz,
                                            double ex, double ez, int pnx,
                                            int cols) {
  const double X = (double)((float)xc - ox), Z = (double)((float)zc - oz);
  const double uc = g.a[0] + g.a[1] * X + g.a[3] * Z + (double)ox;
  const double umin = floor(uc + fmin(0.0, g.a[1] * ex) + fmin(0.0, g.a[3] * ez));
  RowTilt t;
  t.kmin = (int)umin - 1;
  t.u0 = __double2ll_rn((uc - (double)t.kmin) * 4294967296.0);
  t.sx = g.A[0];
  t.sz = g.A[2];
  const long long m3 = t.sz < 0 ? -t.sz : t.sz;
  t.flags = (m3 > t.sx ? 1 : 0) | (t.kmin < -cols || t.kmin > pnx ? 2 : 0);
  t.kmin = min(max(t.kmin, -cols), pnx);
  return t;
}

// Voxel of position i on the snake path over a 4 x 4 patch: i / 4 along the
// outer axis, forwards and backwards in turn along the inner one.
__host__ __device__ constexpr int snake_inner(int i) { return (i >> 2) & 1 ? 3 - (i & 3) : i & 3; }
// HALVES 1: the same over 4 (x) x 2 (z) voxels, the patch of the compensated
// back-projection.
template <bool XIN, int HALVES = 2>
__host__ __device__ constexpr int snake_voxel(int i) {  // z * 4 + x
  return XIN          ? (i >> 2) * 4 + snake_inner(i)
         : HALVES == 2 ? snake_inner(i) * 4 + (i >> 2)
                      : ((i & 1) ^ (i >> 1 & 1)) * 4 + (i >> 1);
}

// Float offset of column k (>= -margin) of row block yb in a row stack of nyb
// blocks per tilt.
__device__ __forceinline__ size_t row_stack_at(int t, int yb, int nyb, int k, int nx, int margin) {
  return (((size_t)t * nyb + yb) * (nx + 2 * margin) + (k + margin)) * kRowTile;
}
// Contiguous copies between global and shared memory (16-byte multiples): a
// load reported to mbarrier m, and an asynchronous float addition.
__device__ __forceinline__ void bulk_load(void *dst, const float *src, unsigned bytes,
                                          unsigned long long *m) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(m))
      : "memory");
}
__device__ __forceinline__ void bulk_add(float *dst, const void *src, unsigned bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(
                   __cvta_generic_to_global(dst)),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}

// One position of a patch's path: OD's weight and a window byte offset (see
// path_records).  Eight bytes: a broadcast read takes a wavefront per four bytes.
struct __align__(8) PathRec {
  float w;
  unsigned a;
};
// A path: its 16 positions, the crossing positions (bit per position) at which
// EV's and OD's column changes, and
//   gather: the positions within [-1, nx-1], RowTilt::flags;
//   splat: the window offsets of the last even and odd column.
struct __align__(16) PatchPath {
  PathRec pos[16];
  unsigned ev, od, c, d;
};

// Paths of the patches at (px, pz) of the tile, one per half warp: lane i % 16
// computes position i of its half's path.
//   gather: positions 0 and 8 hold the window offset of their lower column, a
//     crossing position that of the column to load.
//   splat: a crossing position holds the offset of the column to add to.
template <bool SPLAT, int HALVES = 2>
__device__ __forceinline__ void path_records(const RowTilt &tl, int px, int pz, int lane, int pnx,
                                             PatchPath *path) {
  const int pos = lane & 15, i = pos & (8 * HALVES - 1);  // HALVES 1: the upper 8 repeat
  const int v = tl.flags & 1 ? snake_voxel<true, HALVES>(i) : snake_voxel<false, HALVES>(i);
  const long long U = tl.u0 + (px + (v & 3)) * tl.sx + (pz + (v >> 2)) * tl.sz;
  const int k = (int)(U >> 32);
  const float w = fabsf((float)(int)(unsigned)(U >> 1)) * 4.656612873077393e-10f;  // 2^-31
  const int kp = __shfl_up_sync(0xffffffffu, k, 1);
  const bool cross = pos > 0 && k != kp;
  // the column that comes into reach (gather) or leaves it (splat)
  const int col = SPLAT ? (k > kp ? kp : kp + 1) : (k > kp ? k + 1 : k);
  const int half = lane & 16;
  const unsigned ev = __ballot_sync(0xffffffffu, cross && !(col & 1)) >> half;
  const unsigned od = __ballot_sync(0xffffffffu, cross && (col & 1)) >> half;
  const unsigned in_range =
      __ballot_sync(0xffffffffu, (unsigned)(k + tl.kmin + 1) <= (unsigned)pnx) >> half;
  const unsigned even = (k + (k & 1)) * kColBytes, odd = (k | 1) * kColBytes;
  const bool start = !SPLAT && (pos & 7) == 0;
  path->pos[pos] = PathRec{w, (unsigned)(start ? k : col) * kColBytes};
  if (pos == 15) {
    path->ev = ev;
    path->od = od;
    path->c = SPLAT ? even : in_range & 0xffffu;
    path->d = SPLAT ? odd : tl.flags;
  }
}

__device__ __forceinline__ void lds4(f32x2 &a, f32x2 &b, unsigned addr) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}

// One tilt of a patch: win is the lane's window address.  The path is walked in
// two halves side by side, whose loads overlap.  CHECK: positions outside
// `valid` get nothing.
template <bool XIN, bool CHECK, int HALVES>
__device__ __forceinline__ void gather_patch(f32x2 (&acc)[8 * HALVES][2], unsigned win,
                                             const PatchPath *path, unsigned mask_ev,
                                             unsigned mask_od, unsigned valid) {
  f32x2 ev[HALVES][2], od[HALVES][2];
  uint2 r[2][HALVES];  // the records of this step and the next
  auto fetch = [&](int j) {
#pragma unroll
    for (int h = 0; h < HALVES; ++h)
      r[j & 1][h] = *reinterpret_cast<const uint2 *>(path->pos + 8 * h + j);
  };
  fetch(0);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (j + 1 < 8) fetch(j + 1);
#pragma unroll
    for (int h = 0; h < HALVES; ++h) {
      const int i = 8 * h + j;
      const unsigned at = win + r[j & 1][h].y;
      if (j == 0) {
        // the even one of columns k and k + 1, and the odd one
        const unsigned k1 = (r[0][h].y / kColBytes & 1) * kColBytes;
        lds4(ev[h][0], ev[h][1], at + k1);
        lds4(od[h][0], od[h][1], at + kColBytes - k1);
      } else {
        asm volatile(
            "{\n .reg .pred p, q;\n .reg .b32 t, s;\n and.b32 t, %5, %7;\n setp.ne.u32 p, t, 0;\n"
            " and.b32 s, %6, %7;\n setp.ne.u32 q, s, 0;\n"
            " @p ld.shared.v2.u64 {%0, %1}, [%4];\n @q ld.shared.v2.u64 {%2, %3}, [%4];\n}"
            : "+l"(ev[h][0]), "+l"(ev[h][1]), "+l"(od[h][0]), "+l"(od[h][1])
            : "r"(at), "r"(mask_ev), "r"(mask_od), "r"(1u << i));
      }
    }
#pragma unroll
    for (int h = 0; h < HALVES; ++h) {
      const int i = 8 * h + j, v = snake_voxel<XIN, HALVES>(i);
      const float wf = __uint_as_float(r[j & 1][h].x);
      const f32x2 w = pack2(wf, wf);
      const f32x2 r0 = fma2(w, sub2(od[h][0], ev[h][0]), ev[h][0]);
      const f32x2 r1 = fma2(w, sub2(od[h][1], ev[h][1]), ev[h][1]);
      if (!CHECK || (valid >> i & 1)) {
        acc[v][0] = add2(acc[v][0], r0);
        acc[v][1] = add2(acc[v][1], r1);
      }
    }
  }
}

// Whether quads of the view's voxels at x0, x0 + 4, ... are aligned float4s.
__device__ __forceinline__ bool rows_vec(const VolView &v, int x0) {
  return x0 + 3 < v.nx && ((v.sy | v.sz) & 3) == 0 && (reinterpret_cast<uintptr_t>(v.vol) & 15) == 0;
}
// Four voxels from p, zero where !in or beyond the row's n.
__device__ __forceinline__ void load_quad(const float *p, bool in, bool vec, int n, float (&o)[4]) {
  if (vec) {
    const float4 q = in ? *reinterpret_cast<const float4 *>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
    o[0] = q.x, o[1] = q.y, o[2] = q.z, o[3] = q.w;
  } else {
#pragma unroll
    for (int x = 0; x < 4; ++x) o[x] = in && x < n ? p[x] : 0.f;
  }
}

// Patches of a tile along x and z, a warp each; tiles per SM at 16 warps.
constexpr int kBpPX = kRowBpX / 4, kBpPZ = kRowBpZ / 4, kBpWarps = kBpPX * kBpPZ;
constexpr int kBpPerSm = 16 / kBpWarps;
// Float4s of a tile's row, all sections: patches have 2 HALVES sections.
template <int HALVES>
constexpr int kBpQuads = 2 * HALVES * kBpPZ * kBpPX;
constexpr int kKahanTilts = 16;  // tilts summed plainly between compensated additions
constexpr int kLag = 4;  // a stage is refilled kLag tilts after its use

// Back-projection.  Volume tile of 16 (x) x 8 (z) voxels and 128 rows; warp w
// owns the patch at ((w % 4) 4, (w / 4) 4).  Tilts come through a ring of stages; the warps
// take turns at filling one, which is to start the window's copy and compute
// the eight patches' paths beside it.  (A ninth warp for this leaves 96
// registers a thread, which spills.)
//
// Bound by issue and by latency at 16 warps per SM (128 registers: 64 sums):
// 63 % of issue slots, 5.2 instructions per voxel and tilt where the general
// kernel takes 7 with one row per table entry, 75 % of the shared-memory
// wavefronts.
// 1024 x 1024 x 256 voxels, 61 tilts: 3.83 ms with the row stack's 0.15 ms,
// from 6.69 ms by the general kernel (4.3e12 from 2.4e12 voxel-tilts/s).
//
// KAHAN, for stacks that 16 bits held: 16 x 4 voxels, patches 4 x 2, since the
// sums of a 4 x 4 patch with totals and corrections take 192 registers.  The
// same volume: 6.17 ms from 6.90 ms by the general kernel.
template <int MODE, bool KAHAN>
__global__ void __launch_bounds__(kBpWarps * 32, kBpPerSm)
    bp_rows_kernel(const BpArgs a, const float *__restrict__ rows, int cols, int stages) {
  extern __shared__ __align__(128) unsigned char dsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int HALVES = KAHAN ? 1 : 2, VZ = 2 * HALVES, TZ = VZ * kBpPZ;
  constexpr int Q = kBpQuads<HALVES>;
  const int xc = blockIdx.x * kRowBpX, zl = blockIdx.y * TZ, yc = blockIdx.z * kRowTile;
  const int nt = a.nt;
  const unsigned win_bytes = (unsigned)cols * kColBytes;
  const unsigned stage_bytes = win_bytes + kBpWarps * (unsigned)sizeof(PatchPath);
  RowTilt *tt = reinterpret_cast<RowTilt *>(dsm + (size_t)stages * stage_bytes);
  unsigned long long *full = reinterpret_cast<unsigned long long *>(tt + ((nt + 1) & ~1));
  unsigned long long *empty = full + stages;

  if (tid == 0)
    for (int i = 0; i < stages; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, kBpWarps);
    }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  for (int i = tid; i < nt; i += blockDim.x)
    tt[i] = row_tilt(a.geo[a.t0 + i], xc, zl + a.v.zoff, a.ox, a.oz, kRowBpX - 1, TZ - 1, a.img.nx,
                     cols);
  __syncthreads();

  const float *src = rows + row_stack_at(a.t0, blockIdx.z, gridDim.z, 0, a.img.nx, cols);
  const size_t plane = (size_t)gridDim.z * (a.img.nx + 2 * cols) * kRowTile;
  auto fill = [&](int t, int s) {  // by one warp: tilt t into stage s
    unsigned char *st = dsm + (size_t)s * stage_bytes;
    const RowTilt &tl = tt[t];
    if (lane == 0)
      bulk_load(st, src + (long long)(t * plane) + (long long)tl.kmin * kRowTile, win_bytes,
                full + s);
    PatchPath *paths = reinterpret_cast<PatchPath *>(st + win_bytes);
#pragma unroll 1
    for (int b = 0; b < kBpWarps / 2; ++b) {
      const int w = 2 * b + (lane >> 4);
      path_records<false, HALVES>(tl, w % kBpPX * 4, w / kBpPX * VZ, lane, a.img.nx, paths + w);
    }
    __syncwarp();
    if (lane == 0) mbar_expect_tx(full + s, win_bytes);  // the stage's one arrival
  };
  for (int t = warp; t < min(stages - kLag, nt); t += kBpWarps) fill(t, t);

  // The tile's voxels are read at the end: into L2 meanwhile, one 64-byte
  // segment (a section's 16 x) per row and section.
  for (int i = tid; i < kRowTile * TZ; i += kBpWarps * 32) {
    const int y = yc + i / TZ, z = zl + i % TZ;
    if (y < a.v.ny && z < a.v.nz)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a.v.vol + (size_t)y * a.v.sy +
                                                     (size_t)z * a.v.sz + xc));
  }
  // KAHAN: kKahanTilts tilts sum into acc, which joins the voxel's total by one
  // compensated addition (comp: what the total's last addition lost).
  f32x2 acc[8 * HALVES][2], total[KAHAN ? 8 : 1][2], comp[KAHAN ? 8 : 1][2];
#pragma unroll
  for (int v = 0; v < 8 * HALVES; ++v) {
    acc[v][0] = acc[v][1] = 0ull;
    if (KAHAN) total[v][0] = total[v][1] = comp[v][0] = comp[v][1] = 0ull;
  }

  bool ok = true;
  int s = 0;            // stage of tilt t, and the parity of its use
  unsigned parity = 0;
  for (int t = 0; t < nt; ++t) {
    if ((t & (kBpWarps - 1)) == warp && t + stages - kLag < nt) {
      // the stage of tilt t - kLag, which the slowest warp has left or is about to
      const int s2 = s >= kLag ? s - kLag : s - kLag + stages;
      if (t >= kLag)
        ok = mbar_wait_bounded(empty + s2, s >= kLag ? parity : parity ^ 1u, 1ll << 31, a.err);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) fill(t + stages - kLag, s2);
    }
    ok = ok && mbar_wait_bounded(full + s, parity, 1ll << 31, a.err);
    if (!__all_sync(0xffffffffu, ok)) {
      ok = false;
      break;
    }
    const unsigned char *st = dsm + (size_t)s * stage_bytes;
    const PatchPath *path = reinterpret_cast<const PatchPath *>(st + win_bytes) + warp;
    const unsigned win = smem_u32(st) + lane * (kLaneRows * 4);
    const uint4 m = *reinterpret_cast<const uint4 *>(&path->ev);  // ev, od, in range, flags
    if (m.w & 2) {
      // nothing of the stack in reach
    } else if (MODE == BP_NORM && m.z != 0xffffu) {
      if (m.w & 1) gather_patch<true, true, HALVES>(acc, win, path, m.x, m.y, m.z);
      else gather_patch<false, true, HALVES>(acc, win, path, m.x, m.y, m.z);
    } else {
      if (m.w & 1) gather_patch<true, false, HALVES>(acc, win, path, m.x, m.y, m.z);
      else gather_patch<false, false, HALVES>(acc, win, path, m.x, m.y, m.z);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + s);
    if (KAHAN && (t % kKahanTilts == kKahanTilts - 1 || t + 1 == nt)) {
#pragma unroll
      for (int v = 0; v < 8 * HALVES; ++v)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const f32x2 y = sub2(acc[v][h], comp[v][h]), u = add2(total[v][h], y);
          comp[v][h] = sub2(sub2(u, total[v][h]), y);
          total[v][h] = u;
          acc[v][h] = 0ull;
        }
    }
    if (++s == stages) s = 0, parity ^= 1u;
  }
  if (__syncthreads_or(!ok)) {
    // Report, give the copies in flight a bounded chance to land, and leave the
    // tile's voxels untouched.
    if (!ok && lane == 0) {
      atomicExch(a.err, 1);
      atomicExch(a.err + 1, 1);
      for (int i = 0; i < stages; ++i)
        for (unsigned p = 0; p < 2; ++p) mbar_wait_bounded(full + i, p, 1ll << 24, nullptr);
    }
    return;
  }

  // Epilogue.  The sums go through shared memory, [row][section][16 x] with
  // the 16-byte pieces of a row exchanged so that neither side meets in a
  // bank, and the volume is read and written by sections' rows of 64 bytes.
  float4 *sum = reinterpret_cast<float4 *>(dsm);  // [128][Q]
  {
    const int px = warp % kBpPX, pz = warp / kBpPX * VZ;
#pragma unroll
    for (int r = 0; r < kLaneRows; ++r)
#pragma unroll
      for (int k = 0; k < VZ; ++k) {
        float f[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          float lo, hi;
          unpack2(KAHAN ? total[KAHAN ? k * 4 + x : 0][r >> 1] : acc[k * 4 + x][r >> 1], lo, hi);
          f[x] = r & 1 ? hi : lo;
        }
        sum[(lane * 4 + r) * Q + (((pz + k) * kBpPX + px) ^ (lane & 7))] =
            make_float4(f[0], f[1], f[2], f[3]);
      }
  }
  __syncthreads();
  const int quad = lane % Q;
  const int x0 = xc + quad % kBpPX * 4, z = zl + quad / kBpPX;
  const bool inz = z < a.v.nz && x0 < a.v.nx;
  const bool vec = rows_vec(a.v, x0);
  const int gx = (a.v.nx + kTX - 1) / kTX, gy = (a.v.ny + kTY - 1) / kTY;
  constexpr int kBatch = 8;  // rows whose reads are in flight together
  constexpr int kStep = 32 / Q;  // rows a warp takes at a time
  const int row0 = warp * (kRowTile / kBpWarps) + lane / Q;
#pragma unroll 1
  for (int i0 = 0; i0 < kRowTile / kBpWarps / kStep; i0 += kBatch) {
    float old[kBatch][4], scale[kBatch];
    int slot[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int y = yc + row0 + (i0 + i) * kStep;
      const bool in = inz && y < a.v.ny;
      load_quad(a.v.vol + (size_t)y * a.v.sy + (size_t)z * a.v.sz + x0, in, vec, a.v.nx - x0,
                old[i]);
      scale[i] = 1.f;
      slot[i] = -1;
      if (MODE == BP_SIRT && in) {
        slot[i] = __ldg(a.wslot + ((size_t)(z / kTZ) * gy + y / kTY) * gx + x0 / kTX);
        if (a.wrow) scale[i] = __ldg(a.wrow + y);  // interior tiles: one weight per row
      }
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int row = row0 + (i0 + i) * kStep, y = yc + row;
      if (!inz || y >= a.v.ny) continue;
      const float4 q = sum[row * Q + (quad ^ ((row >> 2) & 7))];
      const float s[4] = {q.x, q.y, q.z, q.w};
      const float sc = MODE == BP_SIRT ? (scale[i] != 0.f ? a.gamma / scale[i] : 0.f) : a.gamma;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        if (MODE == BP_SIRT && slot[i] >= 0) {
          // voxel of the border tile's compact weights (BpArgs::wslot)
          const float w = x0 + x < a.v.nx
                              ? a.wtvol[(size_t)slot[i] * kTileVox +
                                        ((z % kTZ) * kTY + y % kTY) * kTX + (x0 + x) % kTX]
                              : 0.f;
          if (w != 0.f) old[i][x] += s[x] * (a.gamma / w);
        } else {
          old[i][x] += s[x] * sc;
        }
      }
      float *p = a.v.vol + (size_t)y * a.v.sy + (size_t)z * a.v.sz + x0;
      if (vec) {
        *reinterpret_cast<float4 *>(p) = make_float4(old[i][0], old[i][1], old[i][2], old[i][3]);
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (x0 + x < a.v.nx) p[x] = old[i][x];
      }
    }
  }
}

// ------------------------------------------------------------ forward

// Adds the lane's four rows r to window column `addr`.
__device__ __forceinline__ void add_col(unsigned addr, f32x2 r0, f32x2 r1) {
  f32x2 a, b;
  lds4(a, b, addr);
  a = add2(a, r0);
  b = add2(b, r1);
  asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(addr), "l"(a), "l"(b));
}

// One tilt of a patch's splat; win: the lane's window address.  Two running sums
// take the place of EV and OD, a fused multiply-add each per voxel pair.  At a
// crossing one of them goes to its column and starts again at zero; the column's
// rows are read a position ahead (successive crossings never add to the same
// column), and the rest is a real branch (the masks are the same for the whole
// warp), since predicated instructions would be issued at every position.
template <bool XIN>
__device__ __forceinline__ void splat_patch(const f32x2 (&vox)[16][2], unsigned win,
                                            const PatchPath *path) {
  const uint4 m = *reinterpret_cast<const uint4 *>(&path->ev);  // ev, od, last columns
  const unsigned cross = m.x | m.y;
  f32x2 ev0 = 0ull, ev1 = 0ull, od0 = 0ull, od1 = 0ull;
  f32x2 c0 = 0ull, c1 = 0ull;  // rows of the column of the next crossing
  uint2 q[3];
  q[0] = *reinterpret_cast<const uint2 *>(path->pos);
  q[1] = *reinterpret_cast<const uint2 *>(path->pos + 1);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (i + 2 < 16) q[(i + 2) % 3] = *reinterpret_cast<const uint2 *>(path->pos + i + 2);
    if (i > 0)
      asm volatile(
          "{\n .reg .pred p, q;\n .reg .b32 t, s;\n .reg .b64 c, d;\n"
          " and.b32 t, %7, %9;\n setp.eq.u32 p, t, 0;\n @p bra.uni DONE;\n"
          " and.b32 s, %8, %9;\n setp.eq.u32 q, s, 0;\n @q bra.uni ODD;\n"
          " add.rn.f32x2 c, %4, %0;\n add.rn.f32x2 d, %5, %1;\n"
          " st.shared.v2.u64 [%6], {c, d};\n mov.b64 %0, 0;\n mov.b64 %1, 0;\n bra.uni DONE;\n"
          "ODD:\n add.rn.f32x2 c, %4, %2;\n add.rn.f32x2 d, %5, %3;\n"
          " st.shared.v2.u64 [%6], {c, d};\n mov.b64 %2, 0;\n mov.b64 %3, 0;\n"
          "DONE:\n}"
          : "+l"(ev0), "+l"(ev1), "+l"(od0), "+l"(od1)
          : "l"(c0), "l"(c1), "r"(win + q[i % 3].y), "r"(cross), "r"(m.x), "r"(1u << i));
    if (i + 1 < 16)
      asm volatile(
          "{\n .reg .pred p;\n .reg .b32 t;\n and.b32 t, %3, %4;\n setp.ne.u32 p, t, 0;\n"
          " @p ld.shared.v2.u64 {%0, %1}, [%2];\n}"
          : "+l"(c0), "+l"(c1)
          : "r"(win + q[(i + 1) % 3].y), "r"(cross), "r"(2u << i));
    const int v = snake_voxel<XIN>(i);
    const float wf = __uint_as_float(q[i % 3].x), we = 1.f - wf;
    const f32x2 w = pack2(wf, wf), e = pack2(we, we);
    ev0 = fma2(e, vox[v][0], ev0);
    ev1 = fma2(e, vox[v][1], ev1);
    od0 = fma2(w, vox[v][0], od0);
    od1 = fma2(w, vox[v][1], od1);
  }
  add_col(win + m.z, ev0, ev1);
  add_col(win + m.w, od0, od1);
}

// An empty window: as wide as a row-invariant tile's can be (rfp_cols with steps of
// at most one).
constexpr int kZeroCols = kRowFpX + kRowFpZ + 2;
__device__ __align__(128) float g_zero_window[kZeroCols * kRowTile];

constexpr int kFpPX = kRowFpX / 4, kFpPZ = kRowFpZ / 4, kFpWarps = kFpPX * kFpPZ;
constexpr int kFpPerSm = 16 / kFpWarps;
constexpr int kFpQuads = 4 * kFpPZ * kFpPX;

// Forward projection of a tile of 16 (x) x 4 (z) voxels and 128 rows into the
// row stack.  The voxels stay in registers.  The tilts' windows stand in a
// ring of slots and go from warp to warp: warp w adds its patch to a tilt's
// window once warp w - 1 has, so that no two add to it at a time and the
// additions need no atomics; the last warp sends the finished window out as one
// bulk reduction, and once that has read it, has a bulk copy clear the slot for the
// first (whose own stores of zeros took a seventh of the shared-memory wavefronts:
// 512 x 1024 x 128 voxels, 61 tilts 1613 -> 1568 us).  With all warps in step over
// eight windows at a time, barriers and the wait for the reductions took a quarter
// of the time.
//
// Bound by shared-memory wavefronts (78 % of their peak) and, at 16 warps per SM, by
// latency (60 % of issue slots); 7.5 instructions per voxel and tilt: a column that
// leaves the path is a read, an addition and a write of its window.  1024 x 1024 x
// 256 voxels, 61 tilts: 5.72 ms with the row sums' conversion and the weights, from
// 8.12 ms by the general splat alone, whose 32-bit fixed point this replaces by
// float sums.  Four warps in the chain and four CTAs per SM (before the last two
// changes 5.74 ms without the weights): eight and two took 6.07 ms, an 8 x 8 tile
// 5.90 ms, two warps 5.87 ms.
__global__ void __launch_bounds__(kFpWarps * 32, kFpPerSm)
    fp_rows_kernel(const FpArgs a, float *__restrict__ rows, int cols, int slots, int ahead) {
  extern __shared__ __align__(128) unsigned char dsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int xc = blockIdx.x * kRowFpX, zl = blockIdx.y * kRowFpZ, yc = blockIdx.z * kRowTile;
  const int nt = a.nt;
  const unsigned win_bytes = (unsigned)cols * kColBytes;
  // the windows' room also holds the tile's voxels at first
  RowTilt *tt = reinterpret_cast<RowTilt *>(dsm + max(slots * win_bytes, (unsigned)kRowTile * kFpQuads * 16));
  PatchPath *paths = reinterpret_cast<PatchPath *>(tt + ((nt + 1) & ~1)) + warp * 2;
  // per slot: warp w has added to it; the last: it holds zeros (again)
  unsigned long long *hand = reinterpret_cast<unsigned long long *>(
      reinterpret_cast<PatchPath *>(tt + ((nt + 1) & ~1)) + kFpWarps * 2);
  for (int i = tid; i < slots * kFpWarps; i += blockDim.x) mbar_init(hand + i, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  for (int i = tid; i < nt; i += blockDim.x)
    tt[i] = row_tilt(a.geo[a.t0 + i], xc, zl + a.v.zoff, a.ox, a.oz, kRowFpX - 1, kRowFpZ - 1, a.pnx, cols);

  // The tile's voxels, read by sections' rows of 64 bytes, through shared memory
  // (the windows') to the lanes that own their rows, as in the back-projection.
  f32x2 vox[16][2];
  bool any = a.v.vol == nullptr;
  if (a.v.vol) {
    float4 *buf = reinterpret_cast<float4 *>(dsm);  // [128][kFpQuads]
    const int quad = lane % kFpQuads;
    const int x0 = xc + quad % kFpPX * 4, z = zl + quad / kFpPX;
    const bool inz = z < a.v.nz, vec = rows_vec(a.v, x0);
    constexpr int kStep = 32 / kFpQuads;
#pragma unroll 8
    for (int i = 0; i < kRowTile / kFpWarps / kStep; ++i) {
      const int row = warp * (kRowTile / kFpWarps) + lane / kFpQuads + i * kStep, y = yc + row;
      float f[4];
      load_quad(a.v.vol + (size_t)y * a.v.sy + (size_t)z * a.v.sz + x0, inz && y < a.v.ny, vec,
                a.v.nx - x0, f);
      buf[row * kFpQuads + (quad ^ ((row >> 2) & 7))] = make_float4(f[0], f[1], f[2], f[3]);
      any |= f[0] != 0.f || f[1] != 0.f || f[2] != 0.f || f[3] != 0.f;
    }
  }
  if (!__syncthreads_or(any)) return;  // an all-zero tile adds nothing
  {
    const int px = warp % kFpPX, pz = warp / kFpPX * 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float4 f[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (a.v.vol) {
          f[r] = reinterpret_cast<const float4 *>(
              dsm)[(lane * 4 + r) * kFpQuads + (((pz + k) * kFpPX + px) ^ (lane & 7))];
        } else {
          const int x0 = xc + px * 4;
          const bool in = yc + lane * 4 + r < a.v.ny && zl + pz + k < a.v.nz;
          f[r] = make_float4(in && x0 < a.v.nx ? 1.f : 0.f, in && x0 + 1 < a.v.nx ? 1.f : 0.f,
                             in && x0 + 2 < a.v.nx ? 1.f : 0.f, in && x0 + 3 < a.v.nx ? 1.f : 0.f);
        }
      }
      vox[k * 4 + 0][0] = pack2(f[0].x, f[1].x), vox[k * 4 + 0][1] = pack2(f[2].x, f[3].x);
      vox[k * 4 + 1][0] = pack2(f[0].y, f[1].y), vox[k * 4 + 1][1] = pack2(f[2].y, f[3].y);
      vox[k * 4 + 2][0] = pack2(f[0].z, f[1].z), vox[k * 4 + 2][1] = pack2(f[2].z, f[3].z);
      vox[k * 4 + 3][0] = pack2(f[0].w, f[1].w), vox[k * 4 + 3][1] = pack2(f[2].w, f[3].w);
    }
  }
  __syncthreads();

  if (a.v.vol) {
    // Into L2: the voxels of the tile that takes this one's place on the SM.
    unsigned n = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x + ahead;
    const unsigned bx = n % gridDim.x, by = n / gridDim.x % gridDim.y, bz = n / gridDim.x / gridDim.y;
    for (int i = tid; i < kRowTile * kRowFpZ; i += blockDim.x) {
      const int y = bz * kRowTile + i / kRowFpZ, z = by * kRowFpZ + i % kRowFpZ;
      if (y < a.v.ny && z < a.v.nz)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.v.vol + (size_t)y * a.v.sy +
                                                       (size_t)z * a.v.sz + bx * kRowFpX));
    }
  }

  float *dst = rows + row_stack_at(a.t0, blockIdx.z, gridDim.z, 0, a.pnx, cols);
  const size_t plane = (size_t)gridDim.z * (a.pnx + 2 * cols) * kRowTile;
  auto clear = [&](int slot) {  // zeros into a slot, for the first warp's next turn
    unsigned long long *m = hand + (slot + 1) * kFpWarps - 1;
    bulk_load(dsm + (size_t)slot * win_bytes, g_zero_window, win_bytes, m);
    mbar_expect_tx(m, win_bytes);
  };
  if (tid == (kFpWarps - 1) * 32) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int i = 0; i < min(slots, nt); ++i) clear(i);
  }
  bool ok = true;
  int s = 0;             // slot of tilt t, and the parity of its use
  unsigned parity = 0;
  for (int t = 0; t < nt; ++t) {
    if (!(t & 1)) {  // this warp's paths of two tilts
      __syncwarp();
      path_records<true>(tt[min(t + (lane >> 4), nt - 1)], warp % kFpPX * 4, warp / kFpPX * 4, lane,
                         a.pnx, paths + (lane >> 4));
      __syncwarp();
    }
    unsigned char *win = dsm + (size_t)s * win_bytes;
    unsigned long long *h = hand + s * kFpWarps;
    ok = mbar_wait_bounded(warp > 0 ? h + warp - 1 : h + kFpWarps - 1, parity, 1ll << 31, a.err);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) break;
    const RowTilt &tl = tt[t];
    const unsigned at = smem_u32(win) + lane * (kLaneRows * 4);
    if (tl.flags & 1) splat_patch<true>(vox, at, paths + (t & 1));
    else splat_patch<false>(vox, at, paths + (t & 1));
    __syncwarp();
    if (lane == 0) {
      if (warp < kFpWarps - 1) {
        mbar_arrive(h + warp);
      } else {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!(tl.flags & 2))
          bulk_add(dst + (long long)(t * plane) + (long long)tl.kmin * kRowTile, win, win_bytes);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        // the reduction before this one has read its slot
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        if (t > 0 && t - 1 + slots < nt) clear(s > 0 ? s - 1 : slots - 1);
      }
    }
    if (++s == slots) s = 0, parity ^= 1u;
  }
  if (!ok && lane == 0 && a.err) {  // report; the sums of this tile are incomplete
    atomicExch(a.err, 1);
    atomicExch(a.err + 1, 1);
  }
  if (!ok && tid == (kFpWarps - 1) * 32)  // a chance for the zeros in flight to land
    for (int i = 1; i <= slots; ++i)
      for (unsigned p = 0; p < 2; ++p)
        mbar_wait_bounded(hand + i * kFpWarps - 1, p, 1ll << 24, nullptr);
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ------------------------------------------------------------ row stacks

template <typename IT>
__device__ __forceinline__ float img_f(const IT *p, size_t i);
template <>
__device__ __forceinline__ float img_f<float>(const float *p, size_t i) { return __ldg(p + i); }
template <>
__device__ __forceinline__ float img_f<__half>(const __half *p, size_t i) {
  return __half2float(p[i]);
}
template <>
__device__ __forceinline__ float img_f<__nv_bfloat16>(const __nv_bfloat16 *p, size_t i) {
  return __bfloat162float(p[i]);
}

// Lower detector row of voxel row y and the upper one's weight, as the
// reference evaluates them (b1 = b3 = 0, b2 = 1).
__device__ __forceinline__ int voxel_row(const TiltGeo &g, int y, float oy, float &dy) {
  const double v = g.b[0] + g.b[2] * (double)((float)y - oy) + (double)oy;
  const int y0 = (int)floor(v);
  dy = (float)(v - (double)y0);
  return y0;
}

constexpr int kBlendCols = 32, kBlendRows = 64;

// Image stack -> row stack: the blended value of voxel row y at detector column
// k.  NORM: columns -1..nx of the edge-clamped image, rows normalised by their
// in-image weight (zero where neither row is inside); else columns 0..nx-1,
// in-image rows only.  Zero in the other margin columns and below the volume.
template <bool NORM, typename IT>
__global__ void __launch_bounds__(256)
    blend_rows_kernel(const ImgView im, const TiltGeo *__restrict__ geo, int t0, float oy, int vny,
                      int margin, float *__restrict__ out) {
  __shared__ float s[kBlendCols][kBlendRows + 1];
  const int t = blockIdx.z, c0 = blockIdx.x * kBlendCols, r0 = blockIdx.y * kBlendRows;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, tc = im.nx + 2 * margin;
  const TiltGeo &g = geo[t0 + t];
  const IT *p = reinterpret_cast<const IT *>(im.p) + (size_t)(t0 + t) * im.tstride;
  const float sc = im.scale ? im.scale[t0 + t] : 1.f;
  int k = c0 + lane - margin;
  const bool ink = NORM ? k >= -1 && k <= im.nx : k >= 0 && k < im.nx;
  k = min(max(k, 0), im.nx - 1);
#pragma unroll
  for (int i = 0; i < kBlendRows / 8; ++i) {
    const int r = wp + 8 * i, y = r0 + r;
    float v = 0.f;
    if (ink && y < vny) {
      float dy;
      const int y0 = voxel_row(g, y, oy, dy);
      const float w0 = (y0 >= 0 && y0 < im.ny) ? 1 - dy : 0.f;
      const float w1 = (y0 + 1 >= 0 && y0 + 1 < im.ny) ? dy : 0.f;
      const float p0 = w0 != 0.f ? img_f(p, (size_t)y0 * im.nx + k) * sc : 0.f;
      const float p1 = w1 != 0.f ? img_f(p, (size_t)(y0 + 1) * im.nx + k) * sc : 0.f;
      v = w0 * p0 + w1 * p1;
      if (NORM) v = w0 + w1 != 0.f ? v / (w0 + w1) : 0.f;
    }
    s[lane][r] = v;
  }
  __syncthreads();
  float *o = out + ((size_t)(t0 + t) * ((vny + kRowTile - 1) / kRowTile) + r0 / kRowTile) * tc * kRowTile +
             r0 % kRowTile + lane;
#pragma unroll
  for (int i = 0; i < kBlendCols / 8; ++i) {
    const int c = wp + 8 * i;
    if (c0 + c >= tc) break;
#pragma unroll
    for (int h = 0; h < kBlendRows / 32; ++h)
      o[(size_t)(c0 + c) * kRowTile + 32 * h] = s[c][lane + 32 * h];
  }
}

// Row stack -> image stack: val[t][j][k] += the voxel-row sums that splat onto
// detector row j, (1 - dy) of the row whose lower detector row is j and dy of
// the one below.
__global__ void __launch_bounds__(256)
    unblend_rows_kernel(const float *__restrict__ rows, const TiltGeo *__restrict__ geo, int t0,
                        float oy, int vny, int margin, float *__restrict__ val, long long tstride,
                        int nx, int ny) {
  constexpr int kHalo = 3;  // voxel rows j - S - 2 .. j - S + 1, S = floor(b0)
  __shared__ float s[kBlendCols][kBlendRows + kHalo + 2];
  __shared__ int sy0[kBlendRows + kHalo];
  __shared__ float sdy[kBlendRows + kHalo];
  const int t = blockIdx.z, c0 = blockIdx.x * kBlendCols, j0 = blockIdx.y * kBlendRows;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const TiltGeo &g = geo[t0 + t];
  const int tc = nx + 2 * margin, nyb = (vny + kRowTile - 1) / kRowTile;
  const int S = (int)floor(g.b[0]);
  const int y0 = j0 - S - 2;  // first voxel row of the tile
  bool even = true;
  if (threadIdx.x < kBlendRows + kHalo) {
    float dy;
    const int d = voxel_row(g, y0 + threadIdx.x, oy, dy);
    sy0[threadIdx.x] = d;
    sdy[threadIdx.x] = dy;
    even = d == y0 + (int)threadIdx.x + S;
  }
  for (int c = wp; c < kBlendCols; c += 8)
    for (int r = lane; r < kBlendRows + kHalo; r += 32) {
      const int y = y0 + r, k = c0 + c;
      s[c][r] = k < nx && y >= 0 && y < vny
                    ? __ldg(rows + (((size_t)(t0 + t) * nyb + y / kRowTile) * tc + k + margin) *
                                       kRowTile + y % kRowTile)
                    : 0.f;
    }
  even = __syncthreads_and(even);  // every row's lower detector row is S below
  const int k = c0 + lane;
  if (k >= nx) return;
#pragma unroll
  for (int i = 0; i < kBlendRows / 8; ++i) {
    const int r = wp + 8 * i, j = j0 + r;
    if (j >= ny) break;
    float v = 0.f;
    if (even) {
      v = (1 - sdy[r + 2]) * s[lane][r + 2] + sdy[r + 1] * s[lane][r + 1];
    } else {
#pragma unroll
      for (int h = 0; h <= kHalo; ++h) {
        const int q = r + h;
        if (sy0[q] == j) v += (1 - sdy[q]) * s[lane][q];
        else if (sy0[q] == j - 1) v += sdy[q] * s[lane][q];
      }
    }
    if (v != 0.f) {
      float *o = val + (size_t)(t0 + t) * tstride + (size_t)j * nx + k;
      *o += v;
    }
  }
}

// SIRT's step between the projections in one pass: the forward projection's row
// sums -> detector rows -> residual p ps - val/wt (val where wt = 0) -> the
// blended voxel-row stack the back-projection reads (resid_kernel between
// unblend_rows_kernel and blend_rows_kernel: 125 us together on 41 tilts of 512 x
// 512, 70 us in this pass).  A block makes 64 voxel rows of 32 columns.  With S =
// floor(b0), voxel row y's lower detector row is y + S, or next to it where b0 is
// within rounding of an integer: rows r0 + S - 1 .. r0 + S + 65 are needed, and
// voxel rows r0 - 3 .. r0 + 66 for them.
// NORMAL: ADMM's val/wt in the residual's place, nothing where wt is 1e-5 or less
// (admm_normalize's rule); p is not read.  Two ADMM iterations of 61 tilts of 256 x
// 256, 64 sections: 1.91 -> 1.71 ms.
template <typename PT, bool NORMAL>
__global__ void __launch_bounds__(256)
    resid_rows_kernel(const float *__restrict__ sums, int smargin, const PT *__restrict__ p,
                      const float *__restrict__ ps, const float *__restrict__ wt,
                      const TiltGeo *__restrict__ geo, float oy, int nx, int ny,
                      float *__restrict__ rows, int margin) {
  constexpr int kDet = kBlendRows + 3, kVox = kBlendRows + 6;
  __shared__ float f[kBlendCols][kVox + 1];
  __shared__ float r[kBlendCols][kDet + 2];
  __shared__ int sy0[kVox];
  __shared__ float sdy[kVox];
  const int t = blockIdx.z, c0 = blockIdx.x * kBlendCols, r0 = blockIdx.y * kBlendRows;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int nyb = (ny + kRowTile - 1) / kRowTile, tc = nx + 2 * margin;
  const TiltGeo &g = geo[t];
  const int S = (int)floor(g.b[0]), yb = r0 - 3, jb = r0 + S - 1, k0 = c0 - margin;
  // every global read of the block in flight before the first is used
  const int k = k0 + lane;
  const bool ink = k >= 0 && k < nx;
  constexpr int kPer = (kDet + 7) / 8;
  float pv[kPer], wv[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int j = jb + wp + 8 * i;
    const bool in = ink && wp + 8 * i < kDet && j >= 0 && j < ny;
    const size_t at = in ? ((size_t)t * ny + j) * nx + k : 0;
    pv[i] = !NORMAL && in ? img_f(p, at) : 0.f;
    wv[i] = in ? __ldg(wt + at) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < kBlendCols / 8; ++i) {
    const int c = wp + 8 * i, kc = k0 + c;
#pragma unroll
    for (int h = 0; h < (kVox + 31) / 32; ++h) {
      const int q = lane + 32 * h, y = yb + q;
      const bool in = q < kVox && kc >= 0 && kc < nx && y >= 0 && y < ny;
      const float v =
          in ? __ldg(sums + row_stack_at(t, y / kRowTile, nyb, kc, nx, smargin) + y % kRowTile) : 0.f;
      if (q < kVox) f[c][q] = v;
    }
  }
  bool even = true;
  if (threadIdx.x < kVox) {
    float dy;
    const int y0 = voxel_row(g, yb + threadIdx.x, oy, dy);
    sy0[threadIdx.x] = y0;
    sdy[threadIdx.x] = dy;
    even = y0 == yb + (int)threadIdx.x + S;
  }
  even = __syncthreads_and(even);  // every row's lower detector row is S below
  const float scale = ps ? ps[t] : 1.f;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int q = wp + 8 * i, j = jb + q;
    if (q < kDet) {
      float v = 0.f;
      if (even) {
        v = (1 - sdy[q + 2]) * f[lane][q + 2] + sdy[q + 1] * f[lane][q + 1];
      } else {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          if (sy0[q + h] == j) v += (1 - sdy[q + h]) * f[lane][q + h];
          else if (sy0[q + h] == j - 1) v += sdy[q + h] * f[lane][q + h];
        }
      }
      if (NORMAL) v = (double)fabsf(wv[i]) > 10e-6 ? v / wv[i] : 0.f;
      else v = pv[i] * scale - (wv[i] != 0.f ? v / wv[i] : v);
      r[lane][q] = ink && j >= 0 && j < ny ? v : 0.f;
    }
  }
  __syncthreads();
  float *o = rows + row_stack_at(t, r0 / kRowTile, nyb, k0, nx, margin) + r0 % kRowTile + lane;
#pragma unroll
  for (int i = 0; i < kBlendCols / 8; ++i) {
    const int c = wp + 8 * i;
    if (c0 + c >= tc) break;
#pragma unroll
    for (int h = 0; h < kBlendRows / 32; ++h) {
      const int y = r0 + lane + 32 * h, q = y - yb, j = sy0[q];
      float v = 0.f;  // detector rows outside the image hold zeros
      if (y < ny) v = (1 - sdy[q]) * r[c][j - jb] + (sdy[q] != 0.f ? sdy[q] * r[c][j - jb + 1] : 0.f);
      o[(size_t)c * kRowTile + 32 * h] = v;
    }
  }
}

// Projection weights (the splat of ones) of separable geometries whose columns
// do not depend on the row (a2 = 0): the weight of detector pixel (j, k) is a
// column's times a row's,
//   sum over x, z of the tent 1 - |u(x, z) - k|  times  sum over y of 1 - |v(y) - j|,
// so a block sums its tilt's 32 columns in FP64 (the few x per section that
// reach them, |a1| being 0.05 or more) and writes all their pixels.  61 tilts of
// 2048 x 2048, 128 sections: 12.2 ms as a forward projection of ones -> 0.26 ms.
template <bool ADD>
__global__ void __launch_bounds__(256)
    weight_rows_kernel(const TiltGeo *__restrict__ geo, int nx, int ny, int z0, int nz, float ox,
                       float oy, float oz, float *__restrict__ wt, long long tstride) {
  __shared__ double part[8][32];
  const int t = blockIdx.y, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  const TiltGeo &g = geo[t];
  const double a1 = g.a[1], inv = 1.0 / a1, reach = fabs(inv);
  double sum = 0.0;
  for (int z = wp; z < nz; z += 8) {
    const double c = g.a[0] + g.a[3] * (double)((float)(z0 + z) - oz) + (double)ox - (double)k;
    const double xm = (double)ox - c * inv;  // where u = k
    const int x0 = max(0, (int)floor(xm - reach)), x1 = min(nx - 1, (int)ceil(xm + reach));
    for (int x = x0; x <= x1; ++x)
      sum += fmax(0.0, 1.0 - fabs(c + a1 * (double)((float)x - ox)));
  }
  part[wp][lane] = sum;
  __syncthreads();
  double all = 0.0;
#pragma unroll
  for (int w = 0; w < 8; ++w) all += part[w][lane];
  const float cw = (float)all;
  const int S = (int)floor(g.b[0]);
  float *p = wt + (size_t)t * tstride + k;
  for (int j0 = wp * 32; j0 < ny; j0 += 256) {
    // lane: the row weight of detector row j0 + lane, from the voxel rows that
    // can reach it
    const int j = j0 + lane;
    float rw = 0.f;
#pragma unroll
    for (int h = -2; h <= 1; ++h) {
      const int y = j - S + h;
      if (y < 0 || y >= ny) continue;
      float dy;
      const int y0 = voxel_row(g, y, oy, dy);
      if (y0 == j) rw += 1 - dy;
      else if (y0 == j - 1) rw += dy;
    }
    for (int i = 0; i < min(32, ny - j0); ++i) {
      const float r = __shfl_sync(0xffffffffu, rw, i);
      if (k < nx) {
        float *q = p + (size_t)(j0 + i) * nx;
        *q = ADD ? *q + cw * r : cw * r;
      }
    }
  }
}

}  // namespace

// ------------------------------------------------------------ launchers

cudaError_t launch_blend_rows(const ImgView &im, const TiltGeo *geo, int t0, int nt, float oy,
                              int vny, int margin, bool norm, float *rows, cudaStream_t s) {
  const int tc = im.nx + 2 * margin;
  const dim3 grid((tc + kBlendCols - 1) / kBlendCols,
                  (vny + kRowTile - 1) / kRowTile * (kRowTile / kBlendRows), nt);
  auto go = [&](auto *tag) {
    using IT = std::remove_pointer_t<decltype(tag)>;
    if (norm)
      blend_rows_kernel<true, IT><<<grid, 256, 0, s>>>(im, geo, t0, oy, vny, margin, rows);
    else
      blend_rows_kernel<false, IT><<<grid, 256, 0, s>>>(im, geo, t0, oy, vny, margin, rows);
  };
  if (im.dtype == IMG_F16) go((__half *)nullptr);
  else if (im.dtype == IMG_BF16) go((__nv_bfloat16 *)nullptr);
  else go((float *)nullptr);
  return cudaGetLastError();
}

cudaError_t launch_unblend_rows(const float *rows, const TiltGeo *geo, int t0, int nt, float oy,
                                int vny, int margin, float *val, long long tstride, int nx, int ny,
                                cudaStream_t s) {
  const dim3 grid((nx + kBlendCols - 1) / kBlendCols, (ny + kBlendRows - 1) / kBlendRows, nt);
  unblend_rows_kernel<<<grid, 256, 0, s>>>(rows, geo, t0, oy, vny, margin, val, tstride, nx, ny);
  return cudaGetLastError();
}

cudaError_t launch_resid_rows(const float *sums, int smargin, const void *p, int pdtype,
                              const float *ps, const float *wt, const TiltGeo *geo, int nt, float oy,
                              int nx, int ny, float *rows, int margin, cudaStream_t s) {
  const dim3 grid((nx + 2 * margin + kBlendCols - 1) / kBlendCols,
                  (ny + kRowTile - 1) / kRowTile * (kRowTile / kBlendRows), nt);
  auto go = [&](auto *img, auto normal) {
    using PT = std::remove_const_t<std::remove_pointer_t<decltype(img)>>;
    resid_rows_kernel<PT, decltype(normal)::value><<<grid, 256, 0, s>>>(
        sums, smargin, img, ps, wt, geo, oy, nx, ny, rows, margin);
  };
  if (!p) go((const float *)nullptr, std::true_type());
  else if (pdtype == IMG_F16) go((const __half *)p, std::false_type());
  else if (pdtype == IMG_BF16) go((const __nv_bfloat16 *)p, std::false_type());
  else go((const float *)p, std::false_type());
  return cudaGetLastError();
}

cudaError_t launch_weight_rows(const TiltGeo *geo, int nt, int nx, int ny, int z0, int nz, float ox,
                               float oy, float oz, float *wt, long long tstride, bool add,
                               cudaStream_t s) {
  for (int t = 0; t < nt; t += 65535) {
    const dim3 grid((nx + 31) / 32, std::min(65535, nt - t));
    float *w = wt + (size_t)t * tstride;
    if (add)
      weight_rows_kernel<true><<<grid, 256, 0, s>>>(geo + t, nx, ny, z0, nz, ox, oy, oz, w, tstride);
    else
      weight_rows_kernel<false><<<grid, 256, 0, s>>>(geo + t, nx, ny, z0, nz, ox, oy, oz, w, tstride);
  }
  return cudaGetLastError();
}

// Dynamic shared memory of the kernels.
static size_t bp_rows_smem(int cols, int nt, int stages) {
  return (size_t)stages * (cols * kColBytes + kBpWarps * sizeof(PatchPath) + 16) +
         (size_t)((nt + 1) & ~1) * sizeof(RowTilt);  // at least the epilogue's sums
}
static int bp_rows_stages(int cols, int nt) {
  const size_t fixed = bp_rows_smem(cols, nt, 0), per = bp_rows_smem(cols, 0, 1);
  // 16 warps per SM when that leaves windows in flight
  for (size_t room : {kRowSmem / kBpPerSm, kRowSmem})
    if (fixed < room && (room - fixed) / per >= kLag + 2)
      return (int)std::min<size_t>(10, (room - fixed) / per);
  return 0;
}
bool bp_rows_fits(int cols, int nt) { return bp_rows_stages(cols, nt) >= kLag + 2; }

static size_t fp_rows_smem(int cols, int nt, int slots) {
  return std::max<size_t>((size_t)slots * cols * kColBytes, kRowTile * kFpQuads * 16) +
         (size_t)((nt + 1) & ~1) * sizeof(RowTilt) + kFpWarps * 2 * sizeof(PatchPath) +
         slots * kFpWarps * sizeof(unsigned long long);
}
// Slots: one in each warp's hands, one being sent out, and some to spare.
static int fp_rows_slots(int cols, int nt, size_t room) {
  for (int n = kFpWarps + 4; n > kFpWarps; --n)
    if (fp_rows_smem(cols, nt, n) <= room) return n;
  return 0;
}
// CTAs per SM, and the most tilts of a launch whose bookkeeping leaves the SM room
// for them: kFpPerSm for the windows of rotations (20 columns at most), half of it
// for sheared ones.  (512 x 512 x 64 voxels, windows of 20 columns: 150 tilts 1.10
// ms; 160 tilts in one launch of two CTAs per SM 1.46 ms, as two launches 1.21 ms.)
struct FpResident {
  int per_sm, tilts;
  size_t room;
};
static FpResident fp_rows_resident(int cols) {
  const size_t fixed = fp_rows_smem(cols, 0, kFpWarps + 1);
  for (int n : {kFpPerSm, kFpPerSm / 2}) {
    const size_t room = kRowSmem / n;
    if (fixed + 64 * sizeof(RowTilt) <= room)
      return {n, (int)((room - fixed) / sizeof(RowTilt)) & ~1, room};
  }
  return {0, 0, 0};
}
bool fp_rows_fits(int cols) { return cols <= kZeroCols && fp_rows_resident(cols).tilts > 0; }

template <int MODE, bool KAHAN>
static cudaError_t launch_bp_rows_t(const BpArgs &a, const float *rows, int cols, cudaStream_t s) {
  const int stages = bp_rows_stages(cols, a.nt);
  const size_t smem = std::max<size_t>(bp_rows_smem(cols, a.nt, stages),
                                       kRowTile * kBpQuads<KAHAN ? 1 : 2> * 16);
  cudaError_t e = cudaFuncSetAttribute(bp_rows_kernel<MODE, KAHAN>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int tz = KAHAN ? kRowBpZ / 2 : kRowBpZ;
  const dim3 grid((a.v.nx + kRowBpX - 1) / kRowBpX, (a.v.nz + tz - 1) / tz,
                  (a.v.ny + kRowTile - 1) / kRowTile);
  bp_rows_kernel<MODE, KAHAN><<<grid, kBpWarps * 32, smem, s>>>(a, rows, cols, stages);
  return cudaGetLastError();
}

template <bool KAHAN>
static cudaError_t launch_bp_rows_k(int mode, const BpArgs &a, const float *rows, int cols,
                                    cudaStream_t s) {
  if (mode == BP_NORM) return launch_bp_rows_t<BP_NORM, KAHAN>(a, rows, cols, s);
  if (mode == BP_SIRT) return launch_bp_rows_t<BP_SIRT, KAHAN>(a, rows, cols, s);
  return launch_bp_rows_t<BP_SUM, KAHAN>(a, rows, cols, s);
}

cudaError_t launch_bp_rows(int mode, const BpArgs &a, const float *rows, int cols, bool kahan,
                           cudaStream_t s) {
  return kahan ? launch_bp_rows_k<true>(mode, a, rows, cols, s)
               : launch_bp_rows_k<false>(mode, a, rows, cols, s);
}

cudaError_t launch_fp_rows(const FpArgs &a, float *rows, int cols, int nsm, cudaStream_t s) {
  const FpResident fit = fp_rows_resident(cols);
  const int groups = (a.nt + fit.tilts - 1) / fit.tilts, per = (a.nt + groups - 1) / groups;
  const int slots = fp_rows_slots(cols, per, fit.room);
  const size_t smem = fp_rows_smem(cols, per, slots);
  cudaError_t e = cudaFuncSetAttribute(fp_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((a.v.nx + kRowFpX - 1) / kRowFpX, (a.v.nz + kRowFpZ - 1) / kRowFpZ,
                  (a.v.ny + kRowTile - 1) / kRowTile);
  for (int t = 0; t < a.nt; t += per) {
    FpArgs g = a;
    g.t0 = a.t0 + t;
    g.nt = std::min(per, a.nt - t);
    fp_rows_kernel<<<grid, kFpWarps * 32, smem, s>>>(g, rows, cols, slots, fit.per_sm * nsm);
  }
  return cudaGetLastError();
}

}  // namespace trb
