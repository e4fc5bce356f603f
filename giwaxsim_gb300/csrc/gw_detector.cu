// Detector stage: sample I(q) with a rotated detector plane over many
// orientations and sum the weighted samples (tools/comparison.py:790-870,
// tools/detector.py:5-29, :194-300).
//
// One thread owns one pixel for the whole orientation loop, so the sum over
// orientations stays in registers (float64, or Kahan-compensated float32)
// and the image is written once; no atomics.  Per pixel and orientation the
// thread replays the reference's exact float64 arithmetic: the plane
// rotations in BLAS fused order (rot_chain), the shift by np.min(q), the
// floor division by np.diff(qz)[0] and np.clip, then gathers the float32
// I(q) value.  Rotation matrices and weights are computed on the host from
// the plane's corners exactly as the reference does and passed in; identity
// rotations (angle 0) are dropped by the host, which leaves every bit
// unchanged.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "gw_common.cuh"

namespace {

struct DetArgs {
  int nh, nv;
  int ny, nx, nz;
  double qmin_x, qmin_y, qmin_z, dq, inv_dq;
  const double *h, *v;
  const double *init_R;
  int n_init;
  const int *rot_start, *rot_n;
  const double *rot_R;
  const double *w;
  int n_orient;
  const float *iq;
  int64_t sy, sx, sz;  // element strides of iq (the fixed axis' is 0 when iq
                       // is the compact plane of plane mode)
  int kahan;
};

__device__ __forceinline__ void rotate(const double *R, double &x, double &y,
                                       double &z) {
  const double a = rot_chain(R, x, y, z);
  const double b = rot_chain(R + 3, x, y, z);
  const double c = rot_chain(R + 6, x, y, z);
  x = a; y = b; z = c;
}

__device__ __forceinline__ int clip_idx(double p, double qmin, double dq,
                                        double inv_dq, int n) {
  double k = floor_div_exact(GW_DSUB(p, qmin), dq, inv_dq);
  k = fmin(fmax(k, 0.0), (double)(n - 1));
  return (int)k;
}

__device__ __forceinline__ void base_point(const DetArgs &a, int i, int j,
                                           double &x, double &y, double &z) {
  x = 0.0; y = a.h[j]; z = a.v[i];
  for (int k = 0; k < a.n_init; ++k) rotate(a.init_R + 9 * k, x, y, z);
}

__device__ __forceinline__ int64_t gather_index(const DetArgs &a, int o,
                                                double x, double y, double z) {
  const int s = a.rot_start[o], n = a.rot_n[o];
  for (int k = 0; k < n; ++k) rotate(a.rot_R + 9 * (s + k), x, y, z);
  const int ix = clip_idx(x, a.qmin_x, a.dq, a.inv_dq, a.nx);
  const int iy = clip_idx(y, a.qmin_y, a.dq, a.inv_dq, a.ny);
  const int iz = clip_idx(z, a.qmin_z, a.dq, a.inv_dq, a.nz);
  return iy * a.sy + ix * a.sx + iz * a.sz;
}

__global__ void k_detector(DetArgs a, double *acc_out) {
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= a.nh * a.nv) return;
  const int i = pix / a.nh, j = pix % a.nh;
  double x0, y0, z0;
  base_point(a, i, j, x0, y0, z0);
  if (!a.kahan) {
    double acc = 0.0;
    for (int o = 0; o < a.n_orient; ++o) {
      const int64_t idx = gather_index(a, o, x0, y0, z0);
      acc = fma((double)__ldg(a.iq + idx), a.w[o], acc);
    }
    acc_out[pix] = acc;
  } else {
    float s = 0.f, c = 0.f;
    for (int o = 0; o < a.n_orient; ++o) {
      const int64_t idx = gather_index(a, o, x0, y0, z0);
      const float yv = __ldg(a.iq + idx) * (float)a.w[o] - c;
      const float t = s + yv;
      c = (t - s) - yv;
      s = t;
    }
    acc_out[pix] = (double)s - (double)c;
  }
}

// mirror_vertical_horizontal (detector.py:246-275), then NaN/<=0 -> 1e-6 and
// the 1e-6 scale (comparison.py:859-868).
__global__ void k_det_epilogue(const double *q, int nv, int nh, int mirror,
                               double *out) {
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= nv * nh) return;
  const int i = pix / nh, j = pix % nh;
  const int i2 = nv - 1 - i, j2 = nh - 1 - j;
  double v = q[pix];
  if (mirror) {
    v = ((q[(size_t)i * nh + j] + q[(size_t)i * nh + j2]) + q[(size_t)i2 * nh + j]) +
        q[(size_t)i2 * nh + j2];
    const bool crow = (nv & 1) && i == nv / 2;
    const bool ccol = (nh & 1) && j == nh / 2;
    if (crow) v = (q[(size_t)i * nh + j] + q[(size_t)i * nh + j2]) * 2.0;
    if (ccol) v = (q[(size_t)i * nh + j] + q[(size_t)i2 * nh + j]) * 2.0;
    if (crow && ccol) v = q[(size_t)i * nh + j] * 4.0;
  }
  if (v != v) v = 1e-6;
  if (v <= 0.0) v = 1e-6;
  out[pix] = v * 1e-6;
}

__global__ void k_iq_to_f32(const double *in, float *out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (float)in[i];
}

__global__ void k_det_debug(DetArgs a, int o, int64_t *idx) {
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= a.nh * a.nv) return;
  double x, y, z;
  base_point(a, pix / a.nh, pix % a.nh, x, y, z);
  idx[pix] = gather_index(a, o, x, y, z);
}

// ---------------------------------------------------------------- fast path
// Per orientation, the composed rotation M = R_n...R_1 maps the base plane
// point p0 to index space: t = (M p0 - qmin) / dq = A p0 + b.  Evaluated in
// float32, t differs from the exact float64 replay by at most d (a bound the
// host derives from |A|, |p0| and |b|: 10 u S + 1e-5 with u = 2^-24 and S the
// sum of the magnitudes of the terms).  When floor(t-d) and floor(t+d) agree
// after clipping on all three axes the gathered voxel is the exact one;
// otherwise the (pixel, orientation) pair goes to a worklist that
// k_detector_fix replays with the exact float64 chain.
struct OrientFast {
  // an axis whose coordinate is exactly +-0 for every pixel has A = 0, b =
  // its (clipped) index + 0.5 and d = 0: it gathers that index, certainly (d is
  // infinite, and every sample replayed, for an index of 2^22 or more)
  float A[9];
  float b[3];
  float d[3];
  float w;
};
constexpr int kOrientFloats = sizeof(OrientFast) / 4;

constexpr int kDetChunk = 128, kDetFlush = 16;
static_assert(kDetChunk % kDetFlush == 0, "orientation chunks hold whole flush groups");
static_assert(kDetFlush * 2 <= 32, "a flush group's uncertain samples fit one 32-bit mask");

__device__ __forceinline__ bool fast_axis(float t, float d, int n, int &k) {
  // k = clamp(floor(t + d), 0, n-1) (clamping first is the same: NaN and
  // -inf give 0, +inf n-1), by magic-number rounding; clamp(floor(t - d))
  // equals it exactly when max(t - d, 0) >= k
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  const float c = fminf(fmaxf(t + d, 0.f), (float)(n - 1));
  const float r = __fadd_rn(c, kMagic);
  const float fr = __fsub_rn(r, kMagic);
  const bool down = fr > c;
  k = __float_as_int(r) - 0x4B400000 - (down ? 1 : 0);
  return fmaxf(t - d, 0.f) >= (down ? fr - 1.f : fr);
}

__device__ __forceinline__ bool fast_index(const OrientFast &T, const DetArgs &a,
                                           float x, float y, float z,
                                           int64_t &idx) {
  const float tx = fmaf(T.A[0], x, fmaf(T.A[1], y, fmaf(T.A[2], z, T.b[0])));
  const float ty = fmaf(T.A[3], x, fmaf(T.A[4], y, fmaf(T.A[5], z, T.b[1])));
  const float tz = fmaf(T.A[6], x, fmaf(T.A[7], y, fmaf(T.A[8], z, T.b[2])));
  int ix, iy, iz;
  const bool ok = fast_axis(tx, T.d[0], a.nx, ix) & fast_axis(ty, T.d[1], a.ny, iy) &
                  fast_axis(tz, T.d[2], a.nz, iz);
  idx = ((int64_t)iy * a.nx + ix) * a.nz + iz;
  return ok;
}

// ------------------------------------------------------------ plane mode
// When every orientation keeps the same axis at a fixed index (the plane
// rotated about its own normal, the reference's psi rotations), all samples
// lie in one plane of I(q).  The plane is copied to a compact nu x nv array
// (u, v the two free axes in memory order) and each block gathers from it
// through L1 (a copy of the plane in shared memory, where it fits, holds one
// block an SM: 91 rotations of 500 px in 203^2 59 us, without it 50).  A
// block's tile keeps its samples of one orientation within a compact patch of
// the plane.  Indices, worklist decisions and the per-pixel accumulation order are those of the general mode; only
// the order in which k_detector_fix atomically adds the replayed samples
// differs (it is scheduling order in both).
struct PlaneArgs {
  int fa, fi;   // fixed axis (0 x, 1 y, 2 z) and its index
  int ua, va;   // free axes, slower and faster in memory
  int nu, nv;
  const float *P;
};
// The two free rows of an orientation's affine map, packed for three
// 16-byte shared loads: (A_u, b_u), (A_v, b_v), (d_u, d_v, w, -).
// One orientation of the plane gather.  Each member pairs the u axis's
// value with the v axis's (x, y and z coefficients, constant, certainty
// bound), so that both axes' indices are made with paired float32
// instructions; w is the orientation's weight.  Three 16-byte words.
struct __align__(16) PlaneOrient {
  float2 x, y, z, c, d;
  float w, pad;
};
static_assert(sizeof(PlaneOrient) == 48, "three 16-byte words per orientation");
// First worklist slot of this lane's need set bits: one add per warp, as a
// pixel on an index' edge is uncertain at every orientation and an add and its
// answer per sample were the longest warp's time (203 x 203 pixels in
// 101^3, 720 orientations, some pixels at q = 0: 688 us so, now 215).  All lanes
// call.
__device__ __forceinline__ int worklist_slots(unsigned need, int *wl_count) {
  const int lane = threadIdx.x & 31, n = __popc(need);
  int end = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += v;
  }
  int base = 0;
  if (lane == 31) base = atomicAdd(wl_count, end);
  return __shfl_sync(0xffffffffu, base, 31) + end - n;
}

// A block owns a tile of 16 x 16 pixels, a thread two pixels kPlRows rows apart,
// a warp 8 x 4 and the same kPlRows below: small blocks, as a detector has few
// tiles and the last ones set the time (general mode, 2880 orientations of 500
// px 1.37 ms with 32 x 32 tiles, 1.20 with 16 x 16; 300 orientations of 500 px in
// 351^3 0.21 and 0.15 ms, but 0.30 with 16 x 8).  The samples of kPlBatch
// orientations are loaded before the first is used: 300 of 351^3 155 us with 2
// at a time, 153 with 4, 144 with 8; 91 rotations of 1000 px in the plane of
// 403^2 122 -> 108 us against one load at a time, 181 of 100 px 38 -> 25.
constexpr int kPlTile = 16, kPlThreads = 128, kPlRows = 8, kPlBatch = 8;
static_assert(kPlTile * kPlTile == 2 * kPlThreads, "two pixels a thread");
__device__ __forceinline__ int tile_col(int t) { return t / 32 % 2 * 8 + t % 8; }
__device__ __forceinline__ int tile_row(int t) { return t / 64 * 4 + t % 32 / 8; }

// A compile-time bool as a value (selects a lambda's instantiation).
template <bool B>
struct BoolC {
  static constexpr bool value = B;
};

__global__ void k_plane_extract(DetArgs a, PlaneArgs pa, float *P) {
  const int64_t n = (int64_t)pa.nu * pa.nv;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    int idx[3];
    idx[pa.fa] = pa.fi;
    idx[pa.ua] = (int)(t / pa.nv);
    idx[pa.va] = (int)(t % pa.nv);
    P[t] = a.iq[((int64_t)idx[1] * a.nx + idx[0]) * a.nz + idx[2]];
  }
}

// Both axes of fast_index on those rows, u in the first half of each pair
// and v in the second: t = (y c_y + (z c_z + c)) (same operation order), and
// for each axis fast_axis with the floor taken by one addition rounded
// toward minus infinity: r = 1.5 * 2^23 + floor(t + d) exactly for clamped
// values in [0, 2^22), so the index and the certainty test are those of
// fast_axis, in fewer operations.  The paired instructions round each half
// as the scalar ones.  n1 = (nu - 1, nv - 1) as floats.  ZX: the pixels' x
// is +-0 for every pixel, so the x products (exact zeros added to the rest
// of the chain) are left out: fmaf(a, +-0, c) == c for c != 0, and a signed
// zero does not change a floor.
template <bool ZX>
__device__ __forceinline__ bool plane_index(const PlaneOrient &T, float2 n1,
                                            float2 xx, float2 yy, float2 zz,
                                            int &iu, int &iv) {
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  const float2 mg = make_float2(kMagic, kMagic);
  float2 t = __ffma2_rn(T.y, yy, __ffma2_rn(T.z, zz, T.c));
  if (!ZX) t = __ffma2_rn(T.x, xx, t);
  const float2 hi = __fadd2_rn(t, T.d), lo = f2_sub(t, T.d);
  const float2 c = make_float2(fminf(fmaxf(hi.x, 0.f), n1.x), fminf(fmaxf(hi.y, 0.f), n1.y));
  const float2 r = __fadd2_rd(c, mg);
  iu = __float_as_int(r.x) - 0x4B400000;
  iv = __float_as_int(r.y) - 0x4B400000;
  const float2 fl = f2_sub(r, mg);
  return (fmaxf(lo.x, 0.f) >= fl.x) & (fmaxf(lo.y, 0.f) >= fl.y);
}

template <bool ZX>
__global__ void __launch_bounds__(kPlThreads)
k_detector_plane(DetArgs a, const PlaneOrient *ot, PlaneArgs pa,
                 double *acc_out, int2 *wl, int *wl_count, int wl_cap) {
  __shared__ PlaneOrient s_ot[kDetChunk];
  constexpr int KP = 2;  // pixels per thread
  const float2 n1 = make_float2((float)(pa.nu - 1), (float)(pa.nv - 1));
  const int tiles_x = (a.nh + kPlTile - 1) / kPlTile;
  const int j = (blockIdx.x % tiles_x) * kPlTile + tile_col(threadIdx.x);
  const int ib = (blockIdx.x / tiles_x) * kPlTile + tile_row(threadIdx.x);
  int pix[KP];
  bool valid[KP];
  float xf[KP], yf[KP], zf[KP];
  double acc[KP];
  float part[KP];
#pragma unroll
  for (int k = 0; k < KP; ++k) {
    const int i = ib + k * kPlRows;
    valid[k] = i < a.nv && j < a.nh;
    pix[k] = valid[k] ? i * a.nh + j : 0;
    double x0 = 0.0, y0 = 0.0, z0 = 0.0;
    if (valid[k]) base_point(a, i, j, x0, y0, z0);
    xf[k] = (float)x0; yf[k] = (float)y0; zf[k] = (float)z0;
    acc[k] = 0.0;
    part[k] = 0.f;
  }
  const unsigned vmask = (valid[0] ? 0x55555555u : 0u) | (valid[1] ? 0xaaaaaaaau : 0u);
  // tiles wholly inside the detector (all but the last tile row and
  // column) run the loop without the per-pixel validity tests
  auto orient_loop = [&](auto all_valid) {
    constexpr bool AV = decltype(all_valid)::value;
    for (int c0 = 0; c0 < a.n_orient; c0 += kDetChunk) {
      const int nc = min(kDetChunk, a.n_orient - c0);
      __syncthreads();
      for (int t = threadIdx.x; t < nc * 3; t += kPlThreads)
        reinterpret_cast<float4 *>(s_ot)[t] = reinterpret_cast<const float4 *>(ot + c0)[t];
      __syncthreads();
      // groups of kDetFlush orientations (chunks start at multiples of it),
      // two per loop trip, flushed to float64 after each full group
      for (int g0 = 0; g0 < nc; g0 += kDetFlush) {
        const int ge = min(g0 + kDetFlush, nc);
        // bit (oo - g0) KP + k: a sample whose index is not certain in
        // float32, replayed in float64 after the group
        unsigned need_bits = 0;
        for (int oo = g0; oo < ge; oo += kPlBatch) {
          // every index is clamped, so the samples of kPlBatch orientations are
          // loaded unconditionally, all in flight at once
          int at[kPlBatch][KP];
          float w[kPlBatch], v[kPlBatch][KP];
          unsigned ok = 0;
  #pragma unroll
          for (int b = 0; b < kPlBatch; ++b) {
            // three 16-byte loads; each holds two (u, v) pairs
            const float4 *q = reinterpret_cast<const float4 *>(s_ot + min(oo + b, ge - 1));
            const float4 q0 = q[0], q1 = q[1], q2 = q[2];
            PlaneOrient T;
            T.x = make_float2(q0.x, q0.y);
            T.y = make_float2(q0.z, q0.w);
            T.z = make_float2(q1.x, q1.y);
            T.c = make_float2(q1.z, q1.w);
            T.d = make_float2(q2.x, q2.y);
            w[b] = q2.z;
  #pragma unroll
            for (int k = 0; k < KP; ++k) {
              int iu, iv;
              const bool in = plane_index<ZX>(T, n1, make_float2(xf[k], xf[k]),
                                              make_float2(yf[k], yf[k]),
                                              make_float2(zf[k], zf[k]), iu, iv);
              at[b][k] = iu * pa.nv + iv;
              ok |= (unsigned)in << (b * KP + k);
            }
          }
  #pragma unroll
          for (int b = 0; b < kPlBatch; ++b)
  #pragma unroll
            for (int k = 0; k < KP; ++k) v[b][k] = __ldg(pa.P + at[b][k]);
          // (no samples of pixels outside the detector or past the group)
          unsigned want = (1u << (min(kPlBatch, ge - oo) * KP)) - 1u;
          if (!AV) want &= vmask;
          need_bits |= (want & ~ok) << ((oo - g0) * KP);
          ok &= want;
  #pragma unroll
          for (int b = 0; b < kPlBatch; ++b)
  #pragma unroll
            for (int k = 0; k < KP; ++k)
              if (ok >> (b * KP + k) & 1u) part[k] = fmaf(v[b][k], w[b], part[k]);
        }
        // the group's uncertain samples go to the worklist (replayed exactly
        // by k_detector_fix), or, once it is full, are replayed here into the
        // float64 accumulator
        if (__any_sync(0xffffffffu, need_bits != 0)) {
          int slot = worklist_slots(need_bits, wl_count);
          for (; need_bits; ++slot) {
            const int b = __ffs(need_bits) - 1;
            need_bits &= need_bits - 1;
            const int k = b % KP, o = c0 + g0 + b / KP;
            int px = pix[0];
  #pragma unroll
            for (int q = 1; q < KP; ++q)
              if (k == q) px = pix[q];
            if (slot < wl_cap) {
              wl[slot] = make_int2(px, o);
            } else {
              double x, y, z;
              base_point(a, px / a.nh, px % a.nh, x, y, z);
              const double sv = (double)__ldg(a.iq + gather_index(a, o, x, y, z)) * a.w[o];
  #pragma unroll
              for (int q = 0; q < KP; ++q)
                if (k == q) acc[q] += sv;
            }
          }
        }
        if (ge - g0 == kDetFlush) {
  #pragma unroll
          for (int k = 0; k < KP; ++k) { acc[k] += f2d_exact(part[k]); part[k] = 0.f; }
        }
      }
    }
  };
  const int tile_i = (blockIdx.x / tiles_x) * kPlTile, tile_j = (blockIdx.x % tiles_x) * kPlTile;
  if (tile_i + kPlTile <= a.nv && tile_j + kPlTile <= a.nh) orient_loop(BoolC<true>{});
  else orient_loop(BoolC<false>{});
#pragma unroll
  for (int k = 0; k < KP; ++k)
    if (valid[k]) acc_out[pix[k]] = acc[k] + f2d_exact(part[k]);
}

// ------------------------------------------------------------ general mode
// One orientation of the general gather, for two pixels a thread: (x, y)
// pairs of the coefficients of those two axes, (z, z) pairs of the z axis',
// so that an (x, y) pair of one pixel and a z pair of both pixels are each
// one paired float32 instruction.  Six 16-byte words.
struct __align__(16) GenOrient {
  float2 ax, ay, az, c, d;       // x and y axes: of pixel x, y, z; constant; bound
  float2 zx, zy, zz, zc, zd;     // z axis, twice
  float2 w;                      // weight, -
  float2 pad;
};
static_assert(sizeof(GenOrient) == 96, "six 16-byte words per orientation");

// Every orientation's samples of a pixel tile, two pixels a thread, gathered
// from the whole I(q).  The indices, certainty tests and order of the sums are
// those of fast_index with each floor taken by one addition rounded toward
// minus infinity (as in plane_index); an index is the 32-bit sum of the rounded
// additions' bit patterns less a constant, which is exact modulo 2^32 (I(q) has
// fewer than 2^32 elements).  Tiles keep a block's samples of one orientation
// within a small patch of the volume.  Bound by issue.  2880 orientations of
// 500 x 500 pixels in 203^3: 4.75 ms with one axis at a time, rows of 512
// pixels a block and 64-bit indices, 1.20 ms so.  WIDE: 64-bit indices, for I(q)
// of 2^32 elements and more (320 orientations of 500 x 500 pixels in 1626^3: 0.63 ms
// so, 8.30 with every sample's exact index; in 1600^3 0.56).
template <bool ZX, bool KAHAN, bool WIDE>
__global__ void __launch_bounds__(kPlThreads)
k_detector_general(DetArgs a, const GenOrient *ot, double *acc_out, int2 *wl, int *wl_count,
                   int wl_cap) {
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  constexpr int KP = 2;
  static_assert(kDetFlush * KP <= 32, "a group's uncertain samples fit one mask");
  __shared__ GenOrient s_ot[kDetChunk];
  const int tiles_x = (a.nh + kPlTile - 1) / kPlTile;
  const int j = (blockIdx.x % tiles_x) * kPlTile + tile_col(threadIdx.x);
  const int ib = (blockIdx.x / tiles_x) * kPlTile + tile_row(threadIdx.x);
  const float mx = (float)(a.nx - 1), my = (float)(a.ny - 1), mz = (float)(a.nz - 1);
  const unsigned nx = a.nx, nz = a.nz;
  constexpr unsigned kBits = 0x4B400000u;  // kMagic's
  const unsigned base = (kBits * nx + kBits) * nz + kBits;
  int pix[KP];
  bool valid[KP];
  float xf[KP], yf[KP], zf[KP], part[KP], kc[KP];
  double acc[KP];
#pragma unroll
  for (int k = 0; k < KP; ++k) {
    const int i = ib + k * kPlRows;
    valid[k] = i < a.nv && j < a.nh;
    pix[k] = valid[k] ? i * a.nh + j : 0;
    double x0 = 0.0, y0 = 0.0, z0 = 0.0;
    if (valid[k]) base_point(a, i, j, x0, y0, z0);
    xf[k] = (float)x0; yf[k] = (float)y0; zf[k] = (float)z0;
    acc[k] = 0.0;
    part[k] = kc[k] = 0.f;
  }
  const unsigned vmask = (valid[0] ? 0x55555555u : 0u) | (valid[1] ? 0xaaaaaaaau : 0u);
  const float2 px = make_float2(xf[0], xf[1]), py = make_float2(yf[0], yf[1]),
               pz = make_float2(zf[0], zf[1]);
  const float2 mg = make_float2(kMagic, kMagic);
  auto add = [&](int k, float v, float w) {
    if (!KAHAN) {
      part[k] = fmaf(v, w, part[k]);
    } else {
      const float y = v * w - kc[k];
      const float t = part[k] + y;
      kc[k] = (t - part[k]) - y;
      part[k] = t;
    }
  };
  for (int c0 = 0; c0 < a.n_orient; c0 += kDetChunk) {
    const int nc = min(kDetChunk, a.n_orient - c0);
    __syncthreads();
    for (int t = threadIdx.x; t < nc * 6; t += kPlThreads)
      reinterpret_cast<float4 *>(s_ot)[t] = reinterpret_cast<const float4 *>(ot + c0)[t];
    __syncthreads();
    for (int g0 = 0; g0 < nc; g0 += kDetFlush) {
      const int ge = min(g0 + kDetFlush, nc);
      unsigned need = 0;  // bit (oo - g0) KP + k: an uncertain sample
      for (int oo = g0; oo < ge; oo += kPlBatch) {
        // every index is clamped, so the samples of kPlBatch orientations are
        // loaded unconditionally, all in flight at once
        std::conditional_t<WIDE, int64_t, unsigned> at[kPlBatch][KP];
        unsigned ok = 0;
        float w[kPlBatch], v[kPlBatch][KP];
#pragma unroll
        for (int b = 0; b < kPlBatch; ++b) {
          const float4 *q = reinterpret_cast<const float4 *>(s_ot + min(oo + b, ge - 1));
          const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4];
          w[b] = q[5].x;
          const float2 cx = make_float2(q0.x, q0.y), cy = make_float2(q0.z, q0.w),
                       cz = make_float2(q1.x, q1.y), cc = make_float2(q1.z, q1.w),
                       cd = make_float2(q2.x, q2.y);
          // z axis of both pixels
          float2 t = __ffma2_rn(make_float2(q3.x, q3.y), py,
                                __ffma2_rn(make_float2(q3.z, q3.w), pz, make_float2(q4.x, q4.y)));
          if (!ZX) t = __ffma2_rn(make_float2(q2.z, q2.w), px, t);
          const float2 zd = make_float2(q4.z, q4.w);
          const float2 zhi = __fadd2_rn(t, zd), zlo = f2_sub(t, zd);
          const float2 zr = __fadd2_rd(
              make_float2(fminf(fmaxf(zhi.x, 0.f), mz), fminf(fmaxf(zhi.y, 0.f), mz)), mg);
          const float2 zfl = f2_sub(zr, mg);
#pragma unroll
          for (int k = 0; k < KP; ++k) {
            const float2 yy = make_float2(yf[k], yf[k]), zz = make_float2(zf[k], zf[k]);
            float2 u = __ffma2_rn(cy, yy, __ffma2_rn(cz, zz, cc));
            if (!ZX) u = __ffma2_rn(cx, make_float2(xf[k], xf[k]), u);
            const float2 hi = __fadd2_rn(u, cd), lo = f2_sub(u, cd);
            const float2 r = __fadd2_rd(
                make_float2(fminf(fmaxf(hi.x, 0.f), mx), fminf(fmaxf(hi.y, 0.f), my)), mg);
            const float2 fl = f2_sub(r, mg);
            const bool in = (fmaxf(lo.x, 0.f) >= fl.x) & (fmaxf(lo.y, 0.f) >= fl.y) &
                            (fmaxf(k ? zlo.y : zlo.x, 0.f) >= (k ? zfl.y : zfl.x));
            const unsigned ry = __float_as_uint(r.y), rx = __float_as_uint(r.x),
                           rz = __float_as_uint(k ? zr.y : zr.x);
            if constexpr (WIDE)
              at[b][k] = ((int64_t)(ry - kBits) * nx + (rx - kBits)) * nz + (rz - kBits);
            else
              at[b][k] = (ry * nx + rx) * nz + rz - base;
            ok |= (unsigned)in << (b * KP + k);
          }
        }
#pragma unroll
        for (int b = 0; b < kPlBatch; ++b)
#pragma unroll
          for (int k = 0; k < KP; ++k) v[b][k] = __ldg(a.iq + at[b][k]);
        // (no samples of pixels outside the detector or past the group)
        const unsigned want = vmask & ((1u << (min(kPlBatch, ge - oo) * KP)) - 1u);
        need |= (want & ~ok) << ((oo - g0) * KP);
        ok &= want;
#pragma unroll
        for (int b = 0; b < kPlBatch; ++b)
#pragma unroll
          for (int k = 0; k < KP; ++k)
            if (ok >> (b * KP + k) & 1u) add(k, v[b][k], w[b]);
      }
      // uncertain samples: to the worklist (k_detector_fix), or replayed
      // here once it is full
      if (__any_sync(0xffffffffu, need != 0)) {
        int slot = worklist_slots(need, wl_count);
        for (; need; ++slot) {
          const int b = __ffs(need) - 1;
          need &= need - 1;
          const int k = b % KP, o = c0 + g0 + b / KP, p = k ? pix[1] : pix[0];
          if (slot < wl_cap) {
            wl[slot] = make_int2(p, o);
          } else {
            double x, y, z;
            base_point(a, p / a.nh, p % a.nh, x, y, z);
            const float v = __ldg(a.iq + gather_index(a, o, x, y, z));
            if (k == 0) add(0, v, (float)a.w[o]);
            else add(1, v, (float)a.w[o]);
          }
        }
      }
      // float32 partial sums of kDetFlush orientations, float64 across them
      if (!KAHAN && ge - g0 == kDetFlush) {
#pragma unroll
        for (int k = 0; k < KP; ++k) { acc[k] += f2d_exact(part[k]); part[k] = 0.f; }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KP; ++k)
    if (valid[k])
      acc_out[pix[k]] = KAHAN ? f2d_exact(part[k]) - f2d_exact(kc[k]) : acc[k] + f2d_exact(part[k]);
}

// Exact float64 replay of the worklist's (pixel, orientation) pairs.
__global__ void k_detector_fix(DetArgs a, const int2 *wl, const int *wl_count,
                               int wl_cap, double *acc) {
  const int n = min(*wl_count, wl_cap);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += gridDim.x * blockDim.x) {
    const int2 it = wl[e];
    double x, y, z;
    base_point(a, it.x / a.nh, it.x % a.nh, x, y, z);
    const float v = __ldg(a.iq + gather_index(a, it.y, x, y, z));
    atomicAdd(acc + it.x, (double)v * a.w[it.y]);
  }
}

// ------------------------------------------------------------------ adjoint
// Transpose of the epilogue: the image is out = 1e-6 * max'(mirror(acc))
// with max' the NaN/<=0 -> 1e-6 clamp (zero derivative where it acts) and
// mirror the sum over the four flips (a symmetric map: each output pixel
// sums its orbit under the flips, with multiplicity).  Hence
// dL/dacc[p] = 1e-6 * [v_p > 0] * sum over the flips q of p of dL/dout[q],
// v = mirror(acc) being constant on the orbit.
__global__ void k_det_epi_adj(const double *acc, const double *gout, int nv,
                              int nh, int mirror, double *gpix) {
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= nv * nh) return;
  const int i = pix / nh, j = pix % nh;
  const int i2 = nv - 1 - i, j2 = nh - 1 - j;
  const size_t q0 = (size_t)i * nh + j, q1 = (size_t)i * nh + j2,
               q2 = (size_t)i2 * nh + j, q3 = (size_t)i2 * nh + j2;
  double v, g;
  if (mirror) {
    v = ((acc[q0] + acc[q1]) + acc[q2]) + acc[q3];
    g = gout[q0] + gout[q1] + gout[q2] + gout[q3];
  } else {
    v = acc[q0];
    g = gout[q0];
  }
  gpix[pix] = (v == v && v > 0.0) ? 1e-6 * g : 0.0;
}

// Transpose of the orientation sum: every (pixel, orientation) sample adds
// w_o dL/dacc[pixel] to dL/dI at the voxel it gathered.  Indices come from
// the same float32 estimate with exact float64 replay as the forward (the
// ambiguous samples are replayed inline), so they are the forward's.  Bound by
// the float64 adds in L2: a thread takes a square of 2 x 2 pixels, a voxel of
// I(q) covers several, and adds each run of pixels of one voxel once.  The
// orientations are split over blockIdx.y (per_block each) until the blocks
// fill the GPU.  91 rotations of 512 px in 149^3, image and adjoint together:
// 313 us with one pixel a thread, 208 so; 31 of 257 px in 90^3 85 and 53.
constexpr int kAdjThreads = 128, kAdjW = 32, kAdjH = 16, kAdjChunk = 64;
__global__ void __launch_bounds__(kAdjThreads)
k_detector_adj(DetArgs a, const OrientFast *ot, const double *gpix, int per_block,
               double *g_iq) {
  __shared__ OrientFast s_ot[kAdjChunk];
  constexpr int KP = 4;
  const int tiles_x = (a.nh + kAdjW - 1) / kAdjW, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int j0 = blockIdx.x % tiles_x * kAdjW + wp % 2 * 16 + lane % 8 * 2;
  const int i0 = blockIdx.x / tiles_x * kAdjH + wp / 2 * 8 + lane / 8 * 2;
  double x0[KP], y0[KP], z0[KP], g[KP];
  float xf[KP], yf[KP], zf[KP];
  bool live[KP], any = false;
#pragma unroll
  for (int k = 0; k < KP; ++k) {
    const int i = i0 + k / 2, j = j0 + (k / 2 ? 1 - k % 2 : k % 2);  // around the square
    x0[k] = y0[k] = z0[k] = g[k] = 0.0;
    if (i < a.nv && j < a.nh) {
      base_point(a, i, j, x0[k], y0[k], z0[k]);
      g[k] = gpix[(size_t)i * a.nh + j];
    }
    live[k] = g[k] != 0.0;
    any |= live[k];
    xf[k] = (float)x0[k]; yf[k] = (float)y0[k]; zf[k] = (float)z0[k];
  }
  const int o_end = min(a.n_orient, ((int)blockIdx.y + 1) * per_block);
  for (int c0 = blockIdx.y * per_block; c0 < o_end; c0 += kAdjChunk) {
    const int nc = min(kAdjChunk, o_end - c0);
    __syncthreads();
    for (int t = threadIdx.x; t < nc * kOrientFloats; t += kAdjThreads)
      reinterpret_cast<float *>(s_ot)[t] = reinterpret_cast<const float *>(ot + c0)[t];
    __syncthreads();
    if (!any) continue;
    for (int oo = 0; oo < nc; ++oo) {
      const double w = a.w[c0 + oo];
      int64_t cur = -1;
      double sum = 0.0;
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        if (!live[k]) continue;
        int64_t idx;
        if (!fast_index(s_ot[oo], a, xf[k], yf[k], zf[k], idx))
          idx = gather_index(a, c0 + oo, x0[k], y0[k], z0[k]);
        if (idx == cur) {
          sum += g[k];
        } else {
          if (cur >= 0) atomicAdd(g_iq + cur, sum * w);
          cur = idx;
          sum = g[k];
        }
      }
      if (cur >= 0) atomicAdd(g_iq + cur, sum * w);
    }
  }
}

__global__ void k_detector_adj_exact(DetArgs a, const double *gpix,
                                     double *g_iq) {
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= a.nh * a.nv) return;
  const double g = gpix[pix];
  if (g == 0.0) return;
  double x0, y0, z0;
  base_point(a, pix / a.nh, pix % a.nh, x0, y0, z0);
  for (int o = 0; o < a.n_orient; ++o)
    atomicAdd(g_iq + gather_index(a, o, x0, y0, z0), g * a.w[o]);
}

__global__ void k_det_debug_fast(DetArgs a, const OrientFast *ot, int o,
                                 int64_t *idx) {
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= a.nh * a.nv) return;
  double x, y, z;
  base_point(a, pix / a.nh, pix % a.nh, x, y, z);
  int64_t k;
  if (!fast_index(ot[o], a, (float)x, (float)y, (float)z, k))
    k = gather_index(a, o, x, y, z);
  idx[pix] = k;
}

}  // namespace

struct gw_detector_plan {
  gw_ctx *ctx = nullptr;
  gw_detector_params p{};
  int n_orient = 0, n_init = 0;
  double *d_h = nullptr, *d_v = nullptr, *d_init = nullptr, *d_rot = nullptr,
         *d_w = nullptr;
  int *d_rs = nullptr, *d_rn = nullptr;
  float *d_iq_own = nullptr;
  const float *iq = nullptr;
  double *d_acc = nullptr, *d_out = nullptr;
  OrientFast *d_ot = nullptr;   // fast-path orientation table
  int2 *d_wl = nullptr;         // exact-replay worklist
  int *d_wl_count = nullptr;
  int wl_cap = 0;
  double *d_gout = nullptr, *d_gpix = nullptr, *d_giq = nullptr;  // adjoint
  PlaneArgs plane{-1, -1, 0, 0, 0, 0, nullptr};  // plane mode when fa >= 0
  float *d_plane = nullptr;
  // d_plane64 holds the plane of the I(q) that gw_detector_set_iq gave (only
  // that plane was taken); otherwise execute copies the plane from iq
  bool plane_set = false;
  double *d_plane64 = nullptr;
  PlaneOrient *d_po = nullptr;
  GenOrient *d_go = nullptr;    // general mode
  bool zero_x = false;  // every pixel's x is +-0 after the init rotations
  bool executed = false;
};

namespace {
DetArgs det_args(gw_detector_plan *P) {
  DetArgs a{};
  a.nh = P->p.n_h; a.nv = P->p.n_v;
  a.ny = P->p.iq_shape[0]; a.nx = P->p.iq_shape[1]; a.nz = P->p.iq_shape[2];
  a.qmin_x = P->p.qmin_x; a.qmin_y = P->p.qmin_y; a.qmin_z = P->p.qmin_z;
  a.dq = P->p.dq; a.inv_dq = 1.0 / P->p.dq;
  a.h = P->d_h; a.v = P->d_v; a.init_R = P->d_init; a.n_init = P->n_init;
  a.rot_start = P->d_rs; a.rot_n = P->d_rn; a.rot_R = P->d_rot; a.w = P->d_w;
  a.n_orient = P->n_orient; a.iq = P->iq;
  a.sy = (int64_t)a.nx * a.nz; a.sx = a.nz; a.sz = 1;
  a.kahan = P->p.accum == GW_ACCUM_KAHAN32;
  return a;
}

template <typename T>
int up(T **dst, const T *src, size_t n) {
  if (n == 0) { *dst = nullptr; return GW_OK; }
  GW_CUDA(gw::dev_malloc((void **)dst, n * sizeof(T)));
  GW_CUDA(cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice));
  return GW_OK;
}
}  // namespace

extern "C" int gw_detector_plan_create(gw_ctx *ctx, const gw_detector_params *p,
                                       const double *h_axis, const double *v_axis,
                                       const double *init_R, int32_t n_init,
                                       const int32_t *n_rot, const double *rot_R,
                                       const double *weights, int32_t n_orient,
                                       gw_detector_plan **out) {
  if (!ctx || !p || !h_axis || !v_axis || !out || !weights || !n_rot)
    return gw::fail(GW_ERR_ARG, "gw_detector_plan_create: null argument");
  if (p->n_h < 1 || p->n_v < 1 || n_orient < 1 || n_init < 0 || n_init > 3 ||
      p->iq_shape[0] < 1 || p->iq_shape[1] < 1 || p->iq_shape[2] < 1 || !(p->dq > 0))
    return gw::fail(GW_ERR_ARG, "gw_detector_plan_create: invalid sizes");
  if (n_init > 0 && !init_R)
    return gw::fail(GW_ERR_ARG, "gw_detector_plan_create: init_R missing");
  std::vector<int> rs(n_orient), rn(n_orient);
  int total = 0;
  for (int o = 0; o < n_orient; ++o) {
    if (n_rot[o] < 0 || n_rot[o] > 3)
      return gw::fail(GW_ERR_ARG, "gw_detector_plan_create: 0..3 rotations per orientation");
    rs[o] = total;
    rn[o] = n_rot[o];
    total += n_rot[o];
  }
  if (total > 0 && !rot_R)
    return gw::fail(GW_ERR_ARG, "gw_detector_plan_create: rot_R missing");
  GW_CUDA(cudaSetDevice(ctx->device));
  auto *P = new gw_detector_plan();
  P->ctx = ctx;
  P->p = *p;
  P->n_orient = n_orient;
  P->n_init = n_init;
  const size_t npx = (size_t)p->n_h * p->n_v;
  int st;
  if ((st = up(&P->d_h, h_axis, p->n_h)) || (st = up(&P->d_v, v_axis, p->n_v)) ||
      (st = up(&P->d_init, init_R, (size_t)9 * n_init)) ||
      (st = up(&P->d_rot, rot_R, (size_t)9 * total)) ||
      (st = up(&P->d_w, weights, (size_t)n_orient)) ||
      (st = up(&P->d_rs, rs.data(), rs.size())) ||
      (st = up(&P->d_rn, rn.data(), rn.size()))) {
    gw_detector_plan_destroy(P);
    return st;
  }
  cudaError_t e = gw::dev_malloc((void **)&P->d_acc, npx * sizeof(double));
  if (e == cudaSuccess) e = gw::dev_malloc((void **)&P->d_out, npx * sizeof(double));
  if (e != cudaSuccess) {
    gw_detector_plan_destroy(P);
    return gw::cuda_fail(e, "detector buffers", __FILE__, __LINE__);
  }
  if (!p->exact) {
    // corners of the base plane after the initial rotations bound |p0|
    double pmax[3] = {0, 0, 0};
    const double hs[2] = {h_axis[0], h_axis[p->n_h - 1]};
    const double vs[2] = {v_axis[0], v_axis[p->n_v - 1]};
    for (double hh : hs)
      for (double vv : vs) {
        double c[3] = {0.0, hh, vv};
        for (int k = 0; k < n_init; ++k) {
          const double *R = init_R + 9 * k;
          const double a0 = rot_chain(R, c[0], c[1], c[2]);
          const double a1 = rot_chain(R + 3, c[0], c[1], c[2]);
          const double a2 = rot_chain(R + 6, c[0], c[1], c[2]);
          c[0] = a0; c[1] = a1; c[2] = a2;
        }
        for (int k = 0; k < 3; ++k) pmax[k] = std::max(pmax[k], std::fabs(c[k]) * (1 + 1e-12));
      }
    const double inv_dq = 1.0 / p->dq;
    const double qmin[3] = {p->qmin_x, p->qmin_y, p->qmin_z};
    const int dims[3] = {p->iq_shape[1], p->iq_shape[0], p->iq_shape[2]};  // x, y, z
    // Axes whose coordinate is exactly +-0 for every pixel: the plane starts
    // at x = 0 (detector.py:27); a rotation keeps output c at +-0 when each
    // of its row-c entries is 0 or multiplies a coordinate that is +-0
    // (fma of exact zeros).  Such an axis gathers index floor((0-qmin)/dq),
    // a constant; deciding it in float32 would be ambiguous whenever q=0
    // lies on a voxel boundary.
    auto propagate = [](const double *R, const bool in[3], bool out[3]) {
      for (int c = 0; c < 3; ++c) {
        bool z = true;
        for (int k = 0; k < 3; ++k) z = z && (R[3 * c + k] == 0.0 || in[k]);
        out[c] = z;
      }
    };
    bool zero0[3] = {true, false, false};
    for (int k = 0; k < n_init; ++k) {
      bool nz[3];
      propagate(init_R + 9 * k, zero0, nz);
      std::copy(nz, nz + 3, zero0);
    }
    P->zero_x = zero0[0];
    std::vector<OrientFast> ot(n_orient);
    std::vector<int> fix(3 * (size_t)n_orient);  // index of an exactly +-0 axis, or -1
    for (int o = 0; o < n_orient; ++o) {
      bool zero[3] = {zero0[0], zero0[1], zero0[2]};
      for (int r = 0; r < rn[o]; ++r) {
        bool nz[3];
        propagate(rot_R + 9 * (rs[o] + r), zero, nz);
        std::copy(nz, nz + 3, zero);
      }
      double M[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
      for (int r = 0; r < rn[o]; ++r) {
        const double *R = rot_R + 9 * (rs[o] + r);
        double T[9];
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j)
            T[3 * i + j] = R[3 * i] * M[j] + R[3 * i + 1] * M[3 + j] + R[3 * i + 2] * M[6 + j];
        std::copy(T, T + 9, M);
      }
      for (int c = 0; c < 3; ++c) {
        double S = std::fabs(qmin[c] * inv_dq);
        for (int k = 0; k < 3; ++k) {
          ot[o].A[3 * c + k] = (float)(M[3 * c + k] * inv_dq);
          S += std::fabs(M[3 * c + k] * inv_dq) * pmax[k];
        }
        ot[o].b[c] = (float)(-qmin[c] * inv_dq);
        ot[o].d[c] = (float)(10.0 * std::ldexp(1.0, -24) * S + 1e-5);
        fix[3 * o + c] = -1;
        if (zero[c]) {
          double k = floor_div_exact(0.0 - qmin[c], p->dq, inv_dq);
          k = std::min(std::max(k, 0.0), (double)(dims[c] - 1));
          fix[3 * o + c] = (int)k;
          for (int j = 0; j < 3; ++j) ot[o].A[3 * c + j] = 0.f;
          ot[o].b[c] = (float)k + 0.5f;
          // (beyond 2^22 the float32 floors are not exact: always replayed)
          ot[o].d[c] = k < 4194304.0 ? 0.f : INFINITY;
        }
      }
      ot[o].w = (float)weights[o];
    }
    const int64_t pairs = (int64_t)npx * n_orient;
    P->wl_cap = (int)std::max<int64_t>(1 << 16, std::min<int64_t>(pairs / 8, 1 << 26));
    // GW_DET_WORKLIST_CAP shrinks the worklist (tests use it to exercise the
    // in-kernel exact path taken when the list is full)
    if (const char *cap = getenv("GW_DET_WORKLIST_CAP")) P->wl_cap = std::max(1, atoi(cap));
    if ((st = up(&P->d_ot, ot.data(), ot.size()))) {
      gw_detector_plan_destroy(P);
      return st;
    }
    e = gw::dev_malloc((void **)&P->d_wl, (size_t)P->wl_cap * sizeof(int2));
    if (e == cudaSuccess) e = gw::dev_malloc((void **)&P->d_wl_count, sizeof(int));
    if (e != cudaSuccess) {
      gw_detector_plan_destroy(P);
      return gw::cuda_fail(e, "detector worklist", __FILE__, __LINE__);
    }
    // plane mode: one axis at the same fixed index in every orientation
    if (p->accum != GW_ACCUM_KAHAN32 && !p->no_plane) {
      for (int c = 0; c < 3 && P->plane.fa < 0; ++c) {
        bool same = true;
        for (int o = 0; o < n_orient && same; ++o)
          same = fix[3 * o + c] >= 0 && fix[3 * o + c] == fix[c];
        if (!same) continue;
        // free axes in memory order (y, x, z)
        const int order[3] = {1, 0, 2};
        int fr[2], k = 0;
        for (int q : order)
          if (q != c) fr[k++] = q;
        PlaneArgs pa{c, fix[c], fr[0], fr[1], dims[fr[0]], dims[fr[1]], nullptr};
        e = gw::dev_malloc((void **)&P->d_plane, (size_t)pa.nu * pa.nv * sizeof(float));
        if (e != cudaSuccess) {
          gw_detector_plan_destroy(P);
          return gw::cuda_fail(e, "detector plane", __FILE__, __LINE__);
        }
        pa.P = P->d_plane;
        P->plane = pa;
        std::vector<PlaneOrient> po(n_orient);
        for (int o = 0; o < n_orient; ++o) {
          const OrientFast &T = ot[o];
          po[o].x = make_float2(T.A[3 * pa.ua], T.A[3 * pa.va]);
          po[o].y = make_float2(T.A[3 * pa.ua + 1], T.A[3 * pa.va + 1]);
          po[o].z = make_float2(T.A[3 * pa.ua + 2], T.A[3 * pa.va + 2]);
          po[o].c = make_float2(T.b[pa.ua], T.b[pa.va]);
          po[o].d = make_float2(T.d[pa.ua], T.d[pa.va]);
          po[o].w = T.w;
          po[o].pad = 0.f;
        }
        if ((st = up(&P->d_po, po.data(), po.size()))) {
          gw_detector_plan_destroy(P);
          return st;
        }
      }
    }
    if (P->plane.fa < 0) {
      auto two = [](float v) { return make_float2(v, v); };
      std::vector<GenOrient> go(n_orient);
      for (int o = 0; o < n_orient; ++o) {
        const OrientFast &T = ot[o];
        go[o] = GenOrient{make_float2(T.A[0], T.A[3]), make_float2(T.A[1], T.A[4]),
                          make_float2(T.A[2], T.A[5]), make_float2(T.b[0], T.b[1]),
                          make_float2(T.d[0], T.d[1]), two(T.A[6]), two(T.A[7]), two(T.A[8]),
                          two(T.b[2]), two(T.d[2]), make_float2(T.w, 0.f), two(0.f)};
      }
      if ((st = up(&P->d_go, go.data(), go.size()))) {
        gw_detector_plan_destroy(P);
        return st;
      }
    }
  }
  *out = P;
  return GW_OK;
}

extern "C" int gw_detector_plan_destroy(gw_detector_plan *P) {
  if (!P) return GW_OK;
  void *ptrs[] = {P->d_h, P->d_v, P->d_init, P->d_rot, P->d_w, P->d_rs,
                  P->d_rn, P->d_iq_own, P->d_acc, P->d_out, P->d_ot, P->d_wl,
                  P->d_wl_count, P->d_gout, P->d_gpix, P->d_giq, P->d_plane,
                  P->d_po, P->d_plane64, P->d_go};
  for (void *q : ptrs) gw::dev_free(q);
  delete P;
  return GW_OK;
}

// Plane mode reads one plane of I(q) (nu x nv elements): with x or y fixed
// its lines are nz contiguous elements, and one 2-D copy takes them alone.
// 403^3 float64 from pageable memory, x fixed: 1.3 of 524 MB, a call of
// detectormaker_fitting (1000 px, 91 psi) without the 3.0 ms of upload and
// conversion (8.6 ms before, 0.6 to 1.2 by host with the orientation matrices made
// at once).
static int set_iq_plane(gw_detector_plan *P, const double *iq, int32_t on_device) {
  const PlaneArgs &pa = P->plane;
  const size_t nx = P->p.iq_shape[1], nz = P->p.iq_shape[2];
  const size_t line = (size_t)pa.nv * sizeof(double);
  const double *src = iq + (size_t)pa.fi * (pa.fa == 0 ? nz : nx * nz);
  const size_t pitch = (pa.fa == 0 ? nx * nz : nz) * sizeof(double);
  if (!P->d_plane64)
    GW_CUDA(gw::dev_malloc((void **)&P->d_plane64, (size_t)pa.nu * line));
  GW_CUDA(cudaMemcpy2DAsync(P->d_plane64, line, src, pitch, line, pa.nu,
                            on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                            P->ctx->stream));
  // the caller's array is free to change on return
  if (!on_device) GW_CUDA(cudaStreamSynchronize(P->ctx->stream));
  P->iq = nullptr;
  P->plane_set = true;
  return GW_OK;
}

extern "C" int gw_detector_set_iq(gw_detector_plan *P, const double *iq,
                                  int32_t on_device) {
  if (!P || !iq) return gw::fail(GW_ERR_ARG, "gw_detector_set_iq: null argument");
  const int64_t n = (int64_t)P->p.iq_shape[0] * P->p.iq_shape[1] * P->p.iq_shape[2];
  if (P->plane.fa == 0 || P->plane.fa == 1) return set_iq_plane(P, iq, on_device);
  if (!P->d_iq_own)
    GW_CUDA(gw::dev_malloc((void **)&P->d_iq_own, n * sizeof(float)));
  const double *src = iq;
  double *tmp = nullptr;
  if (!on_device) {
    GW_CUDA(gw::dev_malloc((void **)&tmp, n * sizeof(double)));
    cudaError_t e = cudaMemcpyAsync(tmp, iq, n * sizeof(double),
                                    cudaMemcpyHostToDevice, P->ctx->stream);
    if (e != cudaSuccess) { gw::dev_free(tmp); return gw::cuda_fail(e, "iq upload", __FILE__, __LINE__); }
    src = tmp;
  }
  const int blocks = (int)std::min<int64_t>((n + 255) / 256, 8 * P->ctx->sm_count);
  gw::KTimer tm(P->ctx, GW_K_MISC);
  k_iq_to_f32<<<blocks, 256, 0, P->ctx->stream>>>(src, P->d_iq_own, n);
  P->ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (tmp) {
    if (e == cudaSuccess) e = cudaStreamSynchronize(P->ctx->stream);
    gw::dev_free(tmp);
  }
  if (e != cudaSuccess) return gw::cuda_fail(e, "iq conversion", __FILE__, __LINE__);
  P->iq = P->d_iq_own;
  P->plane_set = false;
  return GW_OK;
}

extern "C" int gw_detector_set_iq32_device(gw_detector_plan *P, const float *iq32) {
  if (!P || !iq32) return gw::fail(GW_ERR_ARG, "gw_detector_set_iq32_device: null argument");
  P->iq = iq32;
  P->plane_set = false;
  return GW_OK;
}

namespace {

int tile_count(const gw_detector_plan *P) {
  return ((P->p.n_h + kPlTile - 1) / kPlTile) * ((P->p.n_v + kPlTile - 1) / kPlTile);
}

void launch_plane(gw_detector_plan *P, const DetArgs &a) {
  const PlaneArgs pa = P->plane;
  const int tiles = tile_count(P);
  auto run = [&](auto kernel) {
    kernel<<<tiles, kPlThreads, 0, P->ctx->stream>>>(a, P->d_po, pa, P->d_acc, P->d_wl,
                                                     P->d_wl_count, P->wl_cap);
  };
  P->zero_x ? run(k_detector_plane<true>) : run(k_detector_plane<false>);
}

void launch_general(gw_detector_plan *P, const DetArgs &a) {
  const int tiles = tile_count(P);
  auto run = [&](auto kernel) {
    kernel<<<tiles, kPlThreads, 0, P->ctx->stream>>>(a, P->d_go, P->d_acc, P->d_wl,
                                                     P->d_wl_count, P->wl_cap);
  };
  const bool kahan = P->p.accum == GW_ACCUM_KAHAN32;
  // (the 32-bit gather index holds volumes of fewer than 2^32 elements)
  if ((double)a.nx * a.ny * a.nz >= 4294967296.0) {
    if (kahan) P->zero_x ? run(k_detector_general<true, true, true>)
                         : run(k_detector_general<false, true, true>);
    else P->zero_x ? run(k_detector_general<true, false, true>)
                   : run(k_detector_general<false, false, true>);
  } else {
    if (kahan) P->zero_x ? run(k_detector_general<true, true, false>)
                         : run(k_detector_general<false, true, false>);
    else P->zero_x ? run(k_detector_general<true, false, false>)
                   : run(k_detector_general<false, false, false>);
  }
}

}  // namespace

extern "C" int gw_detector_execute(gw_detector_plan *P) {
  if (!P) return gw::fail(GW_ERR_ARG, "gw_detector_execute: null plan");
  if (!P->iq && !P->plane_set)
    return gw::fail(GW_ERR_STATE, "gw_detector_execute: I(q) not set");
  GW_CUDA(cudaSetDevice(P->ctx->device));
  gw::Range r("giwaxsim: detector image");
  const int npx = P->p.n_h * P->p.n_v;
  DetArgs a = det_args(P);
  if (P->p.exact) {
    gw::KTimer tm(P->ctx, GW_K_DETECTOR);
    k_detector<<<(npx + 127) / 128, 128, 0, P->ctx->stream>>>(a, P->d_acc);
    GW_LAUNCHED(P->ctx);
  } else {
    GW_CUDA(cudaMemsetAsync(P->d_wl_count, 0, sizeof(int), P->ctx->stream));
    if (P->plane.fa >= 0) {
      const PlaneArgs &pa = P->plane;
      {
        gw::KTimer tm(P->ctx, GW_K_MISC);
        const int64_t n = (int64_t)pa.nu * pa.nv;
        const int blocks = (int)std::min<int64_t>((n + 255) / 256, 4 * P->ctx->sm_count);
        if (P->plane_set) {
          k_iq_to_f32<<<blocks, 256, 0, P->ctx->stream>>>(P->d_plane64, P->d_plane, n);
          // exact replays read the plane: the fixed axis' index is always fi
          int64_t st[3] = {0, 0, 0};
          st[pa.ua] = pa.nv;
          st[pa.va] = 1;
          a.iq = P->d_plane;
          a.sx = st[0]; a.sy = st[1]; a.sz = st[2];
        } else {
          k_plane_extract<<<blocks, 256, 0, P->ctx->stream>>>(a, pa, P->d_plane);
        }
        GW_LAUNCHED(P->ctx);
      }
      gw::KTimer tm(P->ctx, GW_K_DETECTOR);
      launch_plane(P, a);
      GW_LAUNCHED(P->ctx);
    } else {
      gw::KTimer tm(P->ctx, GW_K_DETECTOR);
      launch_general(P, a);
      GW_LAUNCHED(P->ctx);
    }
    gw::KTimer tm(P->ctx, GW_K_DET_FIX);
    k_detector_fix<<<2 * P->ctx->sm_count, 256, 0, P->ctx->stream>>>(
        a, P->d_wl, P->d_wl_count, P->wl_cap, P->d_acc);
    GW_LAUNCHED(P->ctx);
  }
  gw::KTimer tm(P->ctx, GW_K_DET_EPI);
  k_det_epilogue<<<(npx + 255) / 256, 256, 0, P->ctx->stream>>>(
      P->d_acc, P->p.n_v, P->p.n_h, P->p.mirror, P->d_out);
  GW_LAUNCHED(P->ctx);
  P->executed = true;
  return GW_OK;
}

extern "C" int gw_detector_device_out(gw_detector_plan *P, const double **out) {
  if (!P || !out) return gw::fail(GW_ERR_ARG, "gw_detector_device_out: null argument");
  *out = P->d_out;
  return GW_OK;
}

extern "C" int gw_detector_get(gw_detector_plan *P, double *out, int32_t on_device) {
  if (!P || !out) return gw::fail(GW_ERR_ARG, "gw_detector_get: null argument");
  if (!P->executed) return gw::fail(GW_ERR_STATE, "gw_detector_get: plan not executed");
  const size_t npx = (size_t)P->p.n_h * P->p.n_v;
  GW_CUDA(cudaMemcpyAsync(out, P->d_out, npx * sizeof(double),
                          on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                          P->ctx->stream));
  return gw::check_device_error(P->ctx, "detector stage");
}

extern "C" int gw_detector_backward(gw_detector_plan *P, const double *g_out,
                                    int32_t out_on_device, double *g_iq,
                                    int32_t iq_on_device) {
  if (!P || !g_out || !g_iq)
    return gw::fail(GW_ERR_ARG, "gw_detector_backward: null argument");
  if (!P->executed)
    return gw::fail(GW_ERR_STATE, "gw_detector_backward: plan not executed");
  GW_CUDA(cudaSetDevice(P->ctx->device));
  const int npx = P->p.n_h * P->p.n_v;
  const size_t niq = (size_t)P->p.iq_shape[0] * P->p.iq_shape[1] * P->p.iq_shape[2];
  cudaStream_t st = P->ctx->stream;
  if (!P->d_gpix) {
    GW_CUDA(gw::dev_malloc((void **)&P->d_gpix, npx * sizeof(double)));
    GW_CUDA(gw::dev_malloc((void **)&P->d_gout, npx * sizeof(double)));
  }
  const double *gout = g_out;
  if (!out_on_device) {
    GW_CUDA(cudaMemcpyAsync(P->d_gout, g_out, npx * sizeof(double),
                            cudaMemcpyHostToDevice, st));
    gout = P->d_gout;
  }
  double *giq = g_iq;
  if (!iq_on_device) {
    if (!P->d_giq) GW_CUDA(gw::dev_malloc((void **)&P->d_giq, niq * sizeof(double)));
    giq = P->d_giq;
  }
  GW_CUDA(cudaMemsetAsync(giq, 0, niq * sizeof(double), st));
  {
    gw::KTimer tm(P->ctx, GW_K_DET_EPI);
    k_det_epi_adj<<<(npx + 255) / 256, 256, 0, st>>>(P->d_acc, gout, P->p.n_v,
                                                     P->p.n_h, P->p.mirror, P->d_gpix);
    GW_LAUNCHED(P->ctx);
  }
  DetArgs a = det_args(P);
  {
    gw::KTimer tm(P->ctx, GW_K_DETECTOR);
    if (P->p.exact)
      k_detector_adj_exact<<<(npx + 127) / 128, 128, 0, st>>>(a, P->d_gpix, giq);
    else {
      const int tiles = ((P->p.n_h + kAdjW - 1) / kAdjW) * ((P->p.n_v + kAdjH - 1) / kAdjH);
      const int splits = std::min((8 * P->ctx->sm_count + tiles - 1) / tiles, (P->n_orient + 7) / 8);
      const int per_block = (P->n_orient + splits - 1) / splits;
      k_detector_adj<<<dim3(tiles, (P->n_orient + per_block - 1) / per_block), kAdjThreads, 0,
                       st>>>(a, P->d_ot, P->d_gpix, per_block, giq);
    }
    GW_LAUNCHED(P->ctx);
  }
  if (!iq_on_device)
    GW_CUDA(cudaMemcpyAsync(g_iq, giq, niq * sizeof(double), cudaMemcpyDeviceToHost, st));
  GW_CUDA(cudaStreamSynchronize(st));
  return gw::check_device_error(P->ctx, "detector backward");
}

extern "C" int gw_detector_debug_indices(gw_detector_plan *P, int32_t orient,
                                         int64_t *flat_idx) {
  if (!P || !flat_idx) return gw::fail(GW_ERR_ARG, "gw_detector_debug_indices: null argument");
  if (orient < 0 || orient >= P->n_orient)
    return gw::fail(GW_ERR_ARG, "gw_detector_debug_indices: orientation out of range");
  const int npx = P->p.n_h * P->p.n_v;
  int64_t *d = nullptr;
  GW_CUDA(gw::dev_malloc((void **)&d, npx * sizeof(int64_t)));
  DetArgs a = det_args(P);
  if (P->p.exact)
    k_det_debug<<<(npx + 255) / 256, 256, 0, P->ctx->stream>>>(a, orient, d);
  else
    k_det_debug_fast<<<(npx + 255) / 256, 256, 0, P->ctx->stream>>>(a, P->d_ot, orient, d);
  P->ctx->launches++;
  cudaError_t e = cudaMemcpyAsync(flat_idx, d, npx * sizeof(int64_t),
                                  cudaMemcpyDeviceToHost, P->ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(P->ctx->stream);
  gw::dev_free(d);
  if (e != cudaSuccess) return gw::cuda_fail(e, "detector debug", __FILE__, __LINE__);
  return GW_OK;
}

extern "C" int gw_detector(gw_ctx *ctx, const gw_detector_params *p,
                           const double *iq, const double *h_axis,
                           const double *v_axis, const double *init_R,
                           int32_t n_init, const int32_t *n_rot,
                           const double *rot_R, const double *weights,
                           int32_t n_orient, double *out) {
  gw_detector_plan *P = nullptr;
  GW_TRY(gw_detector_plan_create(ctx, p, h_axis, v_axis, init_R, n_init, n_rot,
                                 rot_R, weights, n_orient, &P));
  int st = gw_detector_set_iq(P, iq, 0);
  if (st == GW_OK) st = gw_detector_execute(P);
  if (st == GW_OK) st = gw_detector_get(P, out, 0);
  gw_detector_plan_destroy(P);
  return st;
}

// ======================================================================
// Allocation-free detector entry point (no counterpart in the reference).
//
// Some callers cannot allocate device memory at the moment they need a
// detector image: an acquisition or fitting loop that reserved its whole
// GPU memory budget up front (a framework's caching allocator owns it, or a
// real-time pipeline must not pay cudaMalloc/cudaFree, which can block on
// other streams' work or fail under memory pressure mid-run).
// gw_detector_noalloc takes every input and the output as caller-owned
// device pointers and keeps its only scratch -- the float64 per-pixel sum
// over orientations -- in the fixed array below, so it calls no cudaMalloc,
// cudaFree or allocating library routine.
//
// The array is a module-level __device__ variable: every GPU that loads this
// library holds its 8 MiB until the process exits.  It is shared by all
// calls on that GPU and keeps the previous call's contents; the kernel writes
// every pixel it later reads, so nothing has to be cleared.  Calls whose work
// overlaps on the GPU (different streams, or threads issuing concurrently)
// race on it and must be serialised by the caller.
constexpr int kNoAllocMaxPixels = 1 << 20;  // 1024 x 1024 pixels
static __device__ __align__(256) double g_noalloc_sum[kNoAllocMaxPixels];

namespace {

// k_detector with the per-orientation rotation offsets accumulated on the
// fly from n_rot (the caller passes only counts), writing into `sum`.
__global__ void k_detector_noalloc(DetArgs a, const int *n_rot, double *sum) {
  const int pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= a.nh * a.nv) return;
  const int i = pix / a.nh, j = pix % a.nh;
  double x0, y0, z0;
  base_point(a, i, j, x0, y0, z0);
  double acc = 0.0;
  float s = 0.f, c = 0.f;
  int start = 0;
  for (int o = 0; o < a.n_orient; ++o) {
    // counts come from caller memory the host cannot check: clamp them to
    // the documented 0..3, so that `start` only moves forward by at most 3
    const int n = min(max(n_rot[o], 0), 3);
    double x = x0, y = y0, z = z0;
    for (int k = 0; k < n; ++k) rotate(a.rot_R + 9 * (start + k), x, y, z);
    start += n;
    const int ix = clip_idx(x, a.qmin_x, a.dq, a.inv_dq, a.nx);
    const int iy = clip_idx(y, a.qmin_y, a.dq, a.inv_dq, a.ny);
    const int iz = clip_idx(z, a.qmin_z, a.dq, a.inv_dq, a.nz);
    const float v = __ldg(a.iq + ((int64_t)iy * a.nx + ix) * a.nz + iz);
    if (!a.kahan) {
      acc = fma((double)v, a.w[o], acc);
    } else {
      const float yv = v * (float)a.w[o] - c;
      const float t = s + yv;
      c = (t - s) - yv;
      s = t;
    }
  }
  sum[pix] = a.kahan ? (double)s - (double)c : acc;
}

// Device address of g_noalloc_sum, looked up once per device.  In host code
// the symbol names a host-side shadow, not device memory, so it must never
// be passed to a kernel directly.
std::mutex g_noalloc_mu;
double *g_noalloc_ptr[128] = {};

int noalloc_scratch(int device, double **out) {
  if (device < 0 || device >= 128)
    return gw::fail(GW_ERR_ARG, "gw_detector_noalloc: device index out of range");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[device]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_sum);
    if (e != cudaSuccess)
      return gw::cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_sum)", __FILE__,
                           __LINE__);
    g_noalloc_ptr[device] = static_cast<double *>(p);
  }
  *out = g_noalloc_ptr[device];
  return GW_OK;
}

}  // namespace

extern "C" int gw_detector_noalloc(const gw_detector_params *p,
                                   const float *iq32, const double *h_axis,
                                   const double *v_axis, const double *init_R,
                                   int32_t n_init, const int32_t *n_rot,
                                   const double *rot_R, const double *weights,
                                   int32_t n_orient, double *out,
                                   void *stream) {
  if (!p || !iq32 || !h_axis || !v_axis || !n_rot || !weights || !out)
    return gw::fail(GW_ERR_ARG, "gw_detector_noalloc: null argument");
  if (n_init < 0 || n_init > 3 || (n_init > 0 && !init_R))
    return gw::fail(GW_ERR_ARG, "gw_detector_noalloc: n_init must be 0..3 with init_R given");
  if (p->n_h < 1 || p->n_v < 1 || n_orient < 1 || p->iq_shape[0] < 1 ||
      p->iq_shape[1] < 1 || p->iq_shape[2] < 1 || !(p->dq > 0))
    return gw::fail(GW_ERR_ARG, "gw_detector_noalloc: invalid sizes");
  if ((int64_t)p->n_h * p->n_v > kNoAllocMaxPixels)
    return gw::fail(GW_ERR_ARG,
                    "gw_detector_noalloc: detector has " +
                        std::to_string((int64_t)p->n_h * p->n_v) +
                        " pixels; the allocation-free entry point is limited "
                        "to 1048576 (1024 x 1024). Use gw_detector_plan_create "
                        "for larger images.");
  int device = 0;
  GW_CUDA(cudaGetDevice(&device));
  double *sum = nullptr;
  GW_TRY(noalloc_scratch(device, &sum));
  DetArgs a{};
  a.nh = p->n_h; a.nv = p->n_v;
  a.ny = p->iq_shape[0]; a.nx = p->iq_shape[1]; a.nz = p->iq_shape[2];
  a.qmin_x = p->qmin_x; a.qmin_y = p->qmin_y; a.qmin_z = p->qmin_z;
  a.dq = p->dq; a.inv_dq = 1.0 / p->dq;
  a.h = h_axis; a.v = v_axis; a.init_R = init_R; a.n_init = n_init;
  a.rot_start = nullptr; a.rot_n = nullptr; a.rot_R = rot_R; a.w = weights;
  a.n_orient = n_orient; a.iq = iq32;
  a.sy = (int64_t)a.nx * a.nz; a.sx = a.nz; a.sz = 1;
  a.kahan = p->accum == GW_ACCUM_KAHAN32;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int npx = p->n_h * p->n_v;
  k_detector_noalloc<<<(npx + 127) / 128, 128, 0, st>>>(a, n_rot, sum);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return gw::cuda_fail(e, "k_detector_noalloc launch", __FILE__, __LINE__);
  k_det_epilogue<<<(npx + 255) / 256, 256, 0, st>>>(sum, p->n_v, p->n_h,
                                                    p->mirror, out);
  e = cudaGetLastError();
  if (e != cudaSuccess) return gw::cuda_fail(e, "k_det_epilogue launch", __FILE__, __LINE__);
  return GW_OK;
}
