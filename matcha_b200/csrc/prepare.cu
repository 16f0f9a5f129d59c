// Subtomogram preparation before the ball expansion, in every alternation: the patch at the
// current shift, normalised inside a spherical mask and masked, then rotated into the
// current orientation estimate.
//
// Reference behaviour restated here (paths inside swing-research/Matcha):
//   BatchProcessor._extract_rotated_batch   src/matcha/align_subtomograms.py:240-252
//   extract_subtomogram_patch_batch         src/matcha/utils/io_utils.py:113-178 (normalize=True)
//   normalise / mean / std                  src/matcha/utils/volume_ops.py:17-35
//   spherical mask (distance < radius)      src/matcha/utils/volume_ops.py:6-14, setup_utils.py:274-281
//   rotate_volumes_in_batches               src/matcha/utils/volume_rotation.py:49-125
//
// Both resamplings are grid_sample(mode='bilinear', align_corners=True, zero padding) in 3-D:
// corner weights (x part)(y part)(z part), corners outside the box skipped.
//
// extract_staged_kernel: CTA = (one or two output planes z, subtomogram b).  The sample coordinate
// of each axis depends on that axis alone (voxel + shift through the reference's normalised-grid
// round trip 2 g / (N - 1) - 1, then ((u + 1) / 2) (N - 1)).  The CTA copies the rows its masked
// voxels read from planes iz0 and iz0 + 1 with 16-byte loads and stores their z interpolation
// in shared memory; a warp walks rows next to each other, two columns to a lane, and interpolates
// each source row in x once for the two output rows that it lies between, then in y.  It writes
// the pair (p(x), p(x + 1)), the second value from the next lane, wherever one of the two lies in
// the mask (nothing else reads the patch), so that the rotation reads both x corners of a row in
// one 8-byte load, and adds the masked sum and sum of squares to the subtomogram's FP64
// statistics.  Bound by instruction issue; 1000 of 64^3 647 -> 502 us against 300 for the bytes
// (before: a column to a thread, both rows and both values of a pair interpolated for each voxel).
// extract_kernel does the same voxel by voxel from global memory for boxes whose plane does not
// fit in shared memory.
//
// rotate_kernel: CTA = (one or four output planes z, subtomogram b), a warp = a brick of 32 voxels.
// The sample point of output voxel v is R (v - c) + c (c = N / 2, the centre of the odd-padded
// linspace(-1, 1) grid), so |s - c| = |v - c|: voxels farther than radius + 2 from c read only
// masked-out corners and are written as zero without loads, voxels nearer than radius - 1.74
// read only corners inside the mask (four pair loads), and only the shell between tests the
// mask per corner.  Values are normalised as they are read: (p - mean) / std inside the mask,
// 0 outside.  The gathers are bound by the L1 data stage, which takes about eight passes for a
// warp-wide corner read: the pair layout halves the number of reads, and the brick's shape follows
// the rotation, so that few source rows lie under it.  1000 of 64^3 1242 -> 959 us (before: fixed
// 8 x 4 x 1 bricks, and a warp with shell voxels went both ways, corner by corner).
#include <limits.h>
#include <math.h>
#include "common.cuh"

namespace {

constexpr int kPT = 256;

struct Axis {
  int j0, j1;    // the two corner indices, clamped into [0, N) so that every read stays in the box
  float w0, w1;  // their weights
  bool v0, v1;   // whether the unclamped corners lie in [0, N); a corner outside reads 0
};

// One axis of the patch sampling: voxel g shifted by s, through the reference's round trip.
__device__ __forceinline__ Axis patch_axis(int g, float s, int N) {
  const float size = (float)(N - 1);
  const float n = 2.f * ((float)g + s) / size - 1.f;
  float u = ((n + 1.f) / 2.f) * size;
  u = fminf(fmaxf(u, -2.f), (float)N + 1.f);  // beyond this every corner is outside the box
  const float f = floorf(u);
  const int i0 = (int)f;
  Axis a;
  a.w1 = u - f;
  a.w0 = (f + 1.f) - u;
  a.v0 = i0 >= 0 && i0 < N;
  a.v1 = i0 + 1 >= 0 && i0 + 1 < N;
  a.j0 = min(max(i0, 0), N - 1);
  a.j1 = min(max(i0 + 1, 0), N - 1);
  return a;
}

// Adds the block's sums of d1 and d2 to to[0] and to[1] (red: two entries per warp).
__device__ __forceinline__ void block_add(double d1, double d2, double* to, double (&red)[2][kPT / 32]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    d1 += __shfl_xor_sync(0xffffffffu, d1, o);
    d2 += __shfl_xor_sync(0xffffffffu, d2, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    red[0][warp] = d1;
    red[1][warp] = d2;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double s = 0.0;
    for (int w = 0; w < kPT / 32; ++w) s += red[threadIdx.x][w];
    atomicAdd(&to[threadIdx.x], s);
  }
}

// Trilinear value of the patch at one voxel from the eight corners read by at(plane, row, col)
// (plane 0 / 1 = iz0 / iz0 + 1), corners outside the box reading 0.
template <class F>
__device__ __forceinline__ float patch_value(const Axis& ax, const Axis& ay, const Axis& az, F&& at) {
  const bool q00 = az.v0 && ay.v0, q01 = az.v0 && ay.v1, q10 = az.v1 && ay.v0, q11 = az.v1 && ay.v1;
  const float c000 = (q00 && ax.v0) ? at(0, ay.j0, ax.j0) : 0.f, c001 = (q00 && ax.v1) ? at(0, ay.j0, ax.j1) : 0.f;
  const float c010 = (q01 && ax.v0) ? at(0, ay.j1, ax.j0) : 0.f, c011 = (q01 && ax.v1) ? at(0, ay.j1, ax.j1) : 0.f;
  const float c100 = (q10 && ax.v0) ? at(1, ay.j0, ax.j0) : 0.f, c101 = (q10 && ax.v1) ? at(1, ay.j0, ax.j1) : 0.f;
  const float c110 = (q11 && ax.v0) ? at(1, ay.j1, ax.j0) : 0.f, c111 = (q11 && ax.v1) ? at(1, ay.j1, ax.j1) : 0.f;
  const float w00 = ax.w0 * ay.w0, w01 = ax.w1 * ay.w0, w10 = ax.w0 * ay.w1, w11 = ax.w1 * ay.w1;
  float p = c000 * (w00 * az.w0);
  p = fmaf(c001, w01 * az.w0, p);
  p = fmaf(c010, w10 * az.w0, p);
  p = fmaf(c011, w11 * az.w0, p);
  p = fmaf(c100, w00 * az.w1, p);
  p = fmaf(c101, w01 * az.w1, p);
  p = fmaf(c110, w10 * az.w1, p);
  p = fmaf(c111, w11 * az.w1, p);
  return p;
}

// Boxes whose plane does not fit in shared memory: a warp walks rows, 31 columns at a time (the 32nd
// lane's value is only the last pair's second), the eight corners of a voxel from global memory.  Bound
// by the latency of those reads; 4 of 240^3 487 us with both values of a pair read by its thread, 573
// with the pairs before the mask's first column beside them, 290 so.
__global__ void __launch_bounds__(kPT) extract_kernel(const float* __restrict__ vol, int N,
                                                      const float* __restrict__ shift_xyz, int thresh,
                                                      float2* __restrict__ pairs, double* __restrict__ stats) {
  __shared__ double red[2][kPT / 32];
  extern __shared__ Axis s_y[];  // the y axis of every row (N entries)
  const int z = blockIdx.x, b = blockIdx.y;
  const int64_t NN = (int64_t)N * N;
  const float* v = vol + (int64_t)b * NN * N;
  float2* out = pairs + ((int64_t)b * N + z) * NN;
  const float sx = shift_xyz[3 * b], sy = shift_xyz[3 * b + 1], sz = shift_xyz[3 * b + 2];
  for (int y = threadIdx.x; y < N; y += kPT) s_y[y] = patch_axis(y, sy, N);
  __syncthreads();
  const Axis az = patch_axis(z, sz, N);
  const float* pl[2] = {v + (int64_t)az.j0 * NN, v + (int64_t)az.j1 * NN};
  const int c = N / 2, rem = thresh - (z - c) * (z - c);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows = (N + kPT / 32 - 1) / (kPT / 32), y0 = warp * rows, y1 = min(y0 + rows, N);
  float s1 = 0.f, s2 = 0.f;
  for (int x0 = 0; x0 < N; x0 += 31) {
    const bool last = x0 + 32 >= N, own = lane < 31 || last;
    const int x = x0 + lane;
    const Axis ax = patch_axis(x, sx, N);
    const int d0 = x < N ? (x - c) * (x - c) : 1 << 24, d1 = x + 1 < N ? (x + 1 - c) * (x + 1 - c) : 1 << 24;
    for (int y = y0; y < y1; ++y) {
      const int ry = rem - (y - c) * (y - c);
      const bool in0 = d0 < ry, write = min(d0, d1) < ry;
      if (!__any_sync(0xffffffffu, write)) continue;
      float p = 0.f;
      if (write) {
        const Axis ay = s_y[y];
        p = patch_value(ax, ay, az, [&](int k, int row, int col) { return __ldg(pl[k] + (int64_t)row * N + col); });
      }
      const float p1 = __shfl_down_sync(0xffffffffu, p, 1);
      if (own && write) out[(int64_t)y * N + x] = make_float2(p, x + 1 < N ? p1 : 0.f);
      if (own && in0) {
        s1 += p;
        s2 = fmaf(p, p, s2);
      }
    }
    if (last) break;
  }
  block_add(s1, s2, stats + 2 * b, red);
}

// A row of the y axis in shared memory: its weights, and the offsets of its two source rows in the
// staged plane (the complement of the clamped row's when the corner lies outside the box).
struct RowAxis {
  float w0, w1;
  int o0, o1;
};

// Shared memory: the y axis (N entries) and one plane (N^2 floats, the z interpolation of planes
// iz0 and iz0 + 1).
template <int NT>
__global__ void __launch_bounds__(kPT, NT ? 5 : 4) extract_staged_kernel(const float* __restrict__ vol, int n_rt, int planes /* 1 or 2 */,
                                                                const float* __restrict__ shift_xyz, int thresh,
                                                                float2* __restrict__ pairs,
                                                                double* __restrict__ stats) {
  const int N = NT ? NT : n_rt;
  __shared__ double red[2][kPT / 32];
  extern __shared__ float4 smem4[];
  RowAxis* s_y = reinterpret_cast<RowAxis*>(smem4);
  float* s_t = reinterpret_cast<float*>(smem4 + N);
  const int b = blockIdx.y, c = N / 2;
  const int64_t NN = (int64_t)N * N;
  const float* v = vol + (int64_t)b * NN * N;
  const float sx = shift_xyz[3 * b], sy = shift_xyz[3 * b + 1], sz = shift_xyz[3 * b + 2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // FP32 sums of the plane in hand and of the one before: they meet in FP64, so that one or two planes
  // a CTA make no difference
  float s1 = 0.f, s2 = 0.f, p1 = 0.f, p2 = 0.f;
  for (int y = threadIdx.x; y < N; y += kPT) {
    const Axis a = patch_axis(y, sy, N);
    s_y[y] = RowAxis{a.w0, a.w1, a.v0 ? a.j0 * N : ~(a.j0 * N), a.v1 ? a.j1 * N : ~(a.j1 * N)};
  }
  const int z_end = min((int)(blockIdx.x + 1) * planes, N);
  for (int z = blockIdx.x * planes; z < z_end; ++z) {
    const int dz2 = (z - c) * (z - c);
    if (dz2 >= thresh) continue;  // no voxel of this plane lies in the mask
    const int rem = thresh - dz2;  // the plane's masked voxels: (y - c)^2 + (x - c)^2 < rem
    int ky = (int)sqrtf((float)rem);
    while (ky > 0 && ky * ky >= rem) --ky;
    while ((ky + 1) * (ky + 1) < rem) ++ky;
    const int ylo = c - ky > 0 ? c - ky : 0, yhi = c + ky < N - 1 ? c + ky : N - 1;
    float2* out = pairs + ((int64_t)b * N + z) * NN;
    const Axis az = patch_axis(z, sz, N);
    __syncthreads();  // the y axis is there, and the last plane is read
    {
      // from the first row's lower to the last row's upper corner (non-decreasing in y); the other
      // rows are never used
      const int lo = s_y[ylo].o0, hi = s_y[yhi].o1;
      const int from = lo < 0 ? ~lo : lo, n = (hi < 0 ? ~hi : hi) + N - from;
      const float* src0 = v + (int64_t)az.j0 * NN + from;
      const float* src1 = v + (int64_t)az.j1 * NN + from;
      float* dst = s_t + from;
      if ((N & 3) == 0 && ((reinterpret_cast<uintptr_t>(src0) | reinterpret_cast<uintptr_t>(src1)) & 15) == 0) {
        const float4* a4 = reinterpret_cast<const float4*>(src0);
        const float4* b4 = reinterpret_cast<const float4*>(src1);
        float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll 2
        for (int i = threadIdx.x; i < n / 4; i += kPT) {
          const float4 a = az.v0 ? __ldg(a4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float4 e = az.v1 ? __ldg(b4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
          d4[i] = make_float4(fmaf(e.x, az.w1, a.x * az.w0), fmaf(e.y, az.w1, a.y * az.w0),
                              fmaf(e.z, az.w1, a.z * az.w0), fmaf(e.w, az.w1, a.w * az.w0));
        }
      } else {
        for (int i = threadIdx.x; i < n; i += kPT) {
          const float a = az.v0 ? __ldg(src0 + i) : 0.f, e = az.v1 ? __ldg(src1 + i) : 0.f;
          dst[i] = fmaf(e, az.w1, a * az.w0);
        }
      }
    }
    __syncthreads();
    const int rows = (yhi - ylo + kPT / 32) / (kPT / 32);  // of a warp, next to each other
    const int y0 = ylo + warp * rows, y1 = y0 + rows < yhi + 1 ? y0 + rows : yhi + 1;
    p1 = s1;
    p2 = s2;
    s1 = s2 = 0.f;
    // 64 columns at a time, two of a lane; the last one's pair is the next step's first
    for (int x0 = 0; x0 < N; x0 += 63) {
      const bool last = x0 + 64 >= N, two = x0 + 32 < N;
      const int xa = x0 + lane, xb = xa + 32;
      const Axis ax = patch_axis(xa, sx, N), bx = patch_axis(xb, sx, N);
      // squared distances of the two columns from the centre, and the nearer of each pair's
      auto near2 = [&](int x) { return x < N ? (x - c) * (x - c) : 1 << 24; };
      const bool own = lane < 31 || last;
      const int da2 = near2(xa), db2 = own ? near2(xb) : 1 << 24;
      const int na2 = xa < N ? min(da2, near2(xa + 1)) : 1 << 24;
      const int nb2 = own && xb < N ? min(db2, near2(xb + 1)) : 1 << 24;
      auto row = [&](int o) {  // the x interpolation of the source row at offset o
        const float* t = s_t + o;
        const float lo = ax.v0 ? t[ax.j0] : 0.f, hi = ax.v1 ? t[ax.j1] : 0.f;
        float2 r = make_float2(fmaf(hi, ax.w1, lo * ax.w0), 0.f);
        if (two) {
          const float lb = bx.v0 ? t[bx.j0] : 0.f, hb = bx.v1 ? t[bx.j1] : 0.f;
          r.y = fmaf(hb, bx.w1, lb * bx.w0);
        }
        return r;
      };
      int at = -1;  // the source row that r1 holds
      float2 r1 = make_float2(0.f, 0.f);
      for (int y = y0; y < y1; ++y) {
        const RowAxis ay = s_y[y];
        float2 r0 = r1;
        if (ay.o0 != at) r0 = ay.o0 >= 0 ? row(ay.o0) : make_float2(0.f, 0.f);
        r1 = ay.o1 >= 0 ? row(ay.o1) : make_float2(0.f, 0.f);
        at = ay.o1;
        const float pa = fmaf(r1.x, ay.w1, r0.x * ay.w0), pb = fmaf(r1.y, ay.w1, r0.y * ay.w0);
        // the values at x + 1; p(N) lies outside the patch: the pair holds 0 there
        const float b0 = __shfl_sync(0xffffffffu, pb, 0);
        float na = __shfl_down_sync(0xffffffffu, pa, 1), nb = __shfl_down_sync(0xffffffffu, pb, 1);
        na = xa + 1 < N ? (lane < 31 ? na : b0) : 0.f;
        nb = xb + 1 < N ? nb : 0.f;
        const int ry = rem - (y - c) * (y - c);
        float2* o = out + (int64_t)y * N + xa;
        if (na2 < ry) o[0] = make_float2(pa, na);
        if (nb2 < ry) o[32] = make_float2(pb, nb);
        const float ma = da2 < ry ? pa : 0.f, mb = db2 < ry ? pb : 0.f;
        s1 += ma + mb;
        s2 = fmaf(ma, ma, fmaf(mb, mb, s2));
      }
      if (last) break;
    }
  }
  block_add((double)p1 + s1, (double)p2 + s2, stats + 2 * b, red);
}

// Rotation.  CTA = (2^lz_max output planes, subtomogram b); a warp takes a brick of 2^lx x 2^ly x
// 2^lz output voxels at a time.
// BOX: the mask reaches outside the box, so a corner inside the mask may still be outside it.
template <int NT, bool BOX>
__global__ void __launch_bounds__(kPT, NT ? (BOX ? 6 : 7) : 5) rotate_kernel(const float2* __restrict__ pairs, int n_rt,
                                                        const double* __restrict__ tracker,
                                                        const double* __restrict__ stats, double inv_count,
                                                        int thresh, int skip2, int inner2, int lz_max,
                                                        float* __restrict__ out) {
  const int N = NT ? NT : n_rt;
  const int b = blockIdx.y;
  const int64_t NN = (int64_t)N * N;
  const float2* p = pairs + (int64_t)b * NN * N;
  float* o = out + (int64_t)b * NN * N;
  // the rotation of the tracker scaled to unit norm, as its Euler angles are
  const double qw = tracker[4 * b], qx = tracker[4 * b + 1], qy = tracker[4 * b + 2], qz = tracker[4 * b + 3];
  const double k = 2.0 / (qw * qw + qx * qx + qy * qy + qz * qz);
  const float R00 = (float)(1 - k * (qy * qy + qz * qz)), R01 = (float)(k * (qx * qy - qw * qz)),
              R02 = (float)(k * (qx * qz + qw * qy));
  const float R10 = (float)(k * (qx * qy + qw * qz)), R11 = (float)(1 - k * (qx * qx + qz * qz)),
              R12 = (float)(k * (qy * qz - qw * qx));
  const float R20 = (float)(k * (qx * qz - qw * qy)), R21 = (float)(k * (qy * qz + qw * qx)),
              R22 = (float)(1 - k * (qx * qx + qy * qy));
  // mean and standard deviation in the mask (mean(p^2) - mean^2, as the reference)
  const double m = stats[2 * b] * inv_count;
  const float mean = (float)m;
  const float inv_sd = (float)(1.0 / sqrt(fmax(stats[2 * b + 1] * inv_count - m * m, 0.0)));
  const int c = N / 2;
  const float half = (N % 2 == 0) ? 0.5f * (float)N : 0.5f * (float)(N - 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // The brick's extents: 8 along x, so that a row's part of the store is a whole sector (bricks of 4
  // or 2 along x as well: 956 against 860 us, at a mask radius of 28.8), and 4 along y and z together.  A corner read touches a
  // line of L1 for about every source row (y, z) under the brick, that is, for its faces seen along
  // the source's x axis, whose components are the R0k.  A warp walks along x, where a brick finds
  // lines of the one before it (with the warps next to each other along x instead 1258 us there).
  int ly = 2, lz = 0;
  constexpr int lx = 3;
  float best = 1e30f;
  for (int j = 0; j <= lz_max; ++j) {
    const float rows = 4.f * fabsf(R00) + (float)(8 << j) * fabsf(R01) + (float)(8 << (2 - j)) * fabsf(R02);
    if (rows < best) {
      best = rows;
      ly = 2 - j;
      lz = j;
    }
  }
  const int vx = lane & ((1 << lx) - 1), vy = (lane >> lx) & ((1 << ly) - 1), vz = lane >> (lx + ly);
  const int nby = (N + (1 << ly) - 1) >> ly, nrow = nby << (lz_max - lz);
  for (int t = warp; t < nrow; t += kPT / 32) {
    const int y = ((t % nby) << ly) + vy, z = (blockIdx.x << lz_max) + ((t / nby) << lz) + vz;
    const int dy = y - c, dz = z - c;
    const float bx = fmaf(R01, (float)dy, fmaf(R02, (float)dz, half)),
                by = fmaf(R11, (float)dy, fmaf(R12, (float)dz, half)),
                bz = fmaf(R21, (float)dy, fmaf(R22, (float)dz, half));
    for (int x0 = 0; x0 < N; x0 += 1 << lx) {
      const int x = x0 + vx, dx = x - c;
      const bool in_box = x < N && y < N && z < N;
      const int r2 = in_box ? dx * dx + dy * dy + dz * dz : INT_MAX;
      const bool near = r2 < skip2;
      float val = 0.f;
      if (__any_sync(0xffffffffu, near)) {
        const float sx = fmaf(R00, (float)dx, bx);
        const float sy = fmaf(R10, (float)dx, by);
        const float sz = fmaf(R20, (float)dx, bz);
        const float fx = floorf(sx), fy = floorf(sy), fz = floorf(sz);
        const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
        const float wx1 = sx - fx, wy1 = sy - fy, wz1 = sz - fz;
        const float wx0 = (fx + 1.f) - sx, wy0 = (fy + 1.f) - sy, wz0 = (fz + 1.f) - sz;
        // 32-bit offsets: N^3 <= 2^27 pairs
        const float2* q = p + (iz * N + iy) * N + ix;
        const int rs = N, ps = N * N;
        float cv[8] = {};
        // a warp with a corner outside the mask or the box takes the second way whole, not both in turn
        const bool in_corners = !BOX || ((unsigned)ix < (unsigned)(N - 1) && (unsigned)iy < (unsigned)(N - 1) &&
                                         (unsigned)iz < (unsigned)(N - 1));
        const bool inner = __all_sync(0xffffffffu, !near || (r2 < inner2 && in_corners));
        if (near && inner) {
          // every corner lies inside the mask, hence inside the box: four pair loads
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float2 e = __ldg(q + (r >> 1) * ps + (r & 1) * rs);
            cv[2 * r] = e.x - mean;
            cv[2 * r + 1] = e.y - mean;
          }
        } else if (near) {
          const int ex0 = ix - c, ey0 = iy - c, ez0 = iz - c;
          const int e02 = ex0 * ex0, e12 = e02 + 2 * ex0 + 1;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int ey = ey0 + (r & 1), ez = ez0 + (r >> 1), left = thresh - (ey * ey + ez * ez);
            bool in0 = e02 < left, in1 = e12 < left;
            const float2* qr = q + (r >> 1) * ps + (r & 1) * rs;
            if (BOX) {
              const bool row = (unsigned)(iy + (r & 1)) < (unsigned)N && (unsigned)(iz + (r >> 1)) < (unsigned)N;
              in0 = in0 && row && (unsigned)ix < (unsigned)N;
              in1 = in1 && row && (unsigned)(ix + 1) < (unsigned)N;
            }
            // a pair is written where either of its values is in the mask; before the box there is
            // none (row's first corner in the mask: BOX, or an odd box with a mask up to its faces)
            float2 e = make_float2(0.f, 0.f);
            if ((BOX || N % 2) && ix < 0) {
              if (in1) e.y = __ldg(reinterpret_cast<const float*>(qr + 1));
            } else if (in0 || in1) {
              e = __ldg(qr);
            }
            cv[2 * r] = in0 ? e.x - mean : 0.f;
            cv[2 * r + 1] = in1 ? e.y - mean : 0.f;
          }
        }
        const float w00 = wx0 * wy0, w01 = wx1 * wy0, w10 = wx0 * wy1, w11 = wx1 * wy1;
        float s = cv[0] * (w00 * wz0);
        s = fmaf(cv[1], w01 * wz0, s);
        s = fmaf(cv[2], w10 * wz0, s);
        s = fmaf(cv[3], w11 * wz0, s);
        s = fmaf(cv[4], w00 * wz1, s);
        s = fmaf(cv[5], w01 * wz1, s);
        s = fmaf(cv[6], w10 * wz1, s);
        s = fmaf(cv[7], w11 * wz1, s);
        val = near ? s * inv_sd : 0.f;
      }
      if (in_box) o[((int64_t)z * N + y) * N + x] = val;
    }
  }
}

template <int NT>
int launch(const float* volumes, int B, int N, const float* shift_xyz, const double* tracker, int thresh, bool box,
           int skip2, int inner2, double inv_count, float2* work, double* stats, float* out, cudaStream_t st) {
  const size_t ext_smem = (size_t)N * N * sizeof(float) + (size_t)N * sizeof(RowAxis);
  const bool staged = ext_smem <= 220 * 1024;  // boxes up to 235; 48 of 128^3: 235 us, voxel by voxel 844
  if (staged && ext_smem > 48 * 1024)
    MTB_CUDA_TRY(cudaFuncSetAttribute(extract_staged_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      220 * 1024));
  // Where four planes a CTA still give 8 CTAs an SM, the prologues are shared by two planes in the
  // extraction (1000 of 64^3: 557 us with one, 502 with two), and bricks of the rotation reach over four
  // planes (1023, 992 and 959 us with one, two and four) or, past 64^3, where the source under four
  // planes outgrows L1, over two (100 of 96^3 413, 412 and 452 us, 300 of 80^3 753, 703 and 746).  Below,
  // a plane a CTA keeps the SMs busy.
  const bool wide = (int64_t)B * ((N + 3) / 4) >= 148 * 8;
  const int planes = wide ? 2 : 1, lz_max = wide ? (N <= 64 ? 2 : 1) : 0;
  mtb_prof_begin(st);
  if (staged)
    extract_staged_kernel<NT><<<dim3((N + planes - 1) / planes, B), kPT, ext_smem, st>>>(
        volumes, N, planes, shift_xyz, thresh, work, stats);
  else
    extract_kernel<<<dim3(N, B), kPT, (size_t)N * sizeof(Axis), st>>>(volumes, N, shift_xyz, thresh, work, stats);
  mtb_prof_end(st, "extract_kernel");
  MTB_LAUNCH_CHECK();
  const dim3 grid((N + (1 << lz_max) - 1) >> lz_max, B);
  mtb_prof_begin(st);
  if (box)
    rotate_kernel<NT, true><<<grid, kPT, 0, st>>>(work, N, tracker, stats, inv_count, thresh, skip2, inner2,
                                                   lz_max, out);
  else
    rotate_kernel<NT, false><<<grid, kPT, 0, st>>>(work, N, tracker, stats, inv_count, thresh, skip2, inner2,
                                                   lz_max, out);
  mtb_prof_end(st, "rotate_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}

}  // namespace

extern "C" int mtb_prepare_subtomos(const float* volumes, int B, int N, const float* shift_xyz, const double* tracker,
                                    float mask_radius, float* work, double* stats, float* out, mtb_stream_t stream) {
  MTB_ARG_CHECK(B >= 0 && N >= 2 && N <= 512, "bad batch or box size");
  if (B == 0) return MTB_OK;
  MTB_ARG_CHECK(volumes && shift_xyz && tracker && work && stats && out, "null pointer");
  MTB_ARG_CHECK((reinterpret_cast<uintptr_t>(work) & 7) == 0, "work must be 8-byte aligned");
  MTB_ARG_CHECK(mask_radius > 0.f && mask_radius < 1024.f, "mask radius must be in (0, 1024)");
  const cudaStream_t st = (cudaStream_t)stream;
  // integer distances squared d2 satisfy d2 < r^2 exactly when d2 < ceil(r^2)
  const double r = (double)mask_radius, r2max = r * r;
  const int thresh = (int)ceil(r2max);
  int64_t count = 0;  // voxels of the mask: per row, the dx with dx^2 < thresh - dz^2 - dy^2
  const int c = N / 2;
  for (int z = 0; z < N; ++z)
    for (int y = 0; y < N; ++y) {
      const int rem = thresh - (z - c) * (z - c) - (y - c) * (y - c);
      if (rem <= 0) continue;
      int k = (int)sqrt((double)rem);
      while (k > 0 && k * k >= rem) --k;
      while ((k + 1) * (k + 1) < rem) ++k;
      const int lo = -k > -c ? -k : -c, hi = k < N - 1 - c ? k : N - 1 - c;
      if (hi >= lo) count += hi - lo + 1;
    }
  MTB_ARG_CHECK(count > 0, "the mask is empty");
  // A rotation keeps |s - c| = |v - c|, and the corners of s lie within sqrt(3) < 1.74 of it: beyond
  // r + 1.74 all corners are outside the mask, within r - 1.74 all are inside.  What is left covers
  // the rounding of s (1e-4 at 512).  The outer limit is r + 2: the shell in between is empty sums over
  // the deviation, zero, but not a number, as the mask is, where a subtomogram has no deviation.
  const int skip2 = (int)ceil((r + 2.0) * (r + 2.0));
  const int inner2 = r > 1.74 ? (int)floor((r - 1.74) * (r - 1.74)) : 0;
  // the mask stays inside the box when every offset d with d^2 < r^2 is at most min(c, N-1-c)
  const int reach = c < N - 1 - c ? c : N - 1 - c;
  const bool box = r2max > (double)(reach + 1) * (double)(reach + 1);
  MTB_CUDA_TRY(cudaMemsetAsync(stats, 0, (size_t)B * 2 * sizeof(double), st));
  const double inv_count = 1.0 / (double)count;
  float2* pairs = reinterpret_cast<float2*>(work);
  if (N == 64)
    return launch<64>(volumes, B, N, shift_xyz, tracker, thresh, box, skip2, inner2, inv_count, pairs, stats, out,
                      st);
  return launch<0>(volumes, B, N, shift_xyz, tracker, thresh, box, skip2, inner2, inv_count, pairs, stats, out, st);
}
