// SO(3) correlation grid with top-k for oversampling 2 (n = 4 L0 points per axis) on sm_100a.
//
// Reference behaviour restated here: src/matcha/core/SOFFT.py:30-124, src/matcha/core/Matcha.py:27-58,
// :207-236.  With F_j[m'][m] = sum_{l < L0} d^l_{m'm}(beta_j) sigma_{l m' m}, P = 2 L0 - 1:
//   G_j[m'][g] = sum_m F_j[m'][m] e^{2 pi i g m / n}
//   f_j[a][g]  = Re sum_{m'} G_j[m'][g] e^{2 pi i a m' / n} / n^2
//
// The work is FP32 multiply-adds on tiny matrices, so what bounds a straightforward kernel is shared
// memory (an operand or two read per multiply-add) and, for small batches, that one CTA walks all
// n beta values.  Here a thread owns a column (j, g): its P values of G stay in registers from the
// first transform to the second, and the other operand of either (a row of F, a row of the
// twiddle matrix) is the same for the whole warp, so one broadcast 16-byte load feeds twelve or
// six multiply-adds.  A CTA takes 256 / n beta values at a time, and a cluster of up to eight CTAs
// shares a subtomogram's (cluster_size).  Every sum runs in the order of the general kernel in
// search.cu with the same roundings (re_mac, im_mac): near beta = 0 or pi whole diagonals of the grid
// tie but for rounding, and the choice among them must not depend on the path.
//
// Top-k: f goes to shared memory, each thread keeps its column's maximum, and a warp takes out
// its best value while that beats the CTA's C-th best so far; the column that gave it is searched
// again by the whole warp.  One warp merges the warps' lists, and rank 0 the cluster's.  The order
// (value, then smaller index) is total, so the result does not depend on the split.
//
// L0 = 8 (n = 32), 1000 subtomograms: 193 us, before 421 us.  L0 = 16 (n = 64), 64: 239 us,
// before 1207 us; L0 = 8, 16 subtomograms: 22 us, before 119 us.
#include <cooperative_groups.h>
#include <math.h>
#include "common.cuh"
#include "grid.cuh"

namespace {

namespace cg = cooperative_groups;

constexpr int kGT = 256;
constexpr int kWarps = kGT / 32;
constexpr int kCmax = 32;
constexpr int kNone = 0x7fffffff;

// Sizes of one instantiation, in bytes and elements.
template <int L0>
struct Shape {
  static constexpr int n = 4 * L0, P = 2 * L0 - 1, PR = P + 1;
  static constexpr int JB = kGT / n;          // beta values of a pass
  static constexpr int FS = PR * 2 + 4;       // floats of F[.][c]: PR rows (re, im) and 16 bytes
  static constexpr int VS = kGT + 1;          // floats of a row of values
  static constexpr size_t f_bytes = (size_t)JB * P * FS * 4, v_bytes = (size_t)n * VS * 4;
  static constexpr size_t region = ((f_bytes > v_bytes ? f_bytes : v_bytes) + 15) / 16 * 16;
  static constexpr size_t tw_bytes = (size_t)n * PR * 8;
  static constexpr size_t smem = region + 2 * tw_bytes;
};

struct Best {
  float v;
  int i;
};

// v1 before v2 in the kept order
__device__ __forceinline__ bool before(float v1, int i1, float v2, int i2) { return v1 > v2 || (v1 == v2 && i1 < i2); }

// Order-preserving key of a value (zeros of both signs equal); 0 for an empty entry.
__device__ __forceinline__ uint32_t key_of(Best b) {
  if (b.i == kNone) return 0u;
  const uint32_t u = __float_as_uint(b.v + 0.f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// The first of the warp's entries in the kept order, and the lane that holds it.
__device__ __forceinline__ Best warp_best(Best b, int* lane) {
  const uint32_t k = key_of(b), top = __reduce_max_sync(0xffffffffu, k);
  const int i = __reduce_min_sync(0xffffffffu, k == top ? b.i : kNone);
  const uint32_t who = __ballot_sync(0xffffffffu, k == top && b.i == i);
  *lane = __ffs((int)who) - 1;
  Best r;
  r.v = __shfl_sync(0xffffffffu, b.v, *lane);
  r.i = top ? i : kNone;
  return r;
}

template <int L0>
__global__ void __launch_bounds__(kGT, L0 <= 8 ? 4 : 2)
so3_grid_columns_kernel(const float2* __restrict__ sigma, int64_t stride, const float* __restrict__ dtab, int C,
                        float* __restrict__ alpha, float* __restrict__ beta, float* __restrict__ gamma,
                        float* __restrict__ grid_out) {
  using S = Shape<L0>;
  constexpr int n = S::n, P = S::P, PR = S::PR, JB = S::JB;
  const int nk = mtb_dsize(L0 - 1);
  extern __shared__ __align__(16) unsigned char smem[];
  float* sF = reinterpret_cast<float*>(smem);                      // [jb][c][r] (re, im)
  float* sV = sF;                                                  // then [a][column] values
  float2* tw = reinterpret_cast<float2*>(smem + S::region);        // [g][c], c < PR: e^{2 pi i g (c - L0 + 1) / n}
  float2* twt = tw + n * PR;                                       // [c][g]
  __shared__ Best lists[kWarps + 1][kCmax];  // of each warp, and (last) of this CTA so far
  __shared__ Best merged[kCmax];
  __shared__ float2 unit[n];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), parts = (int)cluster.num_blocks(), b = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float2* sig = sigma + (int64_t)b * stride;
  if (tid < n) {
    double sn, cs;
    sincospi(2.0 * tid / n, &sn, &cs);
    unit[tid] = make_float2((float)cs, (float)sn);
  }
  for (int c = tid; c < kCmax; c += kGT) lists[kWarps][c] = Best{-INFINITY, kNone};
  __syncthreads();
  for (int q = tid; q < n * PR; q += kGT) {
    const int g = q / PR, c = q - g * PR;
    int k = (g * (c - (L0 - 1))) % n;
    if (k < 0) k += n;
    const float2 t = c < P ? unit[k] : make_float2(0.f, 0.f);
    tw[q] = t;
    twt[c * n + g] = t;
  }
  const float inv_n2 = 1.f / (float)(n * n);
  const int g = tid % n, jb = tid / n;  // this thread's column of a pass
  const int npass = (n + JB - 1) / JB;
  for (int pass = rank; pass < npass; pass += parts) {
    const int j0 = pass * JB;
    __syncthreads();  // the twiddles are there; the last pass's values and lists are done with
    // F of the pass, one (m', m) of all its beta values per thread
    for (int q = tid; q < P * P; q += kGT) {
      const int r = q / P, c = q - r * P;
      const int mp = r - (L0 - 1), m = c - (L0 - 1);
      const int l0 = max(abs(mp), abs(m));
      float re[JB], im[JB];
#pragma unroll
      for (int i = 0; i < JB; ++i) re[i] = im[i] = 0.f;
#pragma unroll
      for (int l = 0; l < L0; ++l) {
        if (l >= l0) {
          const int idx = mtb_dsize(l - 1) + (mp + l) * (2 * l + 1) + (m + l);
          const float2 s = __ldg(sig + idx);
#pragma unroll
          for (int i = 0; i < JB; ++i) {
            const float d = j0 + i < n ? __ldg(dtab + (int64_t)(j0 + i) * nk + idx) : 0.f;
            re[i] = fmaf(d, s.x, re[i]);
            im[i] = fmaf(d, s.y, im[i]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < JB; ++i)
        *reinterpret_cast<float2*>(sF + (i * P + c) * S::FS + 2 * r) = make_float2(re[i], im[i]);
    }
    __syncthreads();
    const bool own = tid < JB * n && j0 + jb < n;
    float gr[PR], gi[PR];
#pragma unroll
    for (int r = 0; r < PR; ++r) gr[r] = gi[r] = 0.f;
    if (own) {
#pragma unroll 1
      for (int c = 0; c < P; ++c) {
        const float2 t = twt[c * n + g];
        const float4* f4 = reinterpret_cast<const float4*>(sF + (jb * P + c) * S::FS);
#pragma unroll
        for (int r = 0; r < PR; r += 2) {
          const float4 f = f4[r / 2];  // the pad row's value is never used
          gr[r] = re_mac(gr[r], f.x, f.y, t.x, t.y);
          gi[r] = im_mac(gi[r], f.x, f.y, t.x, t.y);
          if (r + 1 < P) {
            gr[r + 1] = re_mac(gr[r + 1], f.z, f.w, t.x, t.y);
            gi[r + 1] = im_mac(gi[r + 1], f.z, f.w, t.x, t.y);
          }
        }
      }
    }
    __syncthreads();  // F is read: the values may overwrite it
    const int base = (j0 + jb) * n * n + g;  // flat index of (j, a, g): base + a n
    Best cur{-INFINITY, kNone};
    if (own) {
      float* out = grid_out ? grid_out + (int64_t)b * n * n * n + base : nullptr;
#pragma unroll 1
      for (int a = 0; a < n; a += 4) {
        float re[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int r = 0; r < PR; r += 2) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 t = *reinterpret_cast<const float4*>(tw + (a + i) * PR + r);
            re[i] = re_mac(re[i], gr[r], gi[r], t.x, t.y);
            if (r + 1 < P) re[i] = re_mac(re[i], gr[r + 1], gi[r + 1], t.z, t.w);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float v = re[i] * inv_n2;
          sV[(a + i) * S::VS + tid] = v;
          if (out) out[(a + i) * n] = v;
          if (v > cur.v || (cur.i == kNone && v == cur.v)) cur = Best{v, base + (a + i) * n};
        }
      }
    }
    __syncwarp();
    // this warp's values that beat the C-th best so far
    const Best last = lists[kWarps][C - 1];
    int cnt = 0;
    for (; cnt < C; ++cnt) {
      int who;
      const Best t = warp_best(cur, &who);
      if (t.i == kNone || !before(t.v, t.i, last.v, last.i)) break;
      if (lane == 0) lists[warp][cnt] = t;
      // the next value of the column that gave it
      const int col = warp * 32 + who, first = (j0 + col / n) * n * n + col % n;
      Best nx{-INFINITY, kNone};
      for (int a = lane; a < n; a += 32) {
        const float v = sV[a * S::VS + col];
        const int i = first + a * n;
        if (before(t.v, t.i, v, i) && before(v, i, nx.v, nx.i)) nx = Best{v, i};
      }
      int dummy;
      nx = warp_best(nx, &dummy);
      if (lane == who) cur = nx;
    }
    for (int c = cnt + lane; c < C; c += 32) lists[warp][c] = Best{-INFINITY, kNone};
    __syncthreads();
    if (warp == 0) {
      // merge the sorted lists: lane q holds the head of list q
      int at = 0;
      for (int c = 0; c < C; ++c) {
        const Best h = lane <= kWarps && at < C ? lists[lane][at] : Best{-INFINITY, kNone};
        int who;
        const Best t = warp_best(h, &who);
        if (lane == 0) merged[c] = t;
        if (lane == who) ++at;
      }
      __syncwarp();
      for (int c = lane; c < C; c += 32) lists[kWarps][c] = merged[c];
    }
  }
  cluster.sync();
  if (rank == 0 && warp == 0) {
    const float bstep = (float)(M_PI / (double)(n - 1));
    const float astep = (float)(2.0 * M_PI / (double)n);
    int at = 0;
    for (int c = 0; c < C; ++c) {
      Best h{-INFINITY, kNone};
      if (lane < parts && at < C) h = cluster.map_shared_rank(&lists[kWarps][0], lane)[at];
      int who;
      const Best t = warp_best(h, &who);
      if (lane == who) ++at;
      if (lane == 0) {
        // fewer than C comparable values (not-a-number): the first points of the grid
        const int i = t.i == kNone ? c : t.i;
        const int o = b * C + c;
        beta[o] = (float)(i / (n * n)) * bstep;
        alpha[o] = (float)((i / n) % n) * astep;
        gamma[o] = (float)(i % n) * astep;
      }
    }
  }
  cluster.sync();  // no CTA leaves while its list is read
}

template <int L0>
int launch(const float2* sigma, int64_t stride, int B, const float* dtab, int C, float* a, float* b, float* g,
           float* grid, cudaStream_t st) {
  using S = Shape<L0>;
  static_assert(S::smem + (kWarps + 2) * kCmax * sizeof(Best) + S::n * sizeof(float2) <= kSmemOptIn, "shared memory");
  MTB_CUDA_TRY(cudaFuncSetAttribute(so3_grid_columns_kernel<L0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)S::smem));
  constexpr int npass = (S::n + S::JB - 1) / S::JB;
  int parts = cluster_size(B, 8);
  while (parts > npass) parts /= 2;
  mtb_prof_begin(st);
  for (int b0 = 0; b0 < B; b0 += 65535) {  // the grid's y limit
    const int nb = B - b0 < 65535 ? B - b0 : 65535;
    const int64_t o = (int64_t)b0 * C;
    MTB_CUDA_TRY(launch_clusters(so3_grid_columns_kernel<L0>, dim3(parts, nb), kGT, S::smem, parts, st,
                                 sigma + b0 * stride, stride, dtab, C, a + o, b + o, g + o,
                                 grid ? grid + (int64_t)b0 * S::n * S::n * S::n : nullptr));
  }
  mtb_prof_end(st, "so3_grid_columns_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}

}  // namespace

bool grid_columns_cover(int L0, int K) { return K == 2 && L0 >= 3 && L0 <= 16; }

int grid_columns_launch(const float2* sigma, int64_t stride, int B, const float* dtab, int L0, int C, float* a,
                        float* b, float* g, float* grid, cudaStream_t st) {
  switch (L0) {
    case 3: return launch<3>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 4: return launch<4>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 5: return launch<5>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 6: return launch<6>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 7: return launch<7>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 8: return launch<8>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 9: return launch<9>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 10: return launch<10>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 11: return launch<11>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 12: return launch<12>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 13: return launch<13>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 14: return launch<14>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 15: return launch<15>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    case 16: return launch<16>(sigma, stride, B, dtab, C, a, b, g, grid, st);
    default: MTB_ARG_CHECK(false, "L0 must be in [3, 16]");
  }
}
