// Backward kernels of the alignment score (the differentiation pattern of the alignment path).
//
// The score of subtomogram b at a rotation R is f_b(R) = Re sum_l sum_{m'm} D^l_{m'm}(R)
// sigma_b[l, m', m] (src/matcha/core/Matcha.py:184, :288), with the reference's convention
// D^l_{m'm}(alpha, beta, gamma) = exp(+i m' alpha) d^l_{m'm}(beta) exp(+i m gamma) and
// sigma_b[l, m', m] = (-1)^(m'+m) sum_k aT[l, -m, k] conj(aV_b[l, -m', k])
// (src/matcha/core/CrossCorrelationMatcher.py:183-212).
//
// score_backward_kernel regenerates D^l(R_b) for l <= L from the angles (FP64 three-term
// recurrences in l per (m', m), the forward pass stores nothing) and, in the same sweep,
//   * grad_sigma_b = w_b conj(D(R_b)): d f / d sigma in PyTorch's convention for a real
//     function of a complex tensor (d/dRe + i d/dIm);
//   * the body-frame gradient g_k = d f_b(R_b exp(t e_k)) / dt at t = 0, k = x, y, z.
//     D(R exp(t e_k)) = D(R) D(exp(t e_k)), so g_k = Re sum D(R) sigma^(k) with
//     sigma^(k)[m', n] = sum_m sigma[m', m] A_k[n, m] and A_k the generator of the
//     representation: A_z = diag(i m); A_y[m+1, m] = -sqrt((l-m)(l+m+1))/2,
//     A_y[m-1, m] = sqrt((l+m)(l-m+1))/2 (the derivative of Edmonds' d^l at beta = 0);
//     A_x[n, m] = i^(m-n) A_y[n, m] (Rx(t) = Rz(-pi/2) Ry(t) Rz(pi/2)).  Unlike the Euler
//     gradient mapped through the z-y-z kinematics, this has no singularity at beta = 0, pi.
//
// sigma_backward_template_kernel: the adjoint of the sigma contraction with respect to the
// template coefficients, grad_aT[l, -m, k] = sum_b sum_m' (-1)^(m'+m) aV_b[l, -m', k]
// grad_sigma_b[l, m', m]; one cluster per degree and 32 columns, summed in a fixed order.
#include <math.h>
#include <cooperative_groups.h>
#include "common.cuh"

namespace {

constexpr int kBT = 256;

__device__ __forceinline__ double2 cmul_d(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ double ipow_d(double x, int n) {
  double r = 1.0;
  while (n) {
    if (n & 1) r *= x;
    x *= x;
    n >>= 1;
  }
  return r;
}

// Shared memory of score_backward_kernel: its tables, in doubles.
size_t score_backward_smem(int L) {
  return ((size_t)2 * (2 * L + 2) + 3 * (2 * L + 1) + 5 * (L + 1)) * sizeof(double);
}

struct LogFactorials {
  double v[257];  // log n!, n <= 2 L <= 256
};

// One cluster per subtomogram, its chains dealt to the CTAs.  FP64 arithmetic and the latency of
// the chains bound it (more CTAs hide more of the latter), so whatever a chain step shares with
// others is tabulated per CTA: sqrt(n) and its reciprocal, of which the roots of the recurrence
//   (l-1) a_l d^l = (2l-1)(l(l-1) cos b - m m') d^{l-1} - l a_{l-1} d^{l-2},
//   a_l = sqrt((l^2-m^2)(l^2-m'^2)),
// and of the generators are products (no root and no division in a step), the log factorials and
// half-angle powers of the chains' first values, the phases.  A thread runs the chain of (m', m),
// m' >= 0, for its mirror image too, d_{-m',-m} = (-1)^{m'-m} d_{m'm}; lanes take consecutive m, so
// that both images are read and written in rows.
// 256 subtomograms at L = 32: 150 us, against 385 us with roots, divisions and log-gammas in
// every chain.
__global__ void __launch_bounds__(kBT)
score_backward_kernel(const float2* __restrict__ sigma, int64_t stride, int L, const float* __restrict__ alpha,
                      const float* __restrict__ beta, const float* __restrict__ gamma, const float* __restrict__ weight,
                      float2* __restrict__ grad_sigma, int64_t gstride, double* __restrict__ grad_body,
                      const __grid_constant__ LogFactorials log_fact) {
  extern __shared__ __align__(16) double dsm[];
  const int W = L + 1, P = 2 * L + 1;
  double2* ea = reinterpret_cast<double2*>(dsm);  // e^{i m alpha}, 0 <= m <= L
  double2* eg = ea + W;                           // e^{i m gamma}
  double* rt = reinterpret_cast<double*>(eg + W); // sqrt(n), n <= 2 L + 1
  double* rr = rt + P + 1;                        // 1 / sqrt(n), n >= 1
  double* lf = rr + P + 1;                        // log n!, n <= 2 L
  double* pc = lf + P;                            // cos(beta / 2)^n
  double* ps = pc + P;                            // (-sin(beta / 2))^n
  double* rl = ps + P;                            // 1 / n, 1 <= n <= L
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), parts = (int)cluster.num_blocks(), b = blockIdx.y;
  const double al = alpha[b], be = beta[b], ga = gamma[b];
  const double w = weight ? (double)weight[b] : 1.0;
  double hs, hc;
  sincos(0.5 * be, &hs, &hc);
  const double cb = cos(be);
  for (int t = threadIdx.x; t <= P; t += kBT) {
    rt[t] = sqrt((double)t);
    rr[t] = t ? 1.0 / sqrt((double)t) : 0.0;
  }
  for (int t = threadIdx.x; t < P; t += kBT) {
    lf[t] = log_fact.v[t];
    pc[t] = ipow_d(hc, t);
    ps[t] = ipow_d(-hs, t);
  }
  for (int t = threadIdx.x; t < W; t += kBT) {
    rl[t] = t ? 1.0 / t : 0.0;
    double sn, cs;
    sincos(t * al, &sn, &cs);
    ea[t] = make_double2(cs, sn);
    sincos(t * ga, &sn, &cs);
    eg[t] = make_double2(cs, sn);
  }
  __syncthreads();
  const float2* sg = sigma + (int64_t)b * stride;
  float2* gs = grad_sigma ? grad_sigma + (int64_t)b * gstride : nullptr;
  double gx = 0.0, gy = 0.0, gz = 0.0;
  // chains (m', m): m' = 0 needs m >= 0 only (its other half are the images)
  // (32 at a time to the cluster's warps, forwards and backwards in turn: the chains get shorter)
  const int warps = parts * (kBT / 32), gw = (int)(threadIdx.x >> 5) * parts + rank;
  for (int k = 0; k * warps * 32 < W * P; ++k) {
    const int e = (k * warps + ((k & 1) ? warps - 1 - gw : gw)) * 32 + (int)(threadIdx.x & 31);
    if (e >= W * P) continue;
    const int mp = e / P, m = e - mp * P - L;
    if (mp == 0 && m < 0) continue;
    const int am = abs(m), l0 = mp > am ? mp : am;
    // first value at l0: d_{M' M} = sqrt((2M')! / ((M'+M)! (M'-M)!)) cos^(M'+M) (-sin)^(M'-M) of
    // the wedge pair M' = l0, with d_{m m'} = (-1)^{m'-m} d_{m' m} and d_{m' m} = d_{-m -m'}
    const bool own = mp >= am;
    const int M = own ? m : (m > 0 ? mp : -mp);
    const double sgn0 = (!own && m > 0 && ((m - mp) & 1)) ? -1.0 : 1.0;
    double dl = sgn0 * exp(0.5 * (lf[2 * l0] - lf[l0 + M] - lf[l0 - M])) * pc[l0 + M] * ps[l0 - M], dlm1 = 0.0;
    const double2 egm = m >= 0 ? eg[am] : make_double2(eg[am].x, -eg[am].y);
    const double2 ph = cmul_d(ea[mp], egm);
    const double sim = ((mp - m) & 1) ? -1.0 : 1.0;  // the image's sign
    const bool image = mp > 0 || m > 0;
    const double mmp = (double)m * mp;
    double a0 = 0.0;  // a_{l-1}; zero at the chain's first degree
    for (int l = l0; l <= L; ++l) {
      if (l > l0) {
        double dn;
        if (l == 1) {
          dn = cb * dl;
        } else {
          const double inv = (rr[l - m] * rr[l + m]) * (rr[l - mp] * rr[l + mp]) * rl[l - 1];
          dn = ((2.0 * l - 1.0) * ((double)l * (l - 1) * cb - mmp) * dl - l * a0 * dlm1) * inv;
        }
        a0 = (rt[l - m] * rt[l + m]) * (rt[l - mp] * rt[l + mp]);
        dlm1 = dl;
        dl = dn;
      }
      const int64_t blk = (int64_t)mtb_dsize(l - 1);
      const int64_t i1 = blk + (int64_t)(mp + l) * (2 * l + 1) + (m + l);
      const int64_t i2 = blk + (int64_t)(l - mp) * (2 * l + 1) + (l - m);
      // D at (m', m), and at (-m', -m): the image's sign times its conjugate
      const double2 D = make_double2(dl * ph.x, dl * ph.y);
      const double2 Di = make_double2(sim * D.x, -sim * D.y);
      if (gs) {
        gs[i1] = make_float2((float)(w * D.x), (float)(-w * D.y));
        if (image) gs[i2] = make_float2((float)(w * Di.x), (float)(-w * Di.y));
      }
      if (grad_body) {
        const double lo = rt[l + m] * rt[l - m + 1], hi = rt[l - m] * rt[l + m + 1];
        // of an image's row s, with am = sqrt((l+m)(l-m+1)), ap = sqrt((l-m)(l+m+1)):
        // sigma^(x) = i/2 (am s[m-1] + ap s[m+1]), sigma^(y) = (ap s[m+1] - am s[m-1]) / 2,
        // sigma^(z) = i m s[m]
        auto add = [&](int64_t at, int mm, double am_, double ap_, double2 d) {
          const float2 s0 = sg[at];
          const float2 sm = mm > -l ? sg[at - 1] : make_float2(0.f, 0.f);
          const float2 sp = mm < l ? sg[at + 1] : make_float2(0.f, 0.f);
          const double ax = am_ * sm.x, ay = am_ * sm.y, bx = ap_ * sp.x, by = ap_ * sp.y;
          gx -= 0.5 * (d.x * (ay + by) + d.y * (ax + bx));
          gy += 0.5 * (d.x * (bx - ax) - d.y * (by - ay));
          gz -= mm * (d.x * s0.y + d.y * s0.x);
        };
        add(i1, m, lo, hi, D);
        if (image) add(i2, -m, hi, lo, Di);
      }
    }
  }
  if (!grad_body) return;  // the same for the whole cluster
  __shared__ double red[3][kBT / 32], sum[3];
  double g[3] = {gx, gy, gz};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g[k] += __shfl_xor_sync(0xffffffffu, g[k], o);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = g[k];
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double s = 0.0;
    for (int i = 0; i < kBT / 32; ++i) s += red[threadIdx.x][i];
    sum[threadIdx.x] = s;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x < 3) {
    double s = 0.0;
    for (int i = 0; i < parts; ++i) s += cluster.map_shared_rank(&sum[threadIdx.x], i)[0];
    grad_body[(int64_t)b * 3 + threadIdx.x] = w * s;
  }
  cluster.sync();  // no CTA leaves while its sums are read
}

// Template gradient of one degree l and kBC columns c of the sigma blocks by one cluster.
// For fixed l the gradient is the product acc[c, k] = sum_{(b, a)} G_b[a, c] V_b[2l - a, k]
// (signs aside) of depth B (2l + 1) and a small output (2l + 1) x K: bound by reading G once.
// So the batch is split over the kR CTAs of a cluster (subtomograms rank, rank + kR, ...), the columns
// over clusters, and inside a CTA a lane owns a column (a warp reads 32 consecutive
// entries of a row of G), a warp owns kBK radial entries in registers and every n_rg-th row.
// The partial sums meet in shared memory, then through distributed shared memory, in a fixed
// order: deterministic, and no workspace.  The rows of V of n_sub subtomograms are gathered at a
// time (kidx: rows mu = -l..l of kpad[l] entries, -1 padded), so a barrier covers n_sub of them.
// 256 subtomograms at L = 32 (98 MB of G): 84 us, against 2487 us for one CTA per degree
// that walked the batch alone.
constexpr int kBC = 32;   // columns
constexpr int kBK = 8;    // radial entries of a warp
constexpr int kBS = 4;    // subtomograms gathered at a time, where they fit
constexpr int kBW = kBT / 32;

template <int kR>
__global__ void __cluster_dims__(kR, 1, 1) __launch_bounds__(kBT)
sigma_backward_template_kernel(const float2* __restrict__ aV, int64_t v_stride, const float2* __restrict__ gsig,
                               int64_t g_stride, int B, int lmax_g, int n_sub, int rows, const int* __restrict__ kpad,
                               const int* __restrict__ koff, const int* __restrict__ kidx,
                               float2* __restrict__ grad_tmpl) {
  extern __shared__ __align__(16) float2 bsm[];
  __shared__ float2 part[kBW][kBK][kBC];  // per warp; later this CTA's sums, [k][column] over the K entries
  int* at = reinterpret_cast<int*>(bsm + n_sub * rows);  // gather index of (a, k), its lowest bit a's parity
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = kR > 1 ? (int)cluster.block_rank() : 0;
  auto meet = [&] { kR > 1 ? cluster.sync() : __syncthreads(); };
  const int l = lmax_g - (int)blockIdx.z;  // the widest degrees first
  const int w = 2 * l + 1, c0 = (int)blockIdx.y * kBC;
  if (c0 >= w) return;  // the same for the whole cluster
  const int K = kpad[l];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = c0 + lane;
  const int* tab = kidx + koff[l];
  const int64_t goff = mtb_dsize(l - 1);
  for (int k0 = 0; k0 < K; k0 += kBW * kBK) {  // one turn unless K > 64
    const int nk = K - k0 < kBW * kBK ? K - k0 : kBW * kBK;
    const int nkt = (nk + kBK - 1) / kBK;  // warps side by side on the radial entries
    const int nrg = kBW / nkt;             // groups of them on different rows
    const int kt = warp % nkt, rg = warp / nkt;
    const int ks = nkt * kBK;
    const int ne = w * ks;
    __syncthreads();
    for (int e = threadIdx.x; e < ne; e += kBT) {
      const int a = e / ks, k = e - a * ks;
      const int idx = k < nk ? __ldg(&tab[(2 * l - a) * K + k0 + k]) : -1;
      at[e] = idx >= 0 ? 2 * idx + (a & 1) : -1;
    }
    float2 acc[kBK];
#pragma unroll
    for (int k = 0; k < kBK; ++k) acc[k] = make_float2(0.f, 0.f);
    for (int b0 = rank; b0 < B; b0 += kR * n_sub) {
      __syncthreads();
      // sV[i][a][k] = (-1)^a aV_b[l, -(a - l), k]
      for (int e = threadIdx.x; e < ne; e += kBT) {
        const int code = at[e];
        float2 v[kBS];
#pragma unroll
        for (int i = 0; i < kBS; ++i) {
          const int b = b0 + i * kR;
          v[i] = i < n_sub && b < B && code >= 0 ? __ldg(&aV[(int64_t)b * v_stride + (code >> 1)])
                                                 : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < kBS; ++i)
          if (i < n_sub) bsm[i * ne + e] = (code & 1) ? make_float2(-v[i].x, -v[i].y) : v[i];
      }
      __syncthreads();
      if (rg < nrg && c < w) {
        // rows r = (i, a) of the gathered subtomograms, eight loads in flight
        const int have = (B - b0 + kR - 1) / kR, R = (have < n_sub ? have : n_sub) * w;
        const float2* g = gsig + (int64_t)b0 * g_stride + goff + c;
        int a = rg;
        while (a >= w) {
          a -= w;
          g += (int64_t)kR * g_stride;
        }
        for (int r = rg; r < R; r += 8 * nrg) {
          float2 gg[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            gg[j] = r + j * nrg < R ? __ldg(g + (int64_t)a * w) : make_float2(0.f, 0.f);
            a += nrg;
            while (a >= w) {
              a -= w;
              g += (int64_t)kR * g_stride;
            }
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (r + j * nrg >= R) break;
            const float4* v4 = reinterpret_cast<const float4*>(bsm + (r + j * nrg) * ks + kt * kBK);
#pragma unroll
            for (int k = 0; k < kBK / 2; ++k) {
              const float4 v = v4[k];
              acc[2 * k].x = fmaf(v.x, gg[j].x, fmaf(-v.y, gg[j].y, acc[2 * k].x));
              acc[2 * k].y = fmaf(v.x, gg[j].y, fmaf(v.y, gg[j].x, acc[2 * k].y));
              acc[2 * k + 1].x = fmaf(v.z, gg[j].x, fmaf(-v.w, gg[j].y, acc[2 * k + 1].x));
              acc[2 * k + 1].y = fmaf(v.z, gg[j].y, fmaf(v.w, gg[j].x, acc[2 * k + 1].y));
            }
          }
        }
      }
    }
    // rows' groups of this CTA, then the CTAs of the cluster, each in order
#pragma unroll
    for (int k = 0; k < kBK; ++k) part[warp][k][lane] = acc[k];
    __syncthreads();
    for (int e = threadIdx.x; e < nkt * kBK * kBC; e += kBT) {
      const int t = e / (kBK * kBC), k = (e / kBC) % kBK, x = e % kBC;
      float2 s = part[t][k][x];
      for (int q = 1; q < nrg; ++q) {
        const float2 u = part[t + q * nkt][k][x];
        s.x += u.x;
        s.y += u.y;
      }
      part[t][k][x] = s;
    }
    meet();
    for (int e = threadIdx.x + rank * kBT; e < nk * kBC; e += kR * kBT) {
      const int k = e / kBC, x = e % kBC, col = c0 + x;
      if (col >= w) continue;
      const int idx = __ldg(&tab[(2 * l - col) * K + k0 + k]);
      if (idx < 0) continue;
      float2 s = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < kR; ++q) {
        const float2* from = &part[k / kBK][k % kBK][x];
        const float2 u = kR > 1 ? cluster.map_shared_rank(from, q)[0] : *from;
        s.x += u.x;
        s.y += u.y;
      }
      if (col & 1) s = make_float2(-s.x, -s.y);
      grad_tmpl[idx] = s;
    }
    meet();  // no CTA leaves, or overwrites its sums, while others read them
  }
}

// ------------------------------------------------------------------ rotations of a batch
// exp([w]x) = I + a [w]x + b [w]x^2 and the right Jacobian I - c1 [w]x + c2 [w]x^2.
__device__ __forceinline__ void so3_coefficients(double th2, double& a, double& b, double& c2) {
  const double th = sqrt(th2);
  if (th < 1e-6) {
    a = 1.0 - th2 / 6.0;
    b = 0.5 - th2 / 24.0;
    c2 = 1.0 / 6.0 - th2 / 120.0;
  } else {
    double sn, cs;
    sincos(th, &sn, &cs);
    a = sn / th;
    b = (1.0 - cs) / th2;
    c2 = (th - sn) / (th2 * th);
  }
}

// Euler angles of Rz(a) Ry(b) Rz(g) exp([omega]x), FP64 up to the FP32 angles.  One thread per
// rotation: the batch's hundred small matrix operations in one launch.
__global__ void rotation_angles_kernel(const double* __restrict__ omega, const double* __restrict__ base, int B,
                                       float* __restrict__ alpha, float* __restrict__ beta, float* __restrict__ gamma) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B) return;
  const double x = omega[3 * i], y = omega[3 * i + 1], z = omega[3 * i + 2];
  const double x2 = x * x, y2 = y * y, z2 = z * z;
  double a, b, c2;
  so3_coefficients(x2 + y2 + z2, a, b, c2);
  const double E[3][3] = {{1.0 - b * (y2 + z2), b * x * y - a * z, b * x * z + a * y},
                          {b * x * y + a * z, 1.0 - b * (x2 + z2), b * y * z - a * x},
                          {b * x * z - a * y, b * y * z + a * x, 1.0 - b * (x2 + y2)}};
  double sa, ca, sb, cb, sg, cg;
  sincos(base[3 * i], &sa, &ca);
  sincos(base[3 * i + 1], &sb, &cb);
  sincos(base[3 * i + 2], &sg, &cg);
  const double Z[3][3] = {{ca * cb * cg - sa * sg, -ca * cb * sg - sa * cg, ca * sb},
                          {sa * cb * cg + ca * sg, -sa * cb * sg + ca * cg, sa * sb},
                          {-sb * cg, sb * sg, cb}};
  double R[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) R[r][c] = Z[r][0] * E[0][c] + Z[r][1] * E[1][c] + Z[r][2] * E[2][c];
  const double s = sqrt(R[0][2] * R[0][2] + R[1][2] * R[1][2]);
  double al, be, ga;
  if (s < 1e-12) {  // beta = 0 or pi: only a + g or a - g is defined, g = 0
    const bool up = R[2][2] > 0;
    al = up ? atan2(R[1][0], R[0][0]) : atan2(-R[1][0], -R[0][0]);
    be = up ? 0.0 : 3.14159265358979323846;
    ga = 0.0;
  } else {
    al = atan2(R[1][2], R[0][2]);
    be = atan2(s, R[2][2]);
    ga = atan2(R[2][1], -R[2][0]);
  }
  alpha[i] = (float)al;
  beta[i] = (float)be;
  gamma[i] = (float)ga;
}

// grad_omega = Jr(omega)^T grad_body.
__global__ void rotation_gradient_kernel(const double* __restrict__ omega, const double* __restrict__ grad_body, int B,
                                         double* __restrict__ grad_omega) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B) return;
  const double x = omega[3 * i], y = omega[3 * i + 1], z = omega[3 * i + 2];
  const double x2 = x * x, y2 = y * y, z2 = z * z;
  double a, c1, c2;
  so3_coefficients(x2 + y2 + z2, a, c1, c2);
  // rows of Jr = I - c1 [w]x + c2 [w]x^2, transposed on the way out
  const double J[3][3] = {{1.0 - c2 * (y2 + z2), c2 * x * y + c1 * z, c2 * x * z - c1 * y},
                          {c2 * x * y - c1 * z, 1.0 - c2 * (x2 + z2), c2 * y * z + c1 * x},
                          {c2 * x * z + c1 * y, c2 * y * z - c1 * x, 1.0 - c2 * (x2 + y2)}};
  const double g[3] = {grad_body[3 * i], grad_body[3 * i + 1], grad_body[3 * i + 2]};
#pragma unroll
  for (int c = 0; c < 3; ++c) grad_omega[3 * i + c] = J[0][c] * g[0] + J[1][c] * g[1] + J[2][c] * g[2];
}

}  // namespace

extern "C" int mtb_score_backward(const float* sigma, int64_t sigma_stride, int B, int L, const float* alpha,
                                  const float* beta, const float* gamma, const float* weight, float* grad_sigma,
                                  int64_t grad_stride, double* grad_body, mtb_stream_t stream) {
  MTB_ARG_CHECK(B >= 0, "negative batch");
  MTB_ARG_CHECK(L >= 0 && L <= 128, "L must be in [0, 128]");
  if (B == 0) return MTB_OK;
  MTB_ARG_CHECK(alpha && beta && gamma, "null angles");
  MTB_ARG_CHECK(grad_sigma || grad_body, "nothing to compute");
  MTB_ARG_CHECK(!grad_body || (sigma && sigma_stride >= mtb_dsize(L)), "sigma row shorter than dsize(L)");
  MTB_ARG_CHECK(!grad_sigma || grad_stride >= mtb_dsize(L), "grad_sigma row shorter than dsize(L)");
  MTB_ARG_CHECK(B <= 2147483647, "batch too large");
  cudaStream_t st = (cudaStream_t)stream;
  mtb_prof_begin(st);
  const int parts = cluster_size(B, 4);
  LogFactorials log_fact;
  for (int n = 0; n < 257; ++n) log_fact.v[n] = n <= 2 * L ? lgamma(n + 1.0) : 0.0;
  for (int b0 = 0; b0 < B; b0 += 65535) {  // the grid's y limit
    const int n = B - b0 < 65535 ? B - b0 : 65535;
    MTB_CUDA_TRY(launch_clusters(score_backward_kernel, dim3(parts, n), kBT, score_backward_smem(L), parts, st,
                                 reinterpret_cast<const float2*>(sigma) + (sigma ? b0 * sigma_stride : 0),
                                 sigma_stride, L, alpha + b0, beta + b0, gamma + b0, weight ? weight + b0 : weight,
                                 grad_sigma ? reinterpret_cast<float2*>(grad_sigma) + b0 * grad_stride : nullptr,
                                 grad_stride, grad_body ? grad_body + (int64_t)3 * b0 : nullptr, log_fact));
  }
  mtb_prof_end(st, "score_backward_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}

// The FLE handle's gather tables (fle.cu) for the template backward.
int fle_sigma_tables(const mtb_fle* h, const int** kpad, const int** koff, const int** kidx, int* lmax, int* kmax,
                     int* ne, const int** kpad_host);

extern "C" int mtb_sigma_backward_template(mtb_fle* h, const float* coeffs, int64_t coeff_stride,
                                           const float* grad_sigma, int64_t grad_stride, int B, int lmax_g,
                                           float* grad_tmpl, mtb_stream_t stream) {
  MTB_ARG_CHECK(h, "null handle");
  const int *kpad, *koff, *kidx, *kpad_host;
  int lmax, kmax, ne;
  if (int rc = fle_sigma_tables(h, &kpad, &koff, &kidx, &lmax, &kmax, &ne, &kpad_host)) return rc;
  MTB_ARG_CHECK(lmax_g >= 0 && lmax_g <= lmax, "lmax_g must be in [0, lmax of the expansion]");
  MTB_ARG_CHECK(B >= 0, "negative batch");
  MTB_ARG_CHECK(grad_tmpl, "null output");
  cudaStream_t st = (cudaStream_t)stream;
  // degrees above lmax_g (and the padding entry ne) get no gradient
  MTB_CUDA_TRY(cudaMemsetAsync(grad_tmpl, 0, (size_t)(ne + 1) * sizeof(float2), st));
  if (B == 0) return MTB_OK;
  MTB_ARG_CHECK(coeffs && grad_sigma, "null pointer");
  MTB_ARG_CHECK(coeff_stride >= ne, "coefficient row shorter than ne");
  MTB_ARG_CHECK(grad_stride >= mtb_dsize(lmax_g), "grad_sigma row shorter than dsize(lmax_g)");
  const int w = 2 * lmax_g + 1, ks = kmax | 1;
  // the degrees accepted: those whose (2l + 1)^2 block fits beside the coefficient rows on an SM
  MTB_ARG_CHECK(((size_t)w * ks + (size_t)w * w + (size_t)w * kmax) * sizeof(float2) <= 227 * 1024,
                "degree too high for the shared-memory staging of the template backward");
  // gathered rows of one subtomogram, the largest over the degrees (at most
  // 64 entries of fewer than 171 rows: 2 l + 1 squared alone is below the limit above)
  size_t rows = 0;
  for (int l = 0; l <= lmax_g; ++l) {
    const int nk = kpad_host[l] < kBW * kBK ? kpad_host[l] : kBW * kBK;
    const size_t n = (size_t)(2 * l + 1) * ((nk + kBK - 1) / kBK * kBK) * sizeof(float2);
    rows = n > rows ? n : rows;
  }
  int n_sub = kBS;
  while (n_sub > 1 && n_sub * rows + rows / 2 > 200 * 1024) --n_sub;
  const size_t smem = n_sub * rows + rows / 2;  // and a gather index for each entry
  // up to kBS subtomograms are one gather of a CTA: eight would only meet (one of 64^3 10.3 us, 13.7)
  const auto kernel = B <= kBS ? sigma_backward_template_kernel<1> : sigma_backward_template_kernel<8>;
  MTB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  mtb_prof_begin(st);
  kernel<<<dim3(B <= kBS ? 1 : 8, (w + kBC - 1) / kBC, lmax_g + 1), kBT, smem, st>>>(
      reinterpret_cast<const float2*>(coeffs), coeff_stride, reinterpret_cast<const float2*>(grad_sigma), grad_stride,
      B, lmax_g, n_sub, (int)(rows / sizeof(float2)), kpad, koff, kidx, reinterpret_cast<float2*>(grad_tmpl));
  mtb_prof_end(st, "sigma_backward_template_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}

extern "C" int mtb_rotation_angles(const double* omega, const double* base, int B, float* alpha, float* beta,
                                   float* gamma, mtb_stream_t stream) {
  MTB_ARG_CHECK(B >= 0, "negative batch");
  if (B == 0) return MTB_OK;
  MTB_ARG_CHECK(omega && base && alpha && beta && gamma, "null pointer");
  const cudaStream_t st = (cudaStream_t)stream;
  mtb_prof_begin(st);
  rotation_angles_kernel<<<(B + 63) / 64, 64, 0, st>>>(omega, base, B, alpha, beta, gamma);
  mtb_prof_end(st, "rotation_angles_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}

extern "C" int mtb_rotation_gradient(const double* omega, const double* grad_body, int B, double* grad_omega,
                                     mtb_stream_t stream) {
  MTB_ARG_CHECK(B >= 0, "negative batch");
  if (B == 0) return MTB_OK;
  MTB_ARG_CHECK(omega && grad_body && grad_omega, "null pointer");
  const cudaStream_t st = (cudaStream_t)stream;
  mtb_prof_begin(st);
  rotation_gradient_kernel<<<(B + 63) / 64, 64, 0, st>>>(omega, grad_body, B, grad_omega);
  mtb_prof_end(st, "rotation_gradient_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}
