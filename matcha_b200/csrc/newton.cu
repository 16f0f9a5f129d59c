// Frequency-marched Wigner-D Newton refinement on sm_100a (one CTA per candidate).
//
// Reference behaviour restated here (paths inside swing-research/Matcha):
//   Newton march  src/matcha/core/Matcha.py:150-205 (_take_step), 239-367 (optimize),
//                 369-398 (stage loop)
//   D             src/matcha/core/WignerDMatrices.py:281-306, 673-801, 1291-1375
//   g, H          src/matcha/core/WignerDGradients.py:155-302
//
// The score of a point (a, b, g) is f = Re sum_l sum_{m'm} e^{i m' a} d^l_{m'm}(b) e^{i m g}
// sigma_{l m' m}.  Its Euler gradient and Hessian are computed here from one sweep per
// fundamental-wedge chain instead of from the full D matrix:
//
//  * Symmetry folding.  d_{m m'} = d_{-m',-m} = (-1)^{m'-m} d_{m'm}, d_{-m,-m'} = d_{m'm}.
//    The four images (M',M), (M,M'), (-M,-M'), (-M',-M) of a wedge pair M' >= |M| carry the
//    phases z1 = e^{i(M'a + Mg)}, z2 = e^{i(Ma + M'g)} and their conjugates, so
//      sum over the images = d^l_{M'M}(b) Re(z1 S1_l + z2 S2_l)
//    with S1 = sigma(M',M) + s conj sigma(-M',-M), S2 = s sigma(M,M') + conj sigma(-M,-M'),
//    s = (-1)^{M'-M} (diagonal and anti-diagonal images coincide and are counted once).
//    S is candidate-independent: it is folded once per subtomogram into a wedge-ordered
//    array, 16 bytes per (l, wedge pair) instead of 32 bytes of sigma.
//  * Phases out of the sum.  z1 and z2 are fixed along a chain (fixed M', M, all l), so a
//    thread accumulates A = sum_l d S, B = sum_l d' S, C = sum_l d'' S per chain and applies
//    z1, z2 and the factors i M', i M of the a- and g-derivatives once at the chain's end.
//  * beta derivatives by differentiated recurrences.  d^l = (al cos b - be) d^{l-1} - ga
//    d^{l-2} (the three-term recurrence in l; al, be, ga from a candidate-independent FP64
//    table) is differentiated twice in b, so d', d'' ride along in registers: no neighbour
//    rows, no shared d blocks and no barriers inside a pass.
//
// Each thread walks whole chains (a wedge pair from l = M' to the stage degree), for the two
// candidates of its CTA at once; chains are dealt to threads in boustrophedon order so that
// long (small M') and short chains mix.
#include <math.h>
#include "common.cuh"
#include "newton.cuh"

namespace {

constexpr int kNT = kNewtonThreads;

enum { A_VAL = 0, A_GA, A_GB, A_GG, A_HAA, A_HAB, A_HAG, A_HBB, A_HBG, A_HGG, A_N };

// A candidate's point with what a pass needs of it.
struct Point {
  double hs, hc;       // sin, cos of beta / 2
  float a, be, ga;
  float sb, cb;        // sin, cos of beta
};

// Per-candidate tables of one pass (NC candidates of one subtomogram per CTA).
template <int NC>
struct Smem {
  float2 (*ea)[kNewtonMaxL + 1];       // e^{i k a}, k = 0 .. Li
  float2 (*eg)[kNewtonMaxL + 1];       // e^{i k g}
  double (*phc)[2 * kNewtonMaxL + 3];  // cos(b/2)^k, k = 0 .. 2 Li + 2
  double (*pt)[2 * kNewtonMaxL + 3];   // (-sin(b/2))^k
  uint32_t* off;                       // 16 wedge_off(l): byte offset of degree l
  float* red;                          // (threads/32) x NC x A_N
  float* res;                          // NC x A_N
};

__device__ __forceinline__ double ipow(double x, int n) {
  double r = 1.0;
  while (n) {
    if (n & 1) r *= x;
    x *= x;
    n >>= 1;
  }
  return r;
}

// Offset of degree l in the wedge-ordered arrays: sum_{j < l} (j + 1)^2.
__host__ __device__ __forceinline__ int64_t wedge_off(int l) { return (int64_t)l * (l + 1) * (2 * l + 1) / 6; }

// Wedge index p = M'^2 + M' + M, 0 <= |M| <= M'.
__device__ __forceinline__ void wedge_pair(int p, int& mp, int& m) {
  mp = (int)sqrtf((float)p);
  while (mp * mp > p) --mp;
  while ((mp + 1) * (mp + 1) <= p) ++mp;
  m = p - mp * mp - mp;
}

// Folded sigma {Re S1, Im S1, Re S2, Im S2} of wedge pair (mp, m) at degree l >= mp, read
// from the reference layout (flat [l][m'][m], w = 2l + 1).
__device__ __forceinline__ float4 fold_entry(const float2* __restrict__ sg, int l, int mp, int m) {
  const int w = 2 * l + 1;
  const float2* blk = sg + mtb_dsize(l - 1);
  auto at = [&](int r, int c) -> float2 { return __ldg(blk + (r + l) * w + (c + l)); };
  const float s = ((mp - m) & 1) ? -1.f : 1.f;
  const float2 s1 = at(mp, m);
  if (mp == 0) return make_float4(s1.x, s1.y, 0.f, 0.f);
  const float2 s4 = at(-mp, -m);
  const float r1 = s1.x + s * s4.x, i1 = s1.y - s * s4.y;
  if (m == mp || m == -mp) return make_float4(r1, i1, 0.f, 0.f);
  const float2 s2 = at(m, mp), s3 = at(-m, -mp);
  return make_float4(r1, i1, s * s2.x + s3.x, s * s2.y - s3.y);
}

// S[b][wedge_off(l) + p] for every degree l <= Lmax and wedge pair p < (l + 1)^2.
__global__ void fold_sigma_kernel(const float2* __restrict__ sigma, int64_t stride, int64_t n_fold,
                                  float4* __restrict__ S) {
  const int l = blockIdx.x, b = blockIdx.y;
  const float2* sg = sigma + (int64_t)b * stride;
  float4* out = S + (int64_t)b * n_fold + wedge_off(l);
  const int n = (l + 1) * (l + 1);
  for (int p = threadIdx.x; p < n; p += blockDim.x) {
    int mp, m;
    wedge_pair(p, mp, m);
    out[p] = fold_entry(sg, l, mp, m);
  }
}

// Recurrence factors {al, be, ga} of d^l_{M'M} = (al cos b - be) d^{l-1} - ga d^{l-2}
// for l > M', from
//   (l-1) sqrt((l^2-m^2)(l^2-m'^2)) d^l = (2l-1)(l(l-1) cos b - m m') d^{l-1}
//                                        - l sqrt(((l-1)^2-m^2)((l-1)^2-m'^2)) d^{l-2},
// in FP64; d^1_{00} = cos b d^0_{00}.  Entries with l <= M' are unused and zero.
__global__ void coef_kernel(int64_t n, float4* __restrict__ coef) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    int l = 0;
    while (wedge_off(l + 1) <= t) ++l;
    const int p = (int)(t - wedge_off(l));
    int mp, m;
    wedge_pair(p, mp, m);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (l == 1 && mp == 0) {
      v.x = 1.f;
    } else if (l >= 2 && l > mp) {
      const double L = l, m2 = (double)m * m, mp2 = (double)mp * mp;
      const double inv = 1.0 / sqrt((L * L - m2) * (L * L - mp2));
      const double xl1 = ((L - 1) * (L - 1) - m2) * ((L - 1) * (L - 1) - mp2);
      v.x = (float)((2 * L - 1) * L * inv);
      v.y = (float)((2 * L - 1) * (double)m * mp * inv / (L - 1));
      v.z = (float)(L * sqrt(fmax(xl1, 0.0)) * inv / (L - 1));
    }
    coef[t] = v;
  }
}

// The point of a candidate: its trigonometric values, once for the CTA.
__device__ __forceinline__ Point make_point(float a, float be, float ga) {
  Point p;
  p.a = a;
  p.be = be;
  p.ga = ga;
  sincos(0.5 * (double)be, &p.hs, &p.hc);
  sincosf(be, &p.sb, &p.cb);
  return p;
}

__device__ __forceinline__ const float4* at_bytes(const float4* base, uint32_t off) {
  return reinterpret_cast<const float4*>(reinterpret_cast<const char*>(base) + off);
}

// Sums of N values over a warp, each by the tree of an exchange between lanes 16, 8, 4, 2 and 1
// apart.  While a lane holds an even number of values it hands half of them over and keeps the
// other half's sums, so the 20 values of a pass cost 30 exchanges instead of 100; a value's
// additions are the same.  out[i] receives the sum of value i.
template <int N, int O>
struct WarpSums {
  static __device__ __forceinline__ void run(float (&x)[N], int lane, int first, float* out) {
    if constexpr (O >= 1 && N % 2 == 0) {
      constexpr int M = N / 2;
      const bool up = lane & O;
      float y[M];
#pragma unroll
      for (int j = 0; j < M; ++j) {
        const float give = up ? x[j] : x[j + M], keep = up ? x[j + M] : x[j];
        y[j] = keep + __shfl_xor_sync(0xffffffffu, give, O);
      }
      first += up ? M : 0;
      WarpSums<M, O / 2>::run(y, lane, first, out);
    } else {
#pragma unroll
      for (int o = O; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < N; ++j) x[j] += __shfl_xor_sync(0xffffffffu, x[j], o);
      if ((lane & (2 * O - 1)) == 0)
#pragma unroll
        for (int j = 0; j < N; ++j) out[first + j] = x[j];
    }
  }
};

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)));
}

// One sweep over the chains of stage degree Li at the NC points pts[c] of one subtomogram's
// candidates: value, and with DERIVS the Euler gradient and Hessian, left in
// sm.res[c * A_N + ..].  The candidates share each chain's loads of the folded sigma and of
// the recurrence factors; their d, d', d'' run side by side.  FOLDED reads the folded sigma S
// of this subtomogram; otherwise each step folds the four images from sigma itself.
//
// Issue and the latency of its L2 loads bound it, and of the 24 M thread instructions a subtomogram took at L = 32 only a third
// were FP32; so everything around the chain steps is kept short: the points' trigonometry and the
// FP64 step are one thread's, tables hold k >= 0 and are filled by all threads, offsets are 32-bit,
// the sums of a warp are exchanged by halves.  March of 1000 subtomograms at L = 32 1104 -> 884 us,
// 64 at L = 64 608 -> 509 us, 16 at L = 16 (five steps) 86 -> 50 us.  (A cp.async ring of four steps
// per thread instead of plain loads measured 1196 and 543 us before these; 96 registers and five
// CTAs per SM 890 and 704 us.)
template <bool DERIVS, bool FOLDED, int NC>
__device__ __forceinline__ void pass(const float4* __restrict__ S, const float2* __restrict__ sg,
                                     const float4* __restrict__ coef, const double* __restrict__ Ctab,
                                     const Point* pts, int Li, const Smem<NC> sm) {
  const int tid = threadIdx.x;
  const double two_pi = 6.283185307179586;
  for (int e = tid; e < NC * 2 * (Li + 1); e += kNT) {
    const int c = e / (2 * (Li + 1)), r = e - c * (2 * (Li + 1)), g = r > Li, k = r - g * (Li + 1);
    double t = (double)k * (double)(g ? pts[c].ga : pts[c].a);
    t -= two_pi * rint(t / two_pi);
    float s, co;
    sincosf((float)t, &s, &co);
    (g ? sm.eg : sm.ea)[c][k] = make_float2(co, s);
  }
  const int np = DERIVS ? 2 * Li + 3 : 2 * Li + 1;
  for (int e = tid; e < NC * 2 * np; e += kNT) {
    const int c = e / (2 * np), r = e - c * (2 * np), h = r >= np, k = r - h * np;
    (h ? sm.pt : sm.phc)[c][k] = ipow(h ? -pts[c].hs : pts[c].hc, k);
  }
  float sb[NC], cb[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    sb[c] = pts[c].sb;
    cb[c] = pts[c].cb;
  }

  constexpr int NA = DERIVS ? A_N : 1;
  float acc[NC][NA];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int i = 0; i < NA; ++i) acc[c][i] = 0.f;
  __syncthreads();

  const int n = (Li + 1) * (Li + 1);
  int k = 0;
  for (int base = 0; base < n; base += kNT, ++k) {
    const int p = base + ((k & 1) ? kNT - 1 - tid : tid);
    if (p >= n) continue;
    float root;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(root) : "f"((float)p + 0.5f));
    const int mp = (int)root, m = p - mp * mp - mp;  // wedge_pair (the half keeps the root off integers)
    // start of the chain at l = M': d = C cos^P (-sin)^Q of b/2, P = M'+M, Q = M'-M
    const int P = mp + m, Q = mp - m;
    const double Cp = Ctab[p];
    float d1[NC], d0[NC], e1[NC], e0[NC], g1[NC], g0[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      d1[c] = (float)(Cp * sm.phc[c][P] * sm.pt[c][Q]);
      d0[c] = 0.f;
      e1[c] = e0[c] = g1[c] = g0[c] = 0.f;
      if (DERIVS) {
        double fp = 0.0, fpp = -(double)(2 * P * Q + P + Q) * sm.phc[c][P] * sm.pt[c][Q];
        if (P >= 1) fp += P * sm.phc[c][P - 1] * sm.pt[c][Q + 1];
        if (Q >= 1) fp -= Q * sm.phc[c][P + 1] * sm.pt[c][Q - 1];
        if (P >= 2) fpp += (double)(P * (P - 1)) * sm.phc[c][P - 2] * sm.pt[c][Q + 2];
        if (Q >= 2) fpp += (double)(Q * (Q - 1)) * sm.phc[c][P + 2] * sm.pt[c][Q - 2];
        e1[c] = (float)(0.5 * Cp * fp);
        g1[c] = (float)(0.25 * Cp * fpp);
      }
    }
    uint32_t off = sm.off[mp] + 16u * (uint32_t)p;
    float4 s;
    if (FOLDED) s = __ldg(at_bytes(S, off));
    else s = fold_entry(sg, mp, mp, m);
    // per candidate: A = sum d S (a1 = S1 part, a2 = S2 part), B = sum d' S, C = sum d'' S
    float A1r[NC], A1i[NC], A2r[NC], A2i[NC];
    float B1r[NC], B1i[NC], B2r[NC], B2i[NC], C1r[NC], C1i[NC], C2r[NC], C2i[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      A1r[c] = d1[c] * s.x; A1i[c] = d1[c] * s.y; A2r[c] = d1[c] * s.z; A2i[c] = d1[c] * s.w;
      B1r[c] = B1i[c] = B2r[c] = B2i[c] = C1r[c] = C1i[c] = C2r[c] = C2i[c] = 0.f;
      if (DERIVS) {
        B1r[c] = e1[c] * s.x; B1i[c] = e1[c] * s.y; B2r[c] = e1[c] * s.z; B2i[c] = e1[c] * s.w;
        C1r[c] = g1[c] * s.x; C1i[c] = g1[c] * s.y; C2r[c] = g1[c] * s.z; C2i[c] = g1[c] * s.w;
      }
    }
    // one chain step from its recurrence factors and folded sigma
    auto step = [&](const float4 cf, const float4 s) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const float t = fmaf(cf.x, cb[c], -cf.y);
        const float v = fmaf(t, d1[c], -cf.z * d0[c]);
        if (DERIVS) {
          const float as = cf.x * sb[c];
          const float vp = fmaf(t, e1[c], -fmaf(as, d1[c], cf.z * e0[c]));
          const float vpp = fmaf(t, g1[c], -fmaf(2.f * as, e1[c], fmaf(cf.x * cb[c], d1[c], cf.z * g0[c])));
          e0[c] = e1[c]; e1[c] = vp;
          g0[c] = g1[c]; g1[c] = vpp;
        }
        d0[c] = d1[c]; d1[c] = v;
        A1r[c] = fmaf(v, s.x, A1r[c]); A1i[c] = fmaf(v, s.y, A1i[c]);
        A2r[c] = fmaf(v, s.z, A2r[c]); A2i[c] = fmaf(v, s.w, A2i[c]);
        if (DERIVS) {
          B1r[c] = fmaf(e1[c], s.x, B1r[c]); B1i[c] = fmaf(e1[c], s.y, B1i[c]);
          B2r[c] = fmaf(e1[c], s.z, B2r[c]); B2i[c] = fmaf(e1[c], s.w, B2i[c]);
          C1r[c] = fmaf(g1[c], s.x, C1r[c]); C1i[c] = fmaf(g1[c], s.y, C1i[c]);
          C2r[c] = fmaf(g1[c], s.z, C2r[c]); C2i[c] = fmaf(g1[c], s.w, C2i[c]);
        }
      }
    };
    // degree l + 1 lies 16 (l + 1)^2 bytes after degree l
    uint32_t inc = 16u * (uint32_t)((mp + 1) * (mp + 1)), grow = 16u * (uint32_t)(2 * mp + 3);
    off += inc;
#pragma unroll 4
    for (int l = mp + 1; l <= Li; ++l) {
      const float4 cf = __ldg(at_bytes(coef, off));
      step(cf, FOLDED ? __ldg(at_bytes(S, off)) : fold_entry(sg, l, mp, m));
      inc += grow;
      grow += 32u;
      off += inc;
    }
    // phases: z1 = e^{i(M'a + Mg)}, z2 = e^{i(Ma + M'g)}
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int am = abs(m);
      float2 eam = sm.ea[c][am], egm = sm.eg[c][am];
      if (m < 0) {
        eam.y = -eam.y;
        egm.y = -egm.y;
      }
      const float2 z1 = cmulf(sm.ea[c][mp], egm);
      const float2 z2 = cmulf(eam, sm.eg[c][mp]);
      // which product of a pair is fused is written out, so that the one- and two-candidate kernels,
      // and later compilers, round alike
      auto real = [](float2 z, float r, float i) { return __fmaf_rn(z.x, r, -__fmul_rn(z.y, i)); };
      auto imag = [](float2 z, float r, float i) { return __fmaf_rn(z.x, i, __fmul_rn(z.y, r)); };
      auto lin = [](float x, float u, float y, float v) { return __fmaf_rn(x, u, __fmul_rn(y, v)); };
      auto add = [](float& to, float v) { to = __fadd_rn(to, v); };
      const float r1 = real(z1, A1r[c], A1i[c]), r2 = real(z2, A2r[c], A2i[c]);
      add(acc[c][A_VAL], __fadd_rn(r1, r2));
      if (DERIVS) {
        const float fM = (float)mp, fm = (float)m;
        const float j1 = imag(z1, A1r[c], A1i[c]), j2 = imag(z2, A2r[c], A2i[c]);
        const float q1 = real(z1, B1r[c], B1i[c]), q2 = real(z2, B2r[c], B2i[c]);
        const float k1 = imag(z1, B1r[c], B1i[c]), k2 = imag(z2, B2r[c], B2i[c]);
        const float h1 = real(z1, C1r[c], C1i[c]), h2 = real(z2, C2r[c], C2i[c]);
        add(acc[c][A_GA], -lin(fM, j1, fm, j2));
        add(acc[c][A_GG], -lin(fm, j1, fM, j2));
        add(acc[c][A_GB], __fadd_rn(q1, q2));
        add(acc[c][A_HAA], -lin(__fmul_rn(fM, fM), r1, __fmul_rn(fm, fm), r2));
        add(acc[c][A_HGG], -lin(__fmul_rn(fm, fm), r1, __fmul_rn(fM, fM), r2));
        acc[c][A_HAG] = __fmaf_rn(-__fmul_rn(fM, fm), __fadd_rn(r1, r2), acc[c][A_HAG]);
        add(acc[c][A_HAB], -lin(fM, k1, fm, k2));
        add(acc[c][A_HBG], -lin(fm, k1, fM, k2));
        add(acc[c][A_HBB], __fadd_rn(h1, h2));
      }
    }
  }

  // ---- block reduction
  const int lane = tid & 31, warp = tid >> 5;
  {
    float x[NC * NA];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int i = 0; i < NA; ++i) x[c * NA + i] = acc[c][i];
    WarpSums<NC * NA, 16>::run(x, lane, 0, sm.red + warp * NC * A_N);
  }
  __syncthreads();
  if (tid < NC * A_N) {
    const int c = tid / A_N, i = tid - (tid / A_N) * A_N;
    if (i < NA) {
      float s2 = 0.f;
      for (int q = 0; q < kNT / 32; ++q) s2 += sm.red[q * NC * A_N + c * NA + i];
      sm.res[c * A_N + i] = s2;
    }
  }
  __syncthreads();
}

// Solve H x = g in FP64 with partial pivoting; false when a pivot is exactly zero
// (torch.linalg.solve raises "singular" there and the reference takes a zero step,
// Matcha.py:316-343).
__device__ bool solve3(const double H[3][3], const double g[3], double x[3]) {
  double A[3][4];
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < 3; ++j) A[i][j] = H[i][j];
    A[i][3] = g[i];
  }
  for (int c = 0; c < 3; ++c) {
    int piv = c;
    for (int r = c + 1; r < 3; ++r)
      if (fabs(A[r][c]) > fabs(A[piv][c])) piv = r;
    if (A[piv][c] == 0.0 || !isfinite(A[piv][c])) return false;
    if (piv != c)
      for (int j = 0; j < 4; ++j) { double t = A[c][j]; A[c][j] = A[piv][j]; A[piv][j] = t; }
    for (int r = c + 1; r < 3; ++r) {
      const double f = A[r][c] / A[c][c];
      for (int j = c; j < 4; ++j) A[r][j] -= f * A[c][j];
    }
  }
  for (int r = 2; r >= 0; --r) {
    double s = A[r][3];
    for (int j = r + 1; j < 3; ++j) s -= A[r][j] * x[j];
    x[r] = s / A[r][r];
  }
  return true;
}

// One CTA per NC candidates of one subtomogram (C % NC == 0).  Each candidate keeps its own
// point, learning rate, gradient and Hessian; the passes evaluate all NC together.
template <bool FOLDED, int NC>
__global__ void __launch_bounds__(kNT, 4)
newton_march_kernel(const float4* __restrict__ S, int64_t n_fold, const float2* __restrict__ sigma, int64_t stride,
                    int BC, int C, float* __restrict__ alpha, float* __restrict__ beta, float* __restrict__ gamma,
                    float* __restrict__ score, const double* __restrict__ Ctab, const float4* __restrict__ coef,
                    NewtonParams P) {
  __shared__ float2 s_ea[NC][kNewtonMaxL + 1], s_eg[NC][kNewtonMaxL + 1];
  __shared__ double s_phc[NC][2 * kNewtonMaxL + 3], s_pt[NC][2 * kNewtonMaxL + 3];
  __shared__ uint32_t s_off[kNewtonMaxL + 1];
  __shared__ float s_red[(kNT / 32) * NC * A_N], s_res[NC * A_N];
  __shared__ Point s_now[NC], s_try[NC];  // each candidate's accepted and trial point
  const Smem<NC> sm{s_ea, s_eg, s_phc, s_pt, s_off, s_red, s_res};

  const int cand0 = blockIdx.x * NC;
  if (cand0 >= BC) return;
  const int b = cand0 / C;
  const float4* Sb = FOLDED ? S + (int64_t)b * n_fold : nullptr;
  const float2* sg = FOLDED ? nullptr : sigma + (int64_t)b * stride;
  const bool grad_step = (P.flags & MTB_SEARCH_GRADIENT_STEP) != 0;
  const float base_lr = grad_step ? 5e-7f : 1.f;
  for (int l = threadIdx.x; l <= P.Lmax; l += kNT) s_off[l] = 16u * (uint32_t)wedge_off(l);

  // candidate c's state (best score, learning rate, gradient and Hessian at the accepted point)
  // is one thread's, in a warp of its own: it takes the FP64 step while the other CTAs of the SM
  // have the issue slots
  const int c = threadIdx.x >> 5;
  const bool owner = (threadIdx.x & 31) == 0 && c < NC;
  // (in shared memory: registers would be live across the passes)
  __shared__ float s_gh[NC][A_N], s_best[NC], s_lr[NC];
  float* gh = s_gh[owner ? c : 0];
  if (owner) s_now[c] = make_point(alpha[cand0 + c], beta[cand0 + c], gamma[cand0 + c]);
  __syncthreads();
  for (int st = 0; st < P.n_stages; ++st) {
    const int Li = P.stages[st];
    if (P.num_steps > 0)
      pass<true, FOLDED, NC>(Sb, sg, coef, Ctab, s_now, Li, sm);
    else
      pass<false, FOLDED, NC>(Sb, sg, coef, Ctab, s_now, Li, sm);
    if (owner) {
#pragma unroll
      for (int i = 0; i < A_N; ++i) gh[i] = s_res[c * A_N + i];
      s_best[c] = gh[A_VAL];
      s_lr[c] = base_lr;
    }
    for (int it = 0; it < P.num_steps; ++it) {
      if (owner) {
        const double g[3] = {gh[A_GA], gh[A_GB], gh[A_GG]};
        const double H[3][3] = {{gh[A_HAA], gh[A_HAB], gh[A_HAG]},
                                {gh[A_HAB], gh[A_HBB], gh[A_HBG]},
                                {gh[A_HAG], gh[A_HBG], gh[A_HGG]}};
        double x[3] = {0.0, 0.0, 0.0};
        if (grad_step) {
          for (int i = 0; i < 3; ++i) x[i] = -g[i];
        } else if (!solve3(H, g, x)) {
          x[0] = x[1] = x[2] = 0.0;
        }
        const Point now = s_now[c];
        const float lr = s_lr[c];
        const float ta = now.a - lr * (float)x[0];
        const float tb = now.be - lr * (float)x[1];
        const float tg = now.ga - lr * (float)x[2];
        s_try[c] = make_point(ta, tb, tg);
      }
      __syncthreads();
      const bool last = (it == P.num_steps - 1);
      if (last)
        pass<false, FOLDED, NC>(Sb, sg, coef, Ctab, s_try, Li, sm);
      else
        pass<true, FOLDED, NC>(Sb, sg, coef, Ctab, s_try, Li, sm);
      if (owner) {
        const float ev = s_res[c * A_N + A_VAL];
        if (ev > s_best[c]) {
          s_now[c] = s_try[c];
          s_best[c] = ev;
          s_lr[c] *= 1.1f;
          if (!last) {
#pragma unroll
            for (int i = 0; i < A_N; ++i) gh[i] = s_res[c * A_N + i];
          }
        } else {
          s_lr[c] *= 0.5f;
        }
      }
    }
    __syncthreads();  // the accepted points, before the next stage's pass
  }
  if (owner) {
    alpha[cand0 + c] = s_now[c].a;
    beta[cand0 + c] = s_now[c].be;
    gamma[cand0 + c] = s_now[c].ga;
    score[cand0 + c] = s_best[c];
  }
}

// The score and its Euler derivatives at one given point per subtomogram, degrees <= Li:
// out[b] = (f, df/da, df/db, df/dg, d2f/da2, d2f/dadb, d2f/dadg, d2f/db2, d2f/dbdg, d2f/dg2),
// the same sweep the march makes at each Newton step, read straight from sigma.
__global__ void __launch_bounds__(kNT)
score_derivs_kernel(const float2* __restrict__ sigma, int64_t stride, const float* __restrict__ alpha,
                    const float* __restrict__ beta, const float* __restrict__ gamma, int Li,
                    const double* __restrict__ Ctab, const float4* __restrict__ coef, float* __restrict__ out) {
  __shared__ float2 s_ea[1][kNewtonMaxL + 1], s_eg[1][kNewtonMaxL + 1];
  __shared__ double s_phc[1][2 * kNewtonMaxL + 3], s_pt[1][2 * kNewtonMaxL + 3];
  __shared__ uint32_t s_off[kNewtonMaxL + 1];
  __shared__ float s_red[(kNT / 32) * A_N], s_res[A_N];
  __shared__ Point s_now[1];
  const Smem<1> sm{s_ea, s_eg, s_phc, s_pt, s_off, s_red, s_res};
  const int b = blockIdx.x;
  for (int l = threadIdx.x; l <= Li; l += kNT) s_off[l] = 16u * (uint32_t)wedge_off(l);
  if (threadIdx.x == 0) s_now[0] = make_point(alpha[b], beta[b], gamma[b]);
  __syncthreads();
  pass<true, false, 1>(nullptr, sigma + (int64_t)b * stride, coef, Ctab, s_now, Li, sm);
  if (threadIdx.x < A_N) out[(int64_t)b * A_N + threadIdx.x] = sm.res[threadIdx.x];
}

}  // namespace

int newton_eval_launch(const float* sigma, int64_t stride, int B, int Li, const float* alpha, const float* beta,
                       const float* gamma, const double* Ctab, const float4* coef, float* out, cudaStream_t st) {
  MTB_ARG_CHECK(Li >= 0 && Li <= kNewtonMaxL, "degree exceeds the Newton march limit");
  if (B == 0) return MTB_OK;
  mtb_prof_begin(st);
  score_derivs_kernel<<<B, kNT, 0, st>>>(reinterpret_cast<const float2*>(sigma), stride, alpha, beta, gamma, Li,
                                         Ctab, coef, out);
  mtb_prof_end(st, "score_derivs_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}

int64_t newton_fold_entries(int Lmax) { return wedge_off(Lmax + 1); }

int newton_build_coef(int Lmax, float4* coef, cudaStream_t st) {
  MTB_ARG_CHECK(Lmax >= 0 && Lmax <= kNewtonMaxL, "Lmax exceeds the Newton march limit");
  const int64_t n = newton_fold_entries(Lmax);
  const int blocks = (int)((n + 255) / 256);
  coef_kernel<<<blocks, 256, 0, st>>>(n, coef);
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}

int newton_launch(const float* sigma, int64_t stride, int B, int C, float* a, float* b, float* g, float* s,
                  const double* Ctab, const float4* coef, float4* fold, const NewtonParams& P, cudaStream_t st) {
  MTB_ARG_CHECK(P.Lmax >= 0 && P.Lmax <= kNewtonMaxL, "Lmax exceeds the Newton march limit");
  if (P.flags & MTB_SEARCH_COMPAT_TOP_BLOCK) return newton_stencil_launch(sigma, stride, B, C, a, b, g, s, Ctab, P, st);
  const int BC = B * C;
  const float2* sg = reinterpret_cast<const float2*>(sigma);
  const int64_t nf = newton_fold_entries(P.Lmax);
  // two candidates of a subtomogram per CTA share its folded-sigma and recurrence-factor loads,
  // where that still leaves a CTA per SM (16 subtomograms at L = 16: one each 50 us, two 56; 64 at
  // L = 64: one 713, two 509)
  const bool pair = (C % 2) == 0 && BC / 2 >= 148;
  if (fold) {
    mtb_prof_begin(st);
    fold_sigma_kernel<<<dim3(P.Lmax + 1, B), 256, 0, st>>>(sg, stride, nf, fold);
    mtb_prof_end(st, "fold_sigma_kernel");
    MTB_LAUNCH_CHECK();
    mtb_prof_begin(st);
    if (pair)
      newton_march_kernel<true, 2><<<BC / 2, kNT, 0, st>>>(fold, nf, sg, stride, BC, C, a, b, g, s, Ctab, coef, P);
    else
      newton_march_kernel<true, 1><<<BC, kNT, 0, st>>>(fold, nf, sg, stride, BC, C, a, b, g, s, Ctab, coef, P);
  } else {
    mtb_prof_begin(st);
    if (pair)
      newton_march_kernel<false, 2><<<BC / 2, kNT, 0, st>>>(nullptr, nf, sg, stride, BC, C, a, b, g, s, Ctab, coef,
                                                             P);
    else
      newton_march_kernel<false, 1><<<BC, kNT, 0, st>>>(nullptr, nf, sg, stride, BC, C, a, b, g, s, Ctab, coef, P);
  }
  mtb_prof_end(st, "newton_march_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}
