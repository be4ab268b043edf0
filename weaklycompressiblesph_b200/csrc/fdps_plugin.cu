// FDPS multiwalk plugin: wcsph_hydro_dispatch / wcsph_hydro_retrieve and the
// Shepard-filter pair, the drop-in for GPU_WC::HydrDispatchKernel /
// GPU_WC::HydrRetrieveKernel (src/kernel.cu:289-409, src/prototype.h:7-10).
//
// Data path per dispatch (one CUDA stream per tag):
//   host:   gather the FP64 fields of each walk's EPI/EPJ records (byte offsets
//           from wcsph_fdps_layout) into pinned FP32 staging records, with
//           positions taken relative to the walk's first i-particle (so FP32
//           keeps full relative precision; the reference instead scales by
//           L, v0, rho0 into half, src/kernel.cu:317-368).  OpenMP over walks.
//   H2D:    one async copy per chunk of walks, overlapping the packing of the
//           next chunk.
//   device: blocks of 32 i of one walk; the walk's j-records are staged through
//           shared memory in tiles and every i sums over all of them (walk
//           semantics of src/kernel.cu:251-274 and src/force.h:38-55).
//   D2H:    results (FP32 acc, div v, dt) copied back per chunk; retrieve
//           waits on the tag's event and scatters into the caller's RESULT
//           records in FP64.
#include <cuda_runtime.h>
#include <omp.h>
#include <algorithm>
#include <cstdarg>
#include <cstring>
#include <mutex>
#include <vector>

#include "f32x2.cuh"
#include "wcsph_common.cuh"
#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace wcsph {

// ------------------------------------------------------------------ errors
static thread_local std::string g_err;

void set_error(const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
}

int cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
  set_error("CUDA error %d (%s) in %s at %s:%d", (int)e, cudaGetErrorString(e), what, file, line);
  return (e == cudaErrorMemoryAllocation) ? WCSPH_E_NOMEM
         : (e == cudaErrorNoDevice || e == cudaErrorNoKernelImageForDevice || e == cudaErrorInsufficientDriver)
             ? WCSPH_E_NODEVICE
             : WCSPH_E_CUDA;
}

// ---------------------------------------------------------- walk kernels
// Staged records (FP32, 48 B): A = (x, y, z, h) relative to the walk origin,
// B = (vx, vy, vz, rho), C = (P/rho^2, c, nu, m).  i-records use the same
// shape (m unused).  Compact staging (36 B), used for a piece of the batch
// whose records all carry the same h, nu and m (the reference hoists them
// from the first particle, src/kernel.cu:303-304,400-401): A = (x, y, z,
// P/rho^2), B as above, and c alone in the C block; h, nu, m travel in
// WalkPair.  The kernels rebuild the full records, so both stagings give the
// same results bit for bit.
struct WalkPair {
  float alpha, beta, c_cfl, eps;
  int vsig_mode, grad_mode;
  float h, nu, m;  // compact staging: the piece's uniform h, nu, m
};

// Walk kernels.  A walk's j-list is a superset of every one of its i's
// neighbours (a few per cent of the (i, j) combinations are in support), so a
// block takes kWalkChunk i-particles of one walk, stages the j-list tile by
// tile in shared memory, and per tile:
//   scan  - the lanes of a warp hold one i each and test 32 candidates at a
//           time (shared-memory broadcasts, two candidates in packed f32x2
//           arithmetic) against a squared radius that covers every pair of the
//           tile (2 max h), shifting the sign of r^2 - R^2 into a 32-bit mask:
//           no ballots, no queues and no predicates in the loop that sees every
//           combination;
//   pairs - the candidates in the masks are evaluated exactly.
// Every sum runs in a fixed order: results do not depend on the launch.
constexpr int kWalkWarps = 4;
constexpr float kWalkPad = INFINITY;  // coordinates and velocities of a tile's padding
constexpr int kWalkChunk = 32;    // i-particles per block
constexpr int kWalkTile = 512;    // j-records per staged tile (device-resident walks, filter)
constexpr int kWalkWords = kWalkTile / 32 / kWalkWarps;  // mask words per warp and tile

// Records of the walks as the kernels read them: (x, y, z, h), (v, rho),
// (P/rho^2, c, nu, m).  SplitRec: the dispatch staging, full (48 bytes) or
// compact (36); InterleavedRec: three float4 per record.
template <bool COMPACT>
struct SplitRec {
  const float4 *iA, *iB, *iC, *jA, *jB, *jC;
  const float *ic, *jc;  // compact: c alone
  float h, nu, m;
  float4* out4;
  float* out_dt;
  static __device__ __forceinline__ float4 a(const float4* A, int q, float h) {
    float4 r = __ldg(&A[q]);
    if (COMPACT) r.w = h;
    return r;
  }
  __device__ __forceinline__ float4 ia(int i) const { return a(iA, i, h); }
  __device__ __forceinline__ float4 ja(int q) const { return a(jA, q, h); }
  __device__ __forceinline__ float4 ib(int i) const { return __ldg(&iB[i]); }
  __device__ __forceinline__ float4 jb(int q) const { return __ldg(&jB[q]); }
  __device__ __forceinline__ float4 icr(int i) const {
    return COMPACT ? make_float4(__ldg(&iA[i].w), __ldg(&ic[i]), nu, m) : __ldg(&iC[i]);
  }
  __device__ __forceinline__ float4 jcr(int q) const {
    return COMPACT ? make_float4(__ldg(&jA[q].w), __ldg(&jc[q]), nu, m) : __ldg(&jC[q]);
  }
  __device__ __forceinline__ void store(int i, const float4& r, float dt) const {
    out4[i] = r;
    out_dt[i] = dt;
  }
};
struct InterleavedRec {
  const float4 *ei, *ej;
  float4* out;
  __device__ __forceinline__ float4 ia(int i) const { return __ldg(&ei[3 * (size_t)i]); }
  __device__ __forceinline__ float4 ib(int i) const { return __ldg(&ei[3 * (size_t)i + 1]); }
  __device__ __forceinline__ float4 icr(int i) const { return __ldg(&ei[3 * (size_t)i + 2]); }
  __device__ __forceinline__ float4 ja(int q) const { return __ldg(&ej[3 * (size_t)q]); }
  __device__ __forceinline__ float4 jb(int q) const { return __ldg(&ej[3 * (size_t)q + 1]); }
  __device__ __forceinline__ float4 jcr(int q) const { return __ldg(&ej[3 * (size_t)q + 2]); }
  __device__ __forceinline__ void store(int i, const float4& r, float dt) const {
    out[2 * (size_t)i] = r;
    out[2 * (size_t)i + 1] = make_float4(dt, 0.f, 0.f, 0.f);
  }
};

// Gradient factor's h part: 1 / 2h and 16 / (pi (2h)^4).
struct GradH {
  float iH, K;
};
__device__ __forceinline__ GradH grad_h(float h) {
  const float iH = __frcp_rn(2.0f * h);
  return GradH{iH, (float)(16.0 / kPi) * iH * iH * iH * iH};
}
// g(r, h) with gradW = g * dr, rinv = 1 / r.
__device__ __forceinline__ float grad_factor(float r, float rinv, const GradH& G) {
  return spline_F(r * G.iH) * G.K * rinv;
}

// Pair terms of i (records a, b, c; gi = grad_h(h_i)) with j (A, B, C): adds to
// acc = (ax, ay, az, -sum m g dr.dv) as force.h:42-54 / kernel.cu:251-273
// evaluate them (FP32).
template <int GRAD>
__device__ __forceinline__ void walk_pair(const float4& a, const float4& b, const float4& c, const GradH& gi,
                                          const float4& A, const float4& B, const float4& C, const WalkPair& pp,
                                          float acc[4]) {
  const float dx = a.x - A.x, dy = a.y - A.y, dz = a.z - A.z;
  const float r2 = dist2(dx, dy, dz);
  if (!(r2 > 0.0f)) return;
  const float hi = a.w, hj = A.w;
  const float r = sqrtf(r2), rinv = __frcp_rn(r);
  float g;
  if (GRAD == WCSPH_GRAD_SYM) {
    g = r < 2.0f * hi ? grad_factor(r, rinv, gi) : 0.0f;
    if (hj != hi) g = 0.5f * (g + (r < 2.0f * hj ? grad_factor(r, rinv, grad_h(hj)) : 0.0f));
  } else {
    const float hb = 0.5f * (hi + hj);
    g = r < 2.0f * hb ? grad_factor(r, rinv, hj == hi ? gi : grad_h(hb)) : 0.0f;
  }
  if (g == 0.0f) return;  // outside the support every term is zero
  const float dvx = b.x - B.x, dvy = b.y - B.y, dvz = b.z - B.z;
  const float drdv = __fmaf_rn(dz, dvz, __fmaf_rn(dy, dvy, __fmul_rn(dx, dvx)));
  const float iden = __frcp_rn(r2 + pp.eps * hi * hj), irho = __frcp_rn(b.w + B.w);
  const float mu = drdv < 0.0f ? 0.5f * (hi + hj) * drdv * iden : 0.0f;
  const float av = (-pp.alpha * 0.5f * (c.y + C.y) * mu + pp.beta * mu * mu) * 2.0f * irho;
  const float pterm = c.x + C.x + av;
  const float visc = 2.0f * (c.z + C.z) * (g * r2) * irho * iden;
  const float m = C.w;
  acc[0] += m * (visc * dvx - pterm * g * dx);
  acc[1] += m * (visc * dvy - pterm * g * dy);
  acc[2] += m * (visc * dvz - pterm * g * dz);
  acc[3] -= m * g * drdv;
}

// Shared memory of a walk block: a tile of NSOA arrays, the masks and the
// warps' sums.
template <int NSOA, int NRES>
struct alignas(16) WalkSmem {
  float t[NSOA][kWalkTile];
  uint32_t mask[kWalkWarps][kWalkWords][32];
  float res[kWalkWarps][NRES][32];
  unsigned hmax;
};

// The largest smoothing length of the block's i and the tile's j bounds every
// pair of the tile: sets S.hmax (h > 0: its bits order like the values).
template <class Smem>
__device__ __forceinline__ void walk_hmax(Smem& S, float h) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) h = fmaxf(h, __shfl_xor_sync(0xffffffffu, h, o));
  if ((threadIdx.x & 31) == 0) atomicMax(&S.hmax, __float_as_uint(h));
}

// Two candidates' coordinates at u, packed.
__device__ __forceinline__ f2 tile2(const float* t, int u) { return *reinterpret_cast<const f2*>(&t[u]); }

// r^2 of i with the two candidates at u (== dist2 per half), and the mask bits
// of r^2 < R^2 (the sign of r^2 - R^2) shifted into m.
template <int TILE>
__device__ __forceinline__ f2 scan2(const float (*t)[TILE], int u, f2 IX, f2 IY, f2 IZ, f2 NB2, f2& DX, f2& DY, f2& DZ,
                                    uint32_t& m) {
  DX = sub2(IX, tile2(t[0], u)), DY = sub2(IY, tile2(t[1], u)), DZ = sub2(IZ, tile2(t[2], u));
  const f2 R2 = fma2(DZ, DZ, fma2(DY, DY, mul2(DX, DX)));
  const f2 T = add2(R2, NB2);
  m = __funnelshift_l(__float_as_uint(lo(T)), m, 1);
  m = __funnelshift_l(__float_as_uint(hi(T)), m, 1);
  return R2;
}

// Calls body(u) for every candidate in this lane's masks (bit 31 - k of word w
// of this warp of WARPS: candidate 32 (warp + WARPS w) + k), the lanes each at
// their own pace.
template <int WARPS, class Body>
__device__ __forceinline__ void walk_candidates(const uint32_t (*mask)[32], int words, int warp, int lane, Body&& body) {
  uint32_t m = 0;
  int w = 0, base = 0;
  while (true) {
    while (m == 0u && w < words) {
      m = mask[w][lane];
      base = 32 * (warp + WARPS * w);
      ++w;
    }
    if (!__any_sync(0xffffffffu, m != 0u)) break;
    if (m) {
      const int k = __clz(m);
      m ^= 0x80000000u >> k;
      body(base + k);
    }
  }
}

// A power of two near 1 / h^2: numerators carry it, so that the cross products of
// walk_block stay in range whatever the unit of length.
__device__ __forceinline__ float quotient_scale(float h) {
  const int e = (int)(__float_as_uint(h) >> 23);
  return __uint_as_float((unsigned)min(max(3 * 127 - 2 * e, 1), 254) << 23);
}

// Device-resident walks: hydro pair sum of kWalkChunk i-particles [ib, ib + nb)
// of a walk over its j-records [j0, j1) (force.h:38-57; GPU variant
// kernel.cu:241-280 when VSIG / GRAD select it).  The block's warps share the
// words of a tile; a lane evaluates its own i's candidates, the warps' sums
// are added in order.  VSIG: v_sig is max(-mu) over every j of the walk with
// r^2 > 0, in support or not (kernel.cu:263): each lane keeps the numerator and
// denominator of the most negative quotient per half and divides them once at
// the end.  Quotients are compared by their cross products, exactly: n d' < n' d
// as the two products' remainders from the rounded n' d, which fma gives without
// error.  (Rounding is monotone, so the largest quotient rounds to the largest
// rounded one.)
template <int VSIG, int GRAD, class Rec>
__device__ __forceinline__ void walk_block(const Rec& R, int ib, int nb, int j0, int j1, const WalkPair& pp) {
  __shared__ WalkSmem<VSIG ? 8 : 4, 5> S;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = ib + min(lane, nb - 1);
  const float4 a = R.ia(i), b = R.ib(i), c = R.icr(i);
  const GradH gi = grad_h(a.w);
  const f2 IX = dup(a.x), IY = dup(a.y), IZ = dup(a.z);
  const f2 VX = dup(b.x), VY = dup(b.y), VZ = dup(b.z), EH = dup(pp.eps * a.w);
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const float scale = quotient_scale(a.w);
  const f2 SC = dup(scale), IHS = dup(scale * a.w);
  f2 NUM = 0ull, DEN = dup(1.0f);  // the numerator negated
  float vs = 0.0f;
  for (int jb = j0; jb < j1; jb += kWalkTile) {
    const int nt = min(kWalkTile, j1 - jb), nt32 = (nt + 31) & ~31;
    __syncthreads();  // the previous tile's readers are done
    if (threadIdx.x == 0) S.hmax = 0u;
    __syncthreads();
    float h = a.w;
    for (int k = threadIdx.x; k < nt32; k += kWalkWarps * 32) {
      if (k < nt) {
        const float4 J = R.ja(jb + k);
        S.t[0][k] = J.x, S.t[1][k] = J.y, S.t[2][k] = J.z, S.t[3][k] = J.w;
        h = fmaxf(h, J.w);
        if (VSIG) {
          const float4 V = R.jb(jb + k);
          S.t[4][k] = V.x, S.t[5][k] = V.y, S.t[6][k] = V.z, S.t[7][k] = V.w;
        }
      } else {  // padding: never within any bound (inf or NaN), never approaching (drdv = +inf or NaN)
        S.t[0][k] = S.t[1][k] = S.t[2][k] = kWalkPad, S.t[3][k] = 0.0f;
        if (VSIG) S.t[4][k] = S.t[5][k] = S.t[6][k] = kWalkPad, S.t[7][k] = 0.0f;
      }
    }
    walk_hmax(S, h);
    __syncthreads();
    const float Rb = 2.0f * __uint_as_float(S.hmax);
    const f2 NB2 = dup(-(Rb * Rb * 1.0001f));
    int words = 0;
    for (int u0 = 32 * warp; u0 < nt32; u0 += 32 * kWalkWarps, ++words) {
      uint32_t m = 0;
#pragma unroll  // the whole word: 749 us a call for 0.3 M particles, 766 by eight pairs
      for (int u = u0; u < u0 + 32; u += 2) {
        f2 DX, DY, DZ;
        const f2 R2 = scan2(S.t, u, IX, IY, IZ, NB2, DX, DY, DZ, m);
        if (VSIG) {
          const f2 HJ = tile2(S.t[3], u);
          const f2 DV = fma2(DZ, sub2(VZ, tile2(S.t[6], u)), fma2(DY, sub2(VY, tile2(S.t[5], u)),
                                                                   mul2(DX, sub2(VX, tile2(S.t[4], u)))));
          const f2 N = mul2(fma2(HJ, SC, IHS), DV), D = fma2(EH, HJ, R2);  // 2 mu scale = N / D where N < 0
          const f2 P = mul2(NUM, D), X = fma2(N, DEN, P);
          const bool t0 = lo(R2) > 0.0f && lo(X) < __fmaf_rn(-lo(NUM), lo(D), lo(P));
          const bool t1 = hi(R2) > 0.0f && hi(X) < __fmaf_rn(-hi(NUM), hi(D), hi(P));
          NUM = pk(t0 ? -lo(N) : lo(NUM), t1 ? -hi(N) : hi(NUM));
          DEN = pk(t0 ? lo(D) : lo(DEN), t1 ? hi(D) : hi(DEN));
        }
      }
      S.mask[warp][words][lane] = m;
    }
    __syncwarp();
    walk_candidates<kWalkWarps>(S.mask[warp], words, warp, lane, [&](int u) {
      const float4 J = make_float4(S.t[0][u], S.t[1][u], S.t[2][u], S.t[3][u]);
      const float4 V = VSIG ? make_float4(S.t[4][u], S.t[5][u], S.t[6][u], S.t[7][u]) : R.jb(jb + u);
      walk_pair<GRAD>(a, b, c, gi, J, V, R.jcr(jb + u), pp, acc);
    });
  }
  if (VSIG) {
    const float half = 0.5f / scale;
    vs = fmaxf(0.0f, fmaxf(half * lo(NUM) / lo(DEN), half * hi(NUM) / hi(DEN)));
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) S.res[warp][k][lane] = acc[k];
  S.res[warp][4][lane] = vs;
  __syncthreads();
  if (warp == 0 && lane < nb) {
#pragma unroll
    for (int w = 1; w < kWalkWarps; ++w) {
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] += S.res[w][k][lane];
      vs = fmaxf(vs, S.res[w][4][lane]);
    }
    R.store(i, make_float4(acc[0], acc[1], acc[2], acc[3] / b.w), pp.c_cfl * a.w / (c.y + vs));  // force.h:56 / kernel.cu:279
  }
}

__device__ __forceinline__ float grad_factor_split(float r, float h) {  // g(r,h) with gradW = g * dr
  const float H = 2.0f * h;
  const float iH = __frcp_rn(H);
  const float K = (float)(16.0 / kPi) * iH * iH * iH * iH;
  return spline_F(r * iH) * K / r;
}

__device__ __forceinline__ float wq_butterfly8(const float v[8], int lane) {
  const unsigned full = 0xffffffffu;
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
  float w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float send = b4 ? v[k] : v[k + 4];
    const float keep = b4 ? v[k + 4] : v[k];
    w[k] = keep + __shfl_xor_sync(full, send, 16);
  }
  float x[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float send = b3 ? w[k] : w[k + 2];
    const float keep = b3 ? w[k + 2] : w[k];
    x[k] = keep + __shfl_xor_sync(full, send, 8);
  }
  const float send = b2 ? x[0] : x[1];
  float y = (b2 ? x[1] : x[0]) + __shfl_xor_sync(full, send, 4);
  y += __shfl_xor_sync(full, y, 2);
  y += __shfl_xor_sync(full, y, 1);
  return y;  // warp total of slot (lane >> 2) & 7
}

// Pair terms of i (records a, b, c) with j (A, B, C): adds to
// acc = (ax, ay, az, -sum m g dr.dv) as force.h:42-54 / kernel.cu:251-273
// evaluate them (FP32).
template <int GRAD>
__device__ __forceinline__ void walk_pair_split(const float4& a, const float4& b, const float4& c, const float4& A,
                                          const float4& B, const float4& C, const WalkPair& pp, float acc[4]) {
  const float dx = a.x - A.x, dy = a.y - A.y, dz = a.z - A.z;
  const float r2 = dist2(dx, dy, dz);
  const float hi = a.w, hj = A.w;
  const float dvx = b.x - B.x, dvy = b.y - B.y, dvz = b.z - B.z;
  const float drdv = __fmaf_rn(dz, dvz, __fmaf_rn(dy, dvy, __fmul_rn(dx, dvx)));
  const float den = r2 + pp.eps * hi * hj;
  const float mu = drdv < 0.0f ? 0.5f * (hi + hj) * drdv / den : 0.0f;
  const float r = sqrtf(r2);
  float g;
  if (GRAD == WCSPH_GRAD_SYM) {
    g = 0.0f;
    if (r < 2.0f * hi) g += grad_factor_split(r, hi);
    if (r < 2.0f * hj) g += grad_factor_split(r, hj);
    g *= 0.5f;
  } else {
    const float hb = 0.5f * (hi + hj);
    g = (r < 2.0f * hb) ? grad_factor_split(r, hb) : 0.0f;
  }
  if (g == 0.0f) return;  // outside the support every term is zero
  const float rho_sum = b.w + B.w;
  const float av = (-pp.alpha * 0.5f * (c.y + C.y) * mu + pp.beta * mu * mu) * 2.0f / rho_sum;
  const float pterm = c.x + C.x + av;
  const float visc = 2.0f * (c.z + C.z) * (g * r2) / rho_sum / den;
  const float m = C.w;
  acc[0] += m * (visc * dvx - pterm * g * dx);
  acc[1] += m * (visc * dvy - pterm * g * dy);
  acc[2] += m * (visc * dvz - pterm * g * dz);
  acc[3] -= m * g * drdv;
}

// Dispatched walks (FP64 results of FP32 sums; the order of every sum is that
// of the queues below).  Per tile of kSplitTile records the block's warps scan
// all 32 i as above; then a warp takes two i at a time, lays each one's
// candidates out in a queue (lane w the bits of word w), and its lanes evaluate
// queue entries l, l + 32, ..., the lane sums combined by a butterfly
// reduce-scatter.  VSIG: v_sig is max(-mu) over every j of the walk with
// r^2 > 0, in support or not (kernel.cu:263), screened with a fast quotient and
// divided exactly where it can raise a lane's maximum.
// The blocks come from a host-built work list of (walk, first i) ordered by
// decreasing n_i n_j: a tree walk can collect j-lists tens of times the median
// (a group whose Morton run spans distant regions), and those blocks start
// first instead of ending last.
// Bound by the issue of the scan.  A dispatch and retrieve of 0.16 M particles
// took 4.62 ms with lanes along the j-list and ballot-built queues, 3.53 ms so;
// what is left is packing on the host and the copies.
constexpr int kSplitTile = 1024;  // 32 mask words
template <int VSIG>
struct alignas(16) SplitSmem {
  float t[VSIG ? 8 : 4][kSplitTile];  // x, y, z, h and, for the GPU variant's v_sig, vx, vy, vz, rho
  uint32_t mask[32][33];              // word, i
  uint16_t queue[kWalkWarps][2][kSplitTile];
  float res[kWalkChunk][5];           // ax, ay, az, -sum m g dr.dv, v_sig
  unsigned hmax;
};

// Lays the set bits of i's mask words out in q as tile indices; returns their number.
__device__ __forceinline__ int mask_queue(const uint32_t (*mask)[33], int words, int i, uint16_t* q, int lane) {
  uint32_t m = lane < words ? mask[lane][i] : 0u;
  int incl = __popc(m);
  const int own = incl;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const int n = __shfl_sync(0xffffffffu, incl, 31);
  for (int k = incl - own; m; ++k) {
    const int u = __clz(m);
    m ^= 0x80000000u >> u;
    q[k] = (uint16_t)(32 * lane + u);
  }
  return n;
}

template <int VSIG, int GRAD, bool COMPACT>
__global__ void __launch_bounds__(kWalkWarps * 32, 4) k_walk_hydro(SplitRec<COMPACT> R, const int* __restrict__ ni_displ,
                                                                   const int* __restrict__ nj_displ,
                                                                   const int2* __restrict__ items, WalkPair pp) {
  extern __shared__ __align__(16) unsigned char walk_smem[];
  SplitSmem<VSIG>& S = *reinterpret_cast<SplitSmem<VSIG>*>(walk_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int2 item = items[blockIdx.x];  // (walk, first i of this block)
  const int ib = item.y, nb = min(kWalkChunk, ni_displ[item.x + 1] - ib);
  const int j0 = nj_displ[item.x], j1 = nj_displ[item.x + 1];
  for (int t = threadIdx.x; t < kWalkChunk * 5; t += blockDim.x) (&S.res[0][0])[t] = 0.0f;
  const int il = ib + min(lane, nb - 1);  // the scan's i of this lane
  const float4 a = R.ia(il);
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (VSIG) b = R.ib(il);
  const f2 IX = dup(a.x), IY = dup(a.y), IZ = dup(a.z), IH = dup(a.w), EH = dup(pp.eps * a.w);
  const f2 VX = dup(b.x), VY = dup(b.y), VZ = dup(b.z);
  float vs = 0.0f;
  for (int jb = j0; jb < j1; jb += kSplitTile) {
    const int nt = min(kSplitTile, j1 - jb), nt32 = (nt + 31) & ~31;
    __syncthreads();  // the previous tile's readers are done; res zeroed
    if (threadIdx.x == 0) S.hmax = 0u;
    __syncthreads();
    float h = a.w;
    for (int k = threadIdx.x; k < nt32; k += kWalkWarps * 32) {
      if (k < nt) {
        const float4 J = R.ja(jb + k);
        S.t[0][k] = J.x, S.t[1][k] = J.y, S.t[2][k] = J.z, S.t[3][k] = J.w;
        h = fmaxf(h, J.w);
        if (VSIG) {
          const float4 V = R.jb(jb + k);
          S.t[4][k] = V.x, S.t[5][k] = V.y, S.t[6][k] = V.z, S.t[7][k] = V.w;
        }
      } else {  // padding: never within any bound (inf or NaN), never approaching (drdv = +inf or NaN)
        S.t[0][k] = S.t[1][k] = S.t[2][k] = kWalkPad, S.t[3][k] = 0.0f;
        if (VSIG) S.t[4][k] = S.t[5][k] = S.t[6][k] = kWalkPad, S.t[7][k] = 0.0f;
      }
    }
    walk_hmax(S, h);
    __syncthreads();
    // every pair of the tile lies within 2 max h (both variants), with margin
    const float Rb = 2.0f * __uint_as_float(S.hmax);
    const f2 NB2 = dup(-(Rb * Rb * 1.0001f));
    const int words = nt32 >> 5;
    for (int w = warp; w < words; w += kWalkWarps) {
      uint32_t m = 0;
      float near = Rb;
#pragma unroll 8
      for (int u = 32 * w; u < 32 * w + 32; u += 2) {
        f2 DX, DY, DZ;
        const f2 R2 = scan2(S.t, u, IX, IY, IZ, NB2, DX, DY, DZ, m);
        near = fminf(near, fminf(lo(R2), hi(R2)));
        if (VSIG) {
          const f2 HJ = tile2(S.t[3], u);
          const f2 DV = fma2(DZ, sub2(VZ, tile2(S.t[6], u)), fma2(DY, sub2(VY, tile2(S.t[5], u)),
                                                                   mul2(DX, sub2(VX, tile2(S.t[4], u)))));
          const f2 N = mul2(add2(IH, HJ), DV), D = fma2(EH, HJ, R2);  // 2 mu = N / D where N < 0
          const f2 Q = mul2(N, rcp2(D));
          const float bound = -1.999998f * vs;
          if (lo(N) < 0.0f && lo(R2) > 0.0f && !(lo(Q) > bound)) vs = fmaxf(vs, -((0.5f * lo(N)) / lo(D)));
          if (hi(N) < 0.0f && hi(R2) > 0.0f && !(hi(Q) > bound)) vs = fmaxf(vs, -((0.5f * hi(N)) / hi(D)));
        }
      }
      if (near == 0.0f)  // the particle itself (or one on top of it) is no pair
        for (uint32_t b = m; b;) {
          const int k = __clz(b), u = 32 * w + k;
          b ^= 0x80000000u >> k;
          if (!(dist2(a.x - S.t[0][u], a.y - S.t[1][u], a.z - S.t[2][u]) > 0.0f)) m ^= 0x80000000u >> k;
        }
      S.mask[w][lane] = m;
    }
    __syncthreads();
    uint16_t *qa = S.queue[warp][0], *qb = S.queue[warp][1];
    for (int ip = 2 * warp; ip < nb; ip += 2 * kWalkWarps) {
      const bool has_b = ip + 1 < nb;
      const int ia = ib + ip, ibb = has_b ? ia + 1 : ia;
      const int na = mask_queue(S.mask, words, ip, qa, lane);
      const int nq = has_b ? mask_queue(S.mask, words, ip + 1, qb, lane) : 0;
      __syncwarp();
      const float4 Aa = R.ia(ia), Ab = R.ia(ibb), Ba = R.ib(ia), Bb = R.ib(ibb), Ca = R.icr(ia), Cb = R.icr(ibb);
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      const int n = max(na, nq);
      for (int k = lane; k < n; k += 32) {
        if (k < na) {
          const int u = qa[k];
          const float4 J = make_float4(S.t[0][u], S.t[1][u], S.t[2][u], S.t[3][u]);
          const float4 V = VSIG ? make_float4(S.t[4][u], S.t[5][u], S.t[6][u], S.t[7][u]) : R.jb(jb + u);
          walk_pair_split<GRAD>(Aa, Ba, Ca, J, V, R.jcr(jb + u), pp, acc);
        }
        if (k < nq) {
          const int u = qb[k];
          const float4 J = make_float4(S.t[0][u], S.t[1][u], S.t[2][u], S.t[3][u]);
          const float4 V = VSIG ? make_float4(S.t[4][u], S.t[5][u], S.t[6][u], S.t[7][u]) : R.jb(jb + u);
          walk_pair_split<GRAD>(Ab, Bb, Cb, J, V, R.jcr(jb + u), pp, acc + 4);
        }
      }
      const float y = wq_butterfly8(acc, lane);
      if ((lane & 3) == 0) {
        const int slot = lane >> 2;
        if (slot < 4) S.res[ip][slot] += y;
        else if (has_b) S.res[ip + 1][slot - 4] += y;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  if (VSIG && lane < nb) atomicMax(reinterpret_cast<unsigned*>(&S.res[lane][4]), __float_as_uint(vs));  // vs >= 0
  __syncthreads();
  for (int t = threadIdx.x; t < nb; t += blockDim.x) {
    const int i = ib + t;
    const float* r = S.res[t];
    R.store(i, make_float4(r[0], r[1], r[2], r[3] / R.ib(i).w),
            pp.c_cfl * R.ia(i).w / (R.icr(i).y + r[4]));  // force.h:56 / kernel.cu:279
  }
}

// Shepard filter (force.h:12-29): rho_i = sum m W / sum (m/rho_j) W over the
// walk's j-list (which contains i itself).  iA = (x,y,z,h); jA = (x,y,z,m/rho),
// jm = m.  One warp a block: a lane sums its i over the whole list in order
// (candidates beyond the support would add exactly zero), so that its chain of
// additions is that of a loop over every record.  Evaluating the spline for the
// few per cent in support instead of for every record: 5.06 -> 2.41 ms for a
// dispatch and retrieve of 0.16 M particles.
__global__ void __launch_bounds__(32, 24) k_walk_filter(const float4* __restrict__ iA, const float4* __restrict__ jA,
                                                        const float* __restrict__ jm, const int* __restrict__ ni_displ,
                                                        const int* __restrict__ nj_displ, const int2* __restrict__ items,
                                                        float* __restrict__ out_dens) {
  __shared__ alignas(16) float t[3][kWalkTile];
  __shared__ uint32_t mask[kWalkTile / 32][32];
  const int2 item = items[blockIdx.x];
  const int ib = item.y, nb = min(kWalkChunk, ni_displ[item.x + 1] - ib);
  const int j0 = nj_displ[item.x], j1 = nj_displ[item.x + 1];
  const int lane = threadIdx.x;
  const int i = ib + min(lane, nb - 1);
  const float4 a = __ldg(&iA[i]);
  const float H = 2.0f * a.w, iH = __frcp_rn(H);
  const f2 IX = dup(a.x), IY = dup(a.y), IZ = dup(a.z), NB2 = dup(-(H * H * 1.0001f));
  float one = 0.f, sum = 0.f;
  for (int jb = j0; jb < j1; jb += kWalkTile) {
    const int nt = min(kWalkTile, j1 - jb), nt32 = (nt + 31) & ~31;
    __syncwarp();
    bool odd = false;
#pragma unroll 4
    for (int k = lane; k < nt32; k += 32) {
      const float4 J = k < nt ? __ldg(&jA[jb + k]) : make_float4(kWalkPad, kWalkPad, kWalkPad, 0.f);
      t[0][k] = J.x, t[1][k] = J.y, t[2][k] = J.z;
      odd |= !isfinite(J.w) || (k < nt && !isfinite(__ldg(&jm[jb + k])));
    }
    // zero times an infinite or NaN weight is a NaN: such a tile is summed whole
    odd = __any_sync(0xffffffffu, odd);
    const int words = nt32 >> 5;
    for (int w = 0; w < words; ++w) {
      uint32_t m = 0;
#pragma unroll 8
      for (int u = 32 * w; u < 32 * w + 32; u += 2) {
        f2 DX, DY, DZ;
        scan2(t, u, IX, IY, IZ, NB2, DX, DY, DZ, m);
      }
      if (odd) m = nt - 32 * w >= 32 ? 0xffffffffu : ~(0xffffffffu >> (nt - 32 * w));
      mask[w][lane] = m;
    }
    __syncwarp();
    walk_candidates<1>(mask, words, 0, lane, [&](int u) {
      const float dx = a.x - t[0][u], dy = a.y - t[1][u], dz = a.z - t[2][u];
      const float w_ = spline_w(sqrtf(dist2(dx, dy, dz)) * iH);
      one += w_ * __ldg(&jA[jb + u].w);
      sum += w_ * __ldg(&jm[jb + u]);
    });
  }
  if (lane < nb) out_dens[i] = sum / one;  // the normalisation Kw cancels
}

// ------------------------------------------------------------ plugin state
struct PinnedBuf {
  void* p = nullptr;
  size_t bytes = 0;
};
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
};

static int ensure_pinned(PinnedBuf& b, size_t bytes) {
  if (b.bytes >= bytes) return 0;
  const size_t want = std::max(bytes, b.bytes * 3 / 2);
  if (b.p) cudaFreeHost(b.p);
  b.p = nullptr;
  b.bytes = 0;
  WCSPH_CUDA(cudaMallocHost(&b.p, want));
  b.bytes = want;
  return 0;
}
static int ensure_dev(DevBuf& b, size_t bytes) {
  if (b.bytes >= bytes) return 0;
  const size_t want = std::max(bytes, b.bytes * 3 / 2);
  if (b.p) cudaFree(b.p);
  b.p = nullptr;
  b.bytes = 0;
  WCSPH_CUDA(cudaMalloc(&b.p, want));
  b.bytes = want;
  return 0;
}

enum Kind { K_NONE = 0, K_HYDRO = 1, K_FILTER = 2 };

struct TagState {
  cudaStream_t stream = nullptr;
  cudaEvent_t done = nullptr;
  int kind = K_NONE;  // what the last dispatch enqueued
  int n_walk = 0;
  long long ni_total = 0;
  long long h2d_bytes = 0, d2h_bytes = 0;  // of the last dispatch
  int pieces = 0, pieces_compact = 0;
  PinnedBuf h_i, h_j, h_off, h_out;
  DevBuf d_i, d_j, d_off, d_out;
};

struct Plugin {
  bool ready = false;
  int device = -1;
  wcsph_fdps_layout layout{};
  wcsph_pair_params pair{};
  TagState tags[WCSPH_FDPS_MAX_TAGS];
};

static Plugin g_plugin;
static std::mutex g_plugin_mu;

static int plugin_ready() {
  if (g_plugin.ready) return 0;
  if (g_plugin.device < 0) {
    int dev = 0;
    WCSPH_CUDA(cudaGetDevice(&dev));
    g_plugin.device = dev;
  }
  WCSPH_CUDA(cudaSetDevice(g_plugin.device));
  for (auto& t : g_plugin.tags) {
    WCSPH_CUDA(cudaStreamCreateWithFlags(&t.stream, cudaStreamNonBlocking));
    WCSPH_CUDA(cudaEventCreateWithFlags(&t.done, cudaEventDisableTiming));
  }
  g_plugin.ready = true;
  return 0;
}

// Store into the pinned staging buffers.  On x86-64 a streaming store: the
// staging is written once and read only by the copy engine, so the lines are
// not fetched into the cache first (about a fifth less host memory traffic).
static inline void st_stage(float4* dst, float x, float y, float z, float w) {
#if defined(__x86_64__)
  _mm_stream_ps(reinterpret_cast<float*>(dst), _mm_set_ps(w, z, y, x));
#else
  *dst = make_float4(x, y, z, w);
#endif
}
static inline void stage_fence() {
#if defined(__x86_64__)
  _mm_sfence();  // streaming stores are weakly ordered: complete them before the copy reads them
#endif
}

static inline double rd(const void* base, int off) {
  double v;
  memcpy(&v, (const char*)base + off, sizeof(double));
  return v;
}
static inline void wr(void* base, int off, double v) { memcpy((char*)base + off, &v, sizeof(double)); }

constexpr int kChunks = 4;  // walks are staged and copied in this many pieces

}  // namespace wcsph

using namespace wcsph;

extern "C" {

int wcsph_abi_version(void) { return WCSPH_ABI_VERSION; }
const char* wcsph_last_error(void) { return g_err.c_str(); }

void wcsph_fdps_default_layout(wcsph_fdps_layout* o) {
  // src/class.h:61-263 on x86-64 with PS::F64vec = 3 doubles.
  *o = wcsph_fdps_layout{96, 0, 24, 48, 56, 64, 72, 80,       // EPI::Hydro
                         112, 0, 24, 48, 56, 64, 72, 80, 88,  // EPJ::Hydro
                         40, 0, 24, 32,                       // RESULT::Hydro
                         32, 0, 24,                           // EPI::Filter
                         40, 0, 24, 32,                       // EPJ::Filter
                         8, 0};                               // RESULT::Filter
}

void wcsph_pair_params_reference_cpu(wcsph_pair_params* o) {
  *o = wcsph_pair_params{0.01, 0.0, 0.3, 0.01, WCSPH_VSIG_REF_CPU, WCSPH_GRAD_HBAR};
}
void wcsph_pair_params_reference_gpu(wcsph_pair_params* o) {
  *o = wcsph_pair_params{0.01, 0.02, 0.3, 0.01, WCSPH_VSIG_SIGNAL, WCSPH_GRAD_SYM};
}

int wcsph_init(int32_t device) {
  std::lock_guard<std::mutex> lk(g_plugin_mu);
  int n = 0;
  WCSPH_CUDA(cudaGetDeviceCount(&n));
  if (device < 0 || device >= n) {
    set_error("wcsph_init: device %d out of range (%d devices)", device, n);
    return WCSPH_E_INVALID;
  }
  if (g_plugin.ready && g_plugin.device != device) {
    set_error("wcsph_init: plugin already bound to device %d", g_plugin.device);
    return WCSPH_E_STATE;
  }
  g_plugin.device = device;
  return plugin_ready();
}

int wcsph_finalize(void) {
  std::lock_guard<std::mutex> lk(g_plugin_mu);
  if (!g_plugin.ready) return 0;
  cudaSetDevice(g_plugin.device);
  for (auto& t : g_plugin.tags) {
    cudaStreamSynchronize(t.stream);
    for (PinnedBuf* b : {&t.h_i, &t.h_j, &t.h_off, &t.h_out})
      if (b->p) cudaFreeHost(b->p), b->p = nullptr, b->bytes = 0;
    for (DevBuf* b : {&t.d_i, &t.d_j, &t.d_off, &t.d_out})
      if (b->p) cudaFree(b->p), b->p = nullptr, b->bytes = 0;
    cudaEventDestroy(t.done);
    cudaStreamDestroy(t.stream);
    t = TagState{};
  }
  g_plugin.ready = false;
  return 0;
}

}  // extern "C"

namespace wcsph {
// Defaults (class.h layout, kernel.cu pair semantics) are installed once,
// before the first explicit configuration or dispatch, never after.
static bool g_configured_once = false;
static void default_config() {
  if (g_configured_once) return;
  wcsph_fdps_default_layout(&g_plugin.layout);
  wcsph_pair_params_reference_gpu(&g_plugin.pair);
  g_configured_once = true;
}
}  // namespace wcsph

extern "C" {

int wcsph_fdps_configure(const wcsph_fdps_layout* layout, const wcsph_pair_params* params) {
  std::lock_guard<std::mutex> lk(g_plugin_mu);
  default_config();
  if (layout) {
    const wcsph_fdps_layout& L = *layout;
    const int sz[3] = {L.epi_size, L.epj_size, L.res_size};
    if (sz[0] <= 0 || sz[1] <= 0 || sz[2] <= 0) {
      set_error("wcsph_fdps_configure: record sizes must be positive");
      return WCSPH_E_INVALID;
    }
    g_plugin.layout = L;
  }
  if (params) {
    if (params->vsig_mode < 0 || params->vsig_mode > 1 || params->grad_mode < 0 || params->grad_mode > 1) {
      set_error("wcsph_fdps_configure: bad vsig_mode/grad_mode");
      return WCSPH_E_INVALID;
    }
    g_plugin.pair = *params;
  }
  return 0;
}

}  // extern "C"

namespace wcsph {

static int check_walk_args(const char* fn, int32_t tag, int32_t n_walk, const void* const* epi, const int32_t* n_epi,
                           const void* const* epj, const int32_t* n_epj) {
  if (tag < 0 || tag >= WCSPH_FDPS_MAX_TAGS) {
    set_error("%s: tag %d outside [0, %d)", fn, tag, WCSPH_FDPS_MAX_TAGS);
    return WCSPH_E_INVALID;
  }
  if (n_walk < 0 || (n_walk > 0 && (!epi || !n_epi || !epj || !n_epj))) {
    set_error("%s: n_walk %d with null arrays", fn, n_walk);
    return WCSPH_E_INVALID;
  }
  for (int w = 0; w < n_walk; ++w)
    if (n_epi[w] < 0 || n_epj[w] < 0 || (n_epi[w] > 0 && !epi[w]) || (n_epj[w] > 0 && !epj[w])) {
      set_error("%s: walk %d has a negative count or a null record pointer", fn, w);
      return WCSPH_E_INVALID;
    }
  return 0;
}

// Where the hydro records of one dispatch are staged (SoA blocks of the
// pinned buffers) and what one piece of it is packed with.
struct HydroPack {
  const wcsph_fdps_layout* L;
  const void* const* epi;
  const void* const* epj;
  const int32_t* n_epi;
  const int32_t* n_epj;
  const long long* ni_d;
  const long long* nj_d;
  float4 *hiA, *hiB, *hiC, *hjA, *hjB, *hjC;
  bool compact;
  double h0, nu0, m0;  // compact: the piece's uniform values
  float *hic, *hjc;    // compact: c of record q at hic[q] / hjc[q], inside the piece's own part of the C blocks
};

// Origin of walk w: its first i-particle's position (or j when it has no i).
// Staged positions are relative to it.
static void walk_origin(const HydroPack& K, int w, double o[3]) {
  const wcsph_fdps_layout& L = *K.L;
  o[0] = o[1] = o[2] = 0.0;
  if (K.n_epi[w] > 0) {
    for (int k = 0; k < 3; ++k) o[k] = rd(K.epi[w], L.epi_pos + 8 * k);
  } else if (K.n_epj[w] > 0) {
    for (int k = 0; k < 3; ++k) o[k] = rd(K.epj[w], L.epj_pos + 8 * k);
  }
}

// Pack staged records [q0, q1) of one side (i or j) of walks w0.. (the walk
// of q0 found by bisection of the displacements), positions relative to each
// walk's origin org[w - w_first].  Full staging: A = (x, y, z, h),
// B = (v, rho), C = (P/rho^2, c, nu, m).  Compact: A = (x, y, z, P/rho^2), B,
// c alone.  Returns false when a record's h, nu or m differs from the piece's
// (the piece is then packed again in full).  Record-parallel: walks of very
// different sizes (a few carry 40-80x the median j-list) split evenly.
template <bool J>
static bool pack_hydro_range(const HydroPack& K, long long q0, long long q1, int w_first, int w_last,
                             const double* org) {
  const wcsph_fdps_layout& L = *K.L;
  const long long* d = J ? K.nj_d : K.ni_d;
  const void* const* base = J ? K.epj : K.epi;
  const int size = J ? L.epj_size : L.epi_size;
  const int o_pos = J ? L.epj_pos : L.epi_pos, o_vel = J ? L.epj_vel : L.epi_vel, o_dens = J ? L.epj_dens : L.epi_dens,
            o_pres = J ? L.epj_pres : L.epi_pres, o_snds = J ? L.epj_snds : L.epi_snds,
            o_smth = J ? L.epj_smth : L.epi_smth, o_visc = J ? L.epj_visc : L.epi_visc;
  float4* A = J ? K.hjA : K.hiA;
  float4* B = J ? K.hjB : K.hiB;
  float4* C = J ? K.hjC : K.hiC;
  float* c1 = J ? K.hjc : K.hic;
  // the walk holding record q0: last w with d[w] <= q0 (empty walks skipped)
  int lo = w_first, hi = w_last;  // invariant: d[lo] <= q0 < d[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (d[mid] <= q0) lo = mid;
    else hi = mid;
  }
  int w = lo;
  bool uniform = true;
  for (long long q = q0; q < q1; ++q) {
    while (q >= d[w + 1]) ++w;
    const char* r = (const char*)base[w] + (size_t)(q - d[w]) * size;
    const double* o = org + 3 * (w - w_first);
    const double dens = rd(r, o_dens);
    const float po = (float)(rd(r, o_pres) / (dens * dens));
    const float x = (float)(rd(r, o_pos) - o[0]), y = (float)(rd(r, o_pos + 8) - o[1]),
                z = (float)(rd(r, o_pos + 16) - o[2]);
    st_stage(&B[q], (float)rd(r, o_vel), (float)rd(r, o_vel + 8), (float)rd(r, o_vel + 16), (float)dens);
    if (K.compact) {
      uniform &= rd(r, o_smth) == K.h0 && rd(r, o_visc) == K.nu0 && (!J || rd(r, L.epj_mass) == K.m0);
      st_stage(&A[q], x, y, z, po);
      c1[q] = (float)rd(r, o_snds);
    } else {
      st_stage(&A[q], x, y, z, (float)rd(r, o_smth));
      st_stage(&C[q], po, (float)rd(r, o_snds), (float)rd(r, o_visc), J ? (float)rd(r, L.epj_mass) : 0.f);
    }
  }
  stage_fence();
  return uniform;
}

// Pack the i- and j-records of walks [w0, w1) on all host threads, in blocks
// of kPackBlock records.  Returns false when the piece's records are not
// uniform in h, nu and m (compact staging only).
constexpr long long kPackBlock = 2048;
static bool pack_hydro_piece(const HydroPack& K, int w0, int w1) {
  std::vector<double> org(3 * (size_t)(w1 - w0));
#pragma omp parallel for schedule(static)
  for (int w = w0; w < w1; ++w) walk_origin(K, w, &org[3 * (size_t)(w - w0)]);
  const long long a0 = K.ni_d[w0], a1 = K.ni_d[w1], b0 = K.nj_d[w0], b1 = K.nj_d[w1];
  const long long ni_blk = (a1 - a0 + kPackBlock - 1) / kPackBlock, nj_blk = (b1 - b0 + kPackBlock - 1) / kPackBlock;
  int mixed = 0;
#pragma omp parallel for schedule(dynamic, 4) reduction(| : mixed)
  for (long long t = 0; t < ni_blk + nj_blk; ++t) {
    bool u;
    if (t < nj_blk) {
      const long long q0 = b0 + t * kPackBlock;
      u = pack_hydro_range<true>(K, q0, std::min(b1, q0 + kPackBlock), w0, w1, org.data());
    } else {
      const long long q0 = a0 + (t - nj_blk) * kPackBlock;
      u = pack_hydro_range<false>(K, q0, std::min(a1, q0 + kPackBlock), w0, w1, org.data());
    }
    mixed |= u ? 0 : 1;
  }
  return !mixed;
}

template <bool COMPACT>
static int launch_walk_hydro(const SplitRec<COMPACT>& R, unsigned nblk, cudaStream_t s, const int* d_ni,
                              const int* d_nj, const int2* items, const WalkPair& pp) {
  auto kern = pp.vsig_mode ? (pp.grad_mode ? k_walk_hydro<1, 1, COMPACT> : k_walk_hydro<1, 0, COMPACT>)
                           : (pp.grad_mode ? k_walk_hydro<0, 1, COMPACT> : k_walk_hydro<0, 0, COMPACT>);
  const int smem = (int)(pp.vsig_mode ? sizeof(SplitSmem<1>) : sizeof(SplitSmem<0>));
  WCSPH_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  kern<<<nblk, kWalkWarps * 32, smem, s>>>(R, d_ni, d_nj, items, pp);
  WCSPH_CUDA(cudaGetLastError());
  return 0;
}

// Shared dispatch body.  kind selects the record shapes and the kernel.
static int dispatch_common(int kind, int32_t tag, int32_t n_walk, const void* const* epi, const int32_t* n_epi,
                           const void* const* epj, const int32_t* n_epj) {
  const char* fn = kind == K_HYDRO ? "wcsph_hydro_dispatch" : "wcsph_filter_dispatch";
  default_config();
  if (int rc = check_walk_args(fn, tag, n_walk, epi, n_epi, epj, n_epj)) return rc;
  if (int rc = plugin_ready()) return rc;
  WCSPH_CUDA(cudaSetDevice(g_plugin.device));
  TagState& T = g_plugin.tags[tag];
  WCSPH_CUDA(cudaStreamSynchronize(T.stream));  // the tag's previous batch owns the buffers until done
  const wcsph_fdps_layout& L = g_plugin.layout;

  // Displacements (src/kernel.cu:306-310), 64-bit so huge batches cannot wrap.
  std::vector<long long> ni_d(n_walk + 1), nj_d(n_walk + 1);
  ni_d[0] = nj_d[0] = 0;
  for (int w = 0; w < n_walk; ++w) {
    ni_d[w + 1] = ni_d[w] + n_epi[w];
    nj_d[w + 1] = nj_d[w] + n_epj[w];
  }
  const long long NI = ni_d[n_walk], NJ = nj_d[n_walk];
  if (NI > INT32_MAX || NJ > INT32_MAX) {
    set_error("%s: %lld i / %lld j records exceed the 2^31 limit of one batch", fn, NI, NJ);
    return WCSPH_E_CAPACITY;
  }
  const size_t i_rec = kind == K_HYDRO ? 3 * sizeof(float4) : sizeof(float4);
  const size_t j_rec = kind == K_HYDRO ? 3 * sizeof(float4) : sizeof(float4) + sizeof(float);
  const size_t o_rec = kind == K_HYDRO ? sizeof(float4) + sizeof(float) : sizeof(float);
  if (int rc = ensure_pinned(T.h_i, i_rec * (NI + 1))) return rc;
  if (int rc = ensure_pinned(T.h_j, j_rec * (NJ + 1))) return rc;
  // Work list of the kernels: (walk, first i) per block of kWalkChunk i.
  long long n_items = 0;
  for (int w = 0; w < n_walk; ++w) n_items += (n_epi[w] + kWalkChunk - 1) / kWalkChunk;
  const size_t off_bytes = sizeof(int) * 2 * (n_walk + 1) + sizeof(int2) * (size_t)n_items;
  if (int rc = ensure_pinned(T.h_off, off_bytes)) return rc;
  if (int rc = ensure_pinned(T.h_out, o_rec * (NI + 1))) return rc;
  if (int rc = ensure_dev(T.d_i, i_rec * (NI + 1))) return rc;
  if (int rc = ensure_dev(T.d_j, j_rec * (NJ + 1))) return rc;
  if (int rc = ensure_dev(T.d_off, off_bytes)) return rc;
  if (int rc = ensure_dev(T.d_out, o_rec * (NI + 1))) return rc;

  int* h_ni = (int*)T.h_off.p;
  int* h_nj = h_ni + (n_walk + 1);
  for (int w = 0; w <= n_walk; ++w) {
    h_ni[w] = (int)ni_d[w];
    h_nj[w] = (int)nj_d[w];
  }
  int* d_ni = (int*)T.d_off.p;
  int* d_nj = d_ni + (n_walk + 1);
  const int chunks = n_walk < kChunks * 64 ? 1 : kChunks;
  // Per dispatch chunk, its blocks in decreasing order of work n_i n_j (ties
  // by position, so the list is reproducible; the order never changes a result).
  int2* h_items = reinterpret_cast<int2*>(h_nj + (n_walk + 1));
  std::vector<long long> item_off(chunks + 1, 0);
  {
    std::vector<std::pair<long long, long long>> key;  // (-work, position)
    long long pos = 0;
    for (int ch = 0; ch < chunks; ++ch) {
      const int w0 = (int)((long long)n_walk * ch / chunks), w1 = (int)((long long)n_walk * (ch + 1) / chunks);
      key.clear();
      std::vector<int2> its;
      for (int w = w0; w < w1; ++w)
        for (int i = 0; i < n_epi[w]; i += kWalkChunk) {
          const long long work = (long long)std::min(kWalkChunk, n_epi[w] - i) * std::max(1, n_epj[w]);
          key.emplace_back(-work, (long long)its.size());
          its.push_back(make_int2(w, (int)(ni_d[w] + i)));
        }
      std::sort(key.begin(), key.end());
      for (const auto& k : key) h_items[pos++] = its[k.second];
      item_off[ch + 1] = pos;
    }
  }
  WCSPH_CUDA(cudaMemcpyAsync(d_ni, h_ni, off_bytes, cudaMemcpyHostToDevice, T.stream));
  T.h2d_bytes = (long long)off_bytes;
  T.d2h_bytes = 0;
  T.pieces = T.pieces_compact = 0;
  const int2* d_items = reinterpret_cast<const int2*>(d_nj + (n_walk + 1));

  // SoA sub-arrays inside the staging buffers.
  float4* hiA = (float4*)T.h_i.p;
  float4* hiB = hiA + NI;
  float4* hiC = hiB + NI;
  float4* hjA = (float4*)T.h_j.p;
  float4* hjB = hjA + NJ;
  float4* hjC = hjB + NJ;
  float* hjm = (float*)(hjA + NJ);  // filter: m after the A block
  float4* diA = (float4*)T.d_i.p;
  float4* djA = (float4*)T.d_j.p;

  for (int ch = 0; ch < chunks; ++ch) {
    const int w0 = (int)((long long)n_walk * ch / chunks), w1 = (int)((long long)n_walk * (ch + 1) / chunks);
    if (w0 == w1) continue;
    bool compact = false;
    WalkPair pp{(float)g_plugin.pair.alpha, (float)g_plugin.pair.beta, (float)g_plugin.pair.c_cfl,
                (float)g_plugin.pair.eps, g_plugin.pair.vsig_mode, g_plugin.pair.grad_mode, 0.f, 0.f, 0.f};
    if (kind == K_HYDRO) {
      // A compact piece keeps c of record q at float 3 a0 + q of the C block:
      // bytes [16 a0, 16 a0 + 4 (a1 - a0)), inside the piece's own part
      // [16 a0, 16 a1) (the copies of earlier pieces may still be reading
      // theirs).
      HydroPack K{&L, epi, epj, n_epi, n_epj, ni_d.data(), nj_d.data(), hiA, hiB, hiC, hjA, hjB, hjC, false, 0, 0, 0,
                  reinterpret_cast<float*>(hiC) + 3 * ni_d[w0], reinterpret_cast<float*>(hjC) + 3 * nj_d[w0]};
      // Compact staging when every record of the piece carries the h, nu and
      // m of its first j-record (checked while packing).
      for (int w = w0; w < w1 && !K.compact; ++w)
        if (n_epj[w] > 0) {
          const char* r = (const char*)epj[w];
          K.compact = true;
          K.h0 = rd(r, L.epj_smth), K.nu0 = rd(r, L.epj_visc), K.m0 = rd(r, L.epj_mass);
        }
      if (!pack_hydro_piece(K, w0, w1) && K.compact) {
        K.compact = false;
        pack_hydro_piece(K, w0, w1);
      }
      compact = K.compact;
      if (compact) pp.h = (float)K.h0, pp.nu = (float)K.nu0, pp.m = (float)K.m0;
      ++T.pieces;
      T.pieces_compact += compact ? 1 : 0;
    } else {
#pragma omp parallel for schedule(dynamic, 16)
      for (int w = w0; w < w1; ++w) {
        const char* pi = (const char*)epi[w];
        const char* pj = (const char*)epj[w];
        double o[3] = {0, 0, 0};
        if (n_epi[w] > 0) {
          for (int k = 0; k < 3; ++k) o[k] = rd(pi, L.fepi_pos + 8 * k);
        } else if (n_epj[w] > 0) {
          for (int k = 0; k < 3; ++k) o[k] = rd(pj, L.fepj_pos + 8 * k);
        }
        for (int i = 0; i < n_epi[w]; ++i) {
          const char* r = pi + (size_t)i * L.fepi_size;
          hiA[ni_d[w] + i] = make_float4((float)(rd(r, L.fepi_pos) - o[0]), (float)(rd(r, L.fepi_pos + 8) - o[1]),
                                         (float)(rd(r, L.fepi_pos + 16) - o[2]), (float)rd(r, L.fepi_smth));
        }
        for (int j = 0; j < n_epj[w]; ++j) {
          const char* r = pj + (size_t)j * L.fepj_size;
          const double m = rd(r, L.fepj_mass);
          hjA[nj_d[w] + j] = make_float4((float)(rd(r, L.fepj_pos) - o[0]), (float)(rd(r, L.fepj_pos + 8) - o[1]),
                                         (float)(rd(r, L.fepj_pos + 16) - o[2]), (float)(m / rd(r, L.fepj_dens)));
          hjm[nj_d[w] + j] = (float)m;
        }
      }
    }
    // H2D of this chunk's records (SoA blocks copied piecewise).
    const long long a0 = ni_d[w0], a1 = ni_d[w1], b0 = nj_d[w0], b1 = nj_d[w1];
    // the third block carries full float4 records, or only c (compact staging,
    // at the start of the piece's part of the block)
    auto h2d = [&](void* dst, const void* src, size_t bytes) -> int {
      if (bytes == 0) return 0;
      WCSPH_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, T.stream));
      T.h2d_bytes += (long long)bytes;
      return 0;
    };
    int rc = 0;
    if (kind == K_HYDRO) {
      if (a1 > a0) {
        rc |= h2d(diA + a0, hiA + a0, sizeof(float4) * (a1 - a0));
        rc |= h2d(diA + NI + a0, hiB + a0, sizeof(float4) * (a1 - a0));
        rc |= h2d(diA + 2 * NI + a0, hiC + a0, (compact ? sizeof(float) : sizeof(float4)) * (a1 - a0));
      }
      if (b1 > b0) {
        rc |= h2d(djA + b0, hjA + b0, sizeof(float4) * (b1 - b0));
        rc |= h2d(djA + NJ + b0, hjB + b0, sizeof(float4) * (b1 - b0));
        rc |= h2d(djA + 2 * NJ + b0, hjC + b0, (compact ? sizeof(float) : sizeof(float4)) * (b1 - b0));
      }
    } else {
      if (a1 > a0) rc |= h2d(diA + a0, hiA + a0, sizeof(float4) * (a1 - a0));
      if (b1 > b0) {
        rc |= h2d(djA + b0, hjA + b0, sizeof(float4) * (b1 - b0));
        rc |= h2d((float*)(djA + NJ) + b0, hjm + b0, sizeof(float) * (b1 - b0));
      }
    }
    if (rc) return rc;
    const unsigned nblk = (unsigned)(item_off[ch + 1] - item_off[ch]);
    const int2* items = d_items + item_off[ch];
    if (kind == K_HYDRO) {
      float4* out4 = (float4*)T.d_out.p;
      float* out_dt = (float*)(out4 + NI);
      const float* ic = reinterpret_cast<const float*>(diA + 2 * NI) + 3 * a0;
      const float* jc = reinterpret_cast<const float*>(djA + 2 * NJ) + 3 * b0;
      if (nblk > 0) {
        rc = compact ? launch_walk_hydro(SplitRec<true>{diA, diA + NI, nullptr, djA, djA + NJ, nullptr, ic, jc, pp.h,
                                                        pp.nu, pp.m, out4, out_dt},
                                         nblk, T.stream, d_ni, d_nj, items, pp)
                     : launch_walk_hydro(SplitRec<false>{diA, diA + NI, diA + 2 * NI, djA, djA + NJ, djA + 2 * NJ,
                                                         nullptr, nullptr, 0.f, 0.f, 0.f, out4, out_dt},
                                         nblk, T.stream, d_ni, d_nj, items, pp);
        if (rc) return rc;
      }
      if (a1 > a0) {
        WCSPH_CUDA(cudaMemcpyAsync((float4*)T.h_out.p + a0, out4 + a0, sizeof(float4) * (a1 - a0),
                                   cudaMemcpyDeviceToHost, T.stream));
        WCSPH_CUDA(cudaMemcpyAsync((float*)((float4*)T.h_out.p + NI) + a0, out_dt + a0, sizeof(float) * (a1 - a0),
                                   cudaMemcpyDeviceToHost, T.stream));
        T.d2h_bytes += (long long)(sizeof(float4) + sizeof(float)) * (a1 - a0);
      }
    } else {
      float* out = (float*)T.d_out.p;
      if (nblk > 0) {
        k_walk_filter<<<nblk, 32, 0, T.stream>>>(diA, djA, (const float*)(djA + NJ), d_ni, d_nj, items, out);
        WCSPH_CUDA(cudaGetLastError());
      }
      if (a1 > a0) {
        WCSPH_CUDA(cudaMemcpyAsync((float*)T.h_out.p + a0, out + a0, sizeof(float) * (a1 - a0), cudaMemcpyDeviceToHost,
                                   T.stream));
        T.d2h_bytes += (long long)sizeof(float) * (a1 - a0);
      }
    }
  }
  WCSPH_CUDA(cudaEventRecord(T.done, T.stream));
  T.kind = kind;
  T.n_walk = n_walk;
  T.ni_total = NI;
  return 0;
}

static int retrieve_common(int kind, int32_t tag, int32_t n_walk, const int32_t* n_i, void* const* force) {
  const char* fn = kind == K_HYDRO ? "wcsph_hydro_retrieve" : "wcsph_filter_retrieve";
  if (tag < 0 || tag >= WCSPH_FDPS_MAX_TAGS) {
    set_error("%s: tag %d outside [0, %d)", fn, tag, WCSPH_FDPS_MAX_TAGS);
    return WCSPH_E_INVALID;
  }
  TagState& T = g_plugin.tags[tag];
  if (!g_plugin.ready || T.kind != kind) {
    set_error("%s: no pending dispatch of this kind for tag %d", fn, tag);
    return WCSPH_E_STATE;
  }
  if (n_walk != T.n_walk || (n_walk > 0 && (!n_i || !force))) {
    set_error("%s: n_walk %d does not match the dispatch (%d) or null arrays", fn, n_walk, T.n_walk);
    return WCSPH_E_INVALID;
  }
  std::vector<long long> off(n_walk + 1);
  off[0] = 0;
  for (int w = 0; w < n_walk; ++w) off[w + 1] = off[w] + n_i[w];
  if (off[n_walk] != T.ni_total) {
    set_error("%s: %lld i-particles requested, %lld dispatched", fn, off[n_walk], T.ni_total);
    return WCSPH_E_INVALID;
  }
  WCSPH_CUDA(cudaEventSynchronize(T.done));
  const wcsph_fdps_layout& L = g_plugin.layout;
  const long long NI = T.ni_total;
  if (kind == K_HYDRO) {
    const float4* o4 = (const float4*)T.h_out.p;
    const float* odt = (const float*)(o4 + NI);
#pragma omp parallel for schedule(dynamic, 64)
    for (int w = 0; w < n_walk; ++w) {
      char* base = (char*)force[w];
      for (int i = 0; i < n_i[w]; ++i) {
        const float4 a = o4[off[w] + i];
        char* r = base + (size_t)i * L.res_size;
        wr(r, L.res_acc, a.x);
        wr(r, L.res_acc + 8, a.y);
        wr(r, L.res_acc + 16, a.z);
        wr(r, L.res_div_v, a.w);
        wr(r, L.res_dt, odt[off[w] + i]);
      }
    }
  } else {
    const float* od = (const float*)T.h_out.p;
#pragma omp parallel for schedule(dynamic, 64)
    for (int w = 0; w < n_walk; ++w) {
      char* base = (char*)force[w];
      for (int i = 0; i < n_i[w]; ++i) wr(base + (size_t)i * L.fres_size, L.fres_dens, od[off[w] + i]);
    }
  }
  T.kind = K_NONE;
  return 0;
}
}  // namespace wcsph

extern "C" {
int wcsph_hydro_dispatch(int32_t tag, int32_t n_walk, const void* const* epi, const int32_t* n_epi,
                         const void* const* epj, const int32_t* n_epj) {
  std::lock_guard<std::mutex> lk(g_plugin_mu);
  return dispatch_common(K_HYDRO, tag, n_walk, epi, n_epi, epj, n_epj);
}
int wcsph_hydro_retrieve(int32_t tag, int32_t n_walk, const int32_t* n_i, void* const* force) {
  std::lock_guard<std::mutex> lk(g_plugin_mu);
  return retrieve_common(K_HYDRO, tag, n_walk, n_i, force);
}
int wcsph_filter_dispatch(int32_t tag, int32_t n_walk, const void* const* epi, const int32_t* n_epi,
                          const void* const* epj, const int32_t* n_epj) {
  std::lock_guard<std::mutex> lk(g_plugin_mu);
  return dispatch_common(K_FILTER, tag, n_walk, epi, n_epi, epj, n_epj);
}
int wcsph_filter_retrieve(int32_t tag, int32_t n_walk, const int32_t* n_i, void* const* result) {
  std::lock_guard<std::mutex> lk(g_plugin_mu);
  return retrieve_common(K_FILTER, tag, n_walk, n_i, result);
}
int wcsph_fdps_stats(int32_t tag, int64_t* out4) {
  if (tag < 0 || tag >= WCSPH_FDPS_MAX_TAGS || !out4) {
    set_error("wcsph_fdps_stats: bad tag %d or null output", tag);
    return WCSPH_E_INVALID;
  }
  std::lock_guard<std::mutex> lk(g_plugin_mu);
  const TagState& T = g_plugin.tags[tag];
  out4[0] = T.h2d_bytes;
  out4[1] = T.d2h_bytes;
  out4[2] = T.pieces_compact;
  out4[3] = T.pieces;
  return 0;
}
}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free walk pair sum.
//
// For callers that cannot allocate device memory: hosts that hand the plugin a
// fixed memory budget and forbid growth, embedders whose allocator owns every
// device byte, and host loops in which a cudaMalloc would synchronise the
// device in the middle of a step.  The caller passes device-resident inputs
// and outputs; the only scratch this path needs, the per-walk displacement
// tables (exclusive prefix sums of the walk sizes), lives in the file-scope
// array below, sized for WCSPH_NOALLOC_MAX_WALKS walks (about 512 KB, held on
// every GPU that loads the library until the process exits).
namespace wcsph {

static __device__ __align__(256) int g_noalloc_displ[2 * (WCSPH_NOALLOC_MAX_WALKS + 1)];

// Exclusive prefix sums of the two count arrays into g_noalloc_displ-shaped
// scratch: displ[0..n] for i-counts, displ[n+1 .. 2n+1] for j-counts.  One
// block; every entry it later reads is written, so nothing needs clearing.
__global__ void __launch_bounds__(1024) k_noalloc_displ(int n, const int* __restrict__ n_epi,
                                                       const int* __restrict__ n_epj, int* displ) {
  __shared__ int warp_tot[2][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n + 1023) / 1024;
  const int b = min(n, tid * per), e = min(n, b + per);
  int si = 0, sj = 0;
  for (int k = b; k < e; ++k) {
    si += n_epi[k];
    sj += n_epj[k];
  }
  int ii = si, ij = sj;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ti = __shfl_up_sync(0xffffffffu, ii, o), tj = __shfl_up_sync(0xffffffffu, ij, o);
    if (lane >= o) ii += ti, ij += tj;
  }
  if (lane == 31) warp_tot[0][warp] = ii, warp_tot[1][warp] = ij;
  __syncthreads();
  if (warp == 0) {
    int wi = warp_tot[0][lane], wj = warp_tot[1][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ti = __shfl_up_sync(0xffffffffu, wi, o), tj = __shfl_up_sync(0xffffffffu, wj, o);
      if (lane >= o) wi += ti, wj += tj;
    }
    warp_tot[0][lane] = wi;
    warp_tot[1][lane] = wj;
  }
  __syncthreads();
  int oi = ii - si + (warp > 0 ? warp_tot[0][warp - 1] : 0);
  int oj = ij - sj + (warp > 0 ? warp_tot[1][warp - 1] : 0);
  for (int k = b; k < e; ++k) {
    displ[k] = oi;
    displ[n + 1 + k] = oj;
    oi += n_epi[k];
    oj += n_epj[k];
  }
  if (tid == 1023) {
    displ[n] = oi;
    displ[2 * n + 1] = oj;
  }
}

// The walk pair sum of k_walk_hydro with records interleaved per particle
// (three float4 per record) and results as two float4 per i-particle.  The walk
// sizes are on the device, so that the host knows no work list: kNoallocSplit
// blocks a walk take its chunks of kWalkChunk i in turn (FDPS's Ngroup = 128,
// param.h:9, gives each one).  Against one thread per i that evaluated every
// record, one block a walk: 7.73 -> 0.75 ms for 0.3 M particles, 0.68 -> 0.06 ms
// for 5,000.
constexpr int kNoallocSplit = 4;
template <int VSIG, int GRAD>
__global__ void __launch_bounds__(kWalkWarps * 32, 5) k_walk_hydro_interleaved(InterleavedRec R,
                                                                               const int* __restrict__ displ,
                                                                               int n_walk, WalkPair pp) {
  const int w = blockIdx.x / kNoallocSplit;
  const int i0 = displ[w], i1 = displ[w + 1];
  const int j0 = displ[n_walk + 1 + w], j1 = displ[n_walk + 2 + w];
  for (int ib = i0 + kWalkChunk * (blockIdx.x % kNoallocSplit); ib < i1; ib += kWalkChunk * kNoallocSplit) {
    walk_block<VSIG, GRAD>(R, ib, min(kWalkChunk, i1 - ib), j0, j1, pp);
    __syncthreads();  // the chunk's sums are read before the next one's are written
  }
}

// Device address of the scratch array, looked up once per device.
static int* g_noalloc_ptr[64];
static std::mutex g_noalloc_mu;

static int noalloc_scratch(int** out) {
  int dev = 0;
  WCSPH_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("wcsph_hydro_walks_noalloc: device ordinal %d is beyond the supported 64", dev);
    return WCSPH_E_NODEVICE;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_displ);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_displ)", __FILE__, __LINE__);
    g_noalloc_ptr[dev] = (int*)p;
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}

}  // namespace wcsph

extern "C" int wcsph_hydro_walks_noalloc(int32_t n_walk, const int32_t* d_n_epi, const int32_t* d_n_epj,
                                         const void* d_epi, const void* d_epj, void* d_out,
                                         const wcsph_pair_params* params, void* stream) {
  if (n_walk < 0 || !params) {
    set_error("wcsph_hydro_walks_noalloc: n_walk %d < 0 or null params", n_walk);
    return WCSPH_E_INVALID;
  }
  if (n_walk > WCSPH_NOALLOC_MAX_WALKS) {
    set_error("wcsph_hydro_walks_noalloc: %d walks exceed the allocation-free limit of %d walks per call", n_walk,
              WCSPH_NOALLOC_MAX_WALKS);
    return WCSPH_E_CAPACITY;
  }
  if (params->vsig_mode < 0 || params->vsig_mode > 1 || params->grad_mode < 0 || params->grad_mode > 1) {
    set_error("wcsph_hydro_walks_noalloc: bad vsig_mode/grad_mode");
    return WCSPH_E_INVALID;
  }
  if (n_walk == 0) return 0;
  if (!d_n_epi || !d_n_epj || !d_epi || !d_epj || !d_out) {
    set_error("wcsph_hydro_walks_noalloc: null device pointer");
    return WCSPH_E_INVALID;
  }
  int* displ = nullptr;
  if (int rc = noalloc_scratch(&displ)) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  k_noalloc_displ<<<1, 1024, 0, s>>>(n_walk, d_n_epi, d_n_epj, displ);
  const WalkPair pp{(float)params->alpha, (float)params->beta, (float)params->c_cfl, (float)params->eps,
                    params->vsig_mode, params->grad_mode};
  auto kern = pp.vsig_mode ? (pp.grad_mode ? k_walk_hydro_interleaved<1, 1> : k_walk_hydro_interleaved<1, 0>)
                           : (pp.grad_mode ? k_walk_hydro_interleaved<0, 1> : k_walk_hydro_interleaved<0, 0>);
  kern<<<n_walk * kNoallocSplit, kWalkWarps * 32, 0, s>>>(
      InterleavedRec{(const float4*)d_epi, (const float4*)d_epj, (float4*)d_out}, displ, n_walk, pp);
  WCSPH_CUDA(cudaGetLastError());
  return 0;
}
