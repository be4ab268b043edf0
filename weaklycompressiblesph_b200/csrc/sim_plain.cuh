// Density and hydro passes of the plain FP32 path and the density pass of the
// other searching passes: every particle's neighbours in the order of the cell
// search (for_each_neighbor), summed one after the other by the particle's lane.
//
// One warp per non-empty cell, up to 32 of its particles at a time.  The
// candidates of the 27 neighbour cells are staged in shared memory with all that
// a pair needs when they lie within the support radius of the batch's bounding
// box; every lane tests 32 of them at a time into a bit mask (packed f32x2, the
// sign of r^2 - H^2), and evaluates the pairs of its masks.  The additions and
// their order are those of a loop over every candidate, so that the block shape
// and the staging never change a bit.
//
// Against one thread per particle that walks the 27 cells itself (k_hydro_particle,
// kept for large solvers with few particles a cell: thread_per_particle), a step's
// hydro pass: dam break of 12,600 particles 163 -> 39 us, of 54,500 186 -> 76,
// of 477,000 559 -> 468, of 1.25 M 1395 -> 1250; cells of 83 particles (8,100 in
// all) 492 -> 340.  Density pass of a lattice of 64,000: 149 -> 81 us.
// Small solvers are bound by the instructions of one cell's warp (9,000, at six
// cycles each), large ones by the same stream at 14 warps an SM.  Two candidates'
// terms are evaluated side by side in packed arithmetic (477,000 particles: one
// at a time 570 us, two scalar streams 523, packed 492, before the tile was cut
// to 384).  Four warps a batch that rank the candidates and share the terms
// through shared memory are no faster for small solvers and slower for large
// (943 us).
#pragma once
#include "sim_scan.cuh"

namespace wcsph {

enum PlainPass { PLAIN_HYDRO, PLAIN_DENSITY };

constexpr int kBatches = 2;  // blocks that share a cell's batches (hydro pass; most density launches have nothing to do)
constexpr int kPlainTile = 384;  // candidates (hydro pass, 477,000 particles: 468 us; 448: 504; 320: 440, but lattices lose)
constexpr int kStage = 2;  // groups of 32 candidates whose loads are in flight together

// Shared memory of a warp.
template <int PASS>
struct alignas(16) PlainTile {
  float pos[3][kPlainTile];                                // shifted by the periodic image
  float4 b[PASS == PLAIN_HYDRO ? kPlainTile : 1];          // v, rho
  float2 pc[PASS == PLAIN_HYDRO ? kPlainTile : 1];         // P / rho^2, c
  float rho[PASS == PLAIN_DENSITY ? kPlainTile : 1];
  uint32_t mask[kPlainTile / 32][32];
};

// Operands of pair_terms for the lane's particle and its instance: packed
// duplicates (the factors carry signs, which are exact).
struct PlainI {
  f2 X, Y, Z, VX, VY, VZ, RHO, PO, CI;
  f2 NIH, NKG, EH2, H, BETA, NAH, NNU4;  // -1/2h, -Kg, eps h^2, h, beta, -alpha/2, -4 nu
};
// The terms of two pairs, one per half (force.h:38-57 for uniform h, m, nu): NG
// is minus the gradient factor.  Which products are fused into an fma is written
// out here, and again one pair at a time in k_hydro_particle: the two agree to the
// bit.
struct PairTerms {
  f2 R2, X, Y, Z, NG, DRDV, MU;
};
__device__ __forceinline__ PairTerms pair_terms(const PlainI& I, const PlainTile<PLAIN_HYDRO>& S, int u0, int u1) {
  PairTerms t;
  const f2 DX = sub2(I.X, pk(S.pos[0][u0], S.pos[0][u1])), DY = sub2(I.Y, pk(S.pos[1][u0], S.pos[1][u1])),
           DZ = sub2(I.Z, pk(S.pos[2][u0], S.pos[2][u1]));
  t.R2 = fma2(DZ, DZ, fma2(DY, DY, mul2(DX, DX)));  // == dist2 per half
  const float4 B0 = S.b[u0], B1 = S.b[u1];
  const float2 p0 = S.pc[u0], p1 = S.pc[u1];
  const f2 RINV = rsqrt2(t.R2), Q = mul2(t.R2, RINV);
  const f2 A = max0_2(fma2(Q, I.NIH, dup(1.0f))), B = max0_2(fma2(Q, I.NIH, dup(0.5f)));
  const f2 F = fma2(mul2(dup(12.0f), B), B, mul2(mul2(dup(-3.0f), A), A));
  t.NG = mul2(mul2(F, I.NKG), RINV);
  const f2 DVX = sub2(I.VX, pk(B0.x, B1.x)), DVY = sub2(I.VY, pk(B0.y, B1.y)), DVZ = sub2(I.VZ, pk(B0.z, B1.z));
  t.DRDV = fma2(DZ, DVZ, fma2(DX, DVX, mul2(DY, DVY)));
  const f2 D = add2(t.R2, I.EH2), R = add2(I.RHO, pk(B0.w, B1.w));
  const f2 RDEN = pk(__frcp_rn(lo(D)), __frcp_rn(hi(D))), RS = pk(__frcp_rn(lo(R)), __frcp_rn(hi(R)));
  const f2 MUr = mul2(mul2(I.H, t.DRDV), RDEN);
  t.MU = pk(lo(t.DRDV) < 0.0f ? lo(MUr) : 0.0f, hi(t.DRDV) < 0.0f ? hi(MUr) : 0.0f);
  const f2 AV = mul2(mul2(fma2(I.BETA, t.MU, mul2(I.NAH, add2(I.CI, pk(p0.y, p1.y)))), t.MU), dup(2.0f));
  const f2 NPG = mul2(fma2(AV, RS, add2(I.PO, pk(p0.x, p1.x))), t.NG);
  const f2 VISC = mul2(mul2(mul2(mul2(I.NNU4, t.NG), t.R2), RS), RDEN);
  t.X = fma2(VISC, DVX, mul2(NPG, DX));
  t.Y = fma2(VISC, DVY, mul2(NPG, DY));
  t.Z = fma2(VISC, DVZ, mul2(NPG, DZ));
  return t;
}
__device__ __forceinline__ bool density_term(const float4& I, int u, const PlainTile<PLAIN_DENSITY>& S, float iH,
                                             float& w) {
  const float r2 = dist2(__fsub_rn(I.x, S.pos[0][u]), __fsub_rn(I.y, S.pos[1][u]), __fsub_rn(I.z, S.pos[2][u]));
  w = spline_w(sqrtf(r2) * iH);
  return r2 > 0.0f;
}

template <int PASS>
__device__ __forceinline__ void cell_pass(const StepArgs& a, PlainTile<PASS>& S) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x;
  const unsigned lt = lanemask_lt();
  float *tx = S.pos[0], *ty = S.pos[1], *tz = S.pos[2];
  const int nrun = *a.run_count;
  const int ox = lane % 3 - 1, oy = (lane / 3) % 3 - 1, oz = lane / 9 - 1;  // neighbour cell of lane < 27
  unsigned long long pairs = 0;
  for (int k = blockIdx.x; k < nrun; k += gridDim.x) {
    const int lin = a.run_list[k];
    const int s = a.cell_start[lin], e = a.cell_end[lin];
    if (s + 32 * (int)blockIdx.y >= e) continue;  // blockIdx.y: every gridDim.y-th batch of a cell
    const int inst = a.alt.flags[s] & kInstMask;
    const InstParams& P = a.params[inst];
    const int ph = a.phase[inst];
    const int kind = PASS == PLAIN_DENSITY ? density_kind(a, P, a.dyn[inst], ph) : 0;
    if (PASS == PLAIN_DENSITY ? !kind : !wants_force(P, a.dyn[inst], ph)) {
      if (PASS == PLAIN_HYDRO)
        for (int p = s + 32 * blockIdx.y + lane; p < e; p += 32 * gridDim.y) copy_state(a, p);
      continue;
    }
    const int nx = P.ncell[0], ny = P.ncell[1];
    const int local = lin - P.cell_base;
    const int cx = local % nx, cy = (local / nx) % ny, cz = local / (nx * ny);

    // the neighbour cells, one per lane, and the runs they form
    int start = 0, end = 0;
    float shx = 0.f, shy = 0.f, shz = 0.f;
    if (lane < 27) {
      int x, y, z;
      if (neighbor_cell(P, 0, cx + ox, x, shx) && neighbor_cell(P, 1, cy + oy, y, shy) &&
          neighbor_cell(P, 2, cz + oz, z, shz)) {
        const int l2 = P.cell_base + (z * ny + y) * nx + x;
        start = a.cell_start[l2];
        end = a.cell_end[l2];
      }
    }
    const unsigned some = __ballot_sync(full, end > start);  // non-empty cells
    const unsigned before = some & lt;
    const int prev = before ? 31 - __clz(before) : 0;
    const int prev_end = __shfl_sync(full, end, prev);
    const float px = __shfl_sync(full, shx, prev), py = __shfl_sync(full, shy, prev), pz = __shfl_sync(full, shz, prev);
    const bool head =
        end > start && (!before || prev_end != start || px != shx || py != shy || pz != shz);
    const unsigned heads = __ballot_sync(full, head);
    const unsigned later = lane < 31 ? heads >> (lane + 1) : 0u;
    const int next_head = later ? lane + __ffs(later) : 32;  // first lane of the next run
    const unsigned upto = next_head < 32 ? some & ((1u << next_head) - 1u) : some;
    const int run_end = __shfl_sync(full, end, upto ? 31 - __clz(upto) : 0);
    // candidate k of the search lies in the run of the last head whose first <= k, at slot k + its delta
    int first = head ? run_end - start : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(full, first, o);
      if (lane >= o) first += t;
    }
    const int total = __shfl_sync(full, first, 31);
    if (head) first -= run_end - start;  // lanes that head no run: first of the run after theirs
    const int delta = start - first;
    const float H2 = P.H2, cull = H2 * kCullMargin, iH = P.inv_H;
    const f2 NH2 = dup(-H2);
    const int vs = P.vsig_mode;
    const bool shep = kind == 2;

    for (int ib = s + 32 * blockIdx.y; ib < e; ib += 32 * gridDim.y) {
      const int p = ib + lane;
      const bool mine = p < e;
      float4 I = make_float4(kFarLane, kFarLane, kFarLane, 0.f), IB = make_float4(0.f, 0.f, 0.f, 1.f);
      float ci = 0.f;
      if (mine) {
        I = a.jr[p].a;
        IB = a.jr[p].b;
        if (PASS == PLAIN_HYDRO) ci = a.jC[p];
      }
      const float big = __int_as_float(0x7f800000);
      const float bx0 = warp_min_f(mine ? I.x : big), bx1 = warp_max_f(mine ? I.x : -big);
      const float by0 = warp_min_f(mine ? I.y : big), by1 = warp_max_f(mine ? I.y : -big);
      const float bz0 = warp_min_f(mine ? I.z : big), bz1 = warp_max_f(mine ? I.z : -big);
      const f2 IX = dup(I.x), IY = dup(I.y), IZ = dup(I.z);
      const float rho_i = IB.w;
      PlainI i2;
      if (PASS == PLAIN_HYDRO) {
        i2.X = IX, i2.Y = IY, i2.Z = IZ, i2.VX = dup(IB.x), i2.VY = dup(IB.y), i2.VZ = dup(IB.z);
        i2.RHO = dup(IB.w), i2.PO = dup(I.w), i2.CI = dup(ci);
        i2.NIH = dup(-iH), i2.NKG = dup(-P.Kg), i2.EH2 = dup(P.eh2), i2.H = dup(P.h);
        i2.BETA = dup(P.beta), i2.NAH = dup(-(P.alpha * 0.5f)), i2.NNU4 = dup(-P.nu4);
      }
      float ax = 0.f, ay = 0.f, az = 0.f, ndsum = -0.f, vsig = 0.f;
      float sum = 0.5f, one = 0.5f / rho_i;  // self term: w(0) = 1/2
      unsigned cnt = 0;

      int k0 = 0;  // candidates staged or culled so far
      do {
        int tn = 0;  // staged candidates
        for (; k0 < total && tn + 32 * kStage <= kPlainTile; k0 += 32 * kStage) {
          float4 J[kStage], B[kStage];
          float c[kStage], sx[kStage], sy[kStage], sz[kStage];
#pragma unroll
          for (int r = 0; r < kStage; ++r) {
            const int k = k0 + 32 * r + lane;
            int run = 0;  // the last lane with first <= k: the run's head
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
              if (__shfl_sync(full, first, run + o) <= k) run += o;
            const int q = k + __shfl_sync(full, delta, run);
            sx[r] = __shfl_sync(full, shx, run), sy[r] = __shfl_sync(full, shy, run), sz[r] = __shfl_sync(full, shz, run);
            if (k < total) {
              J[r] = __ldg(&a.jr[q].a);
              if (PASS == PLAIN_HYDRO || shep) B[r] = __ldg(&a.jr[q].b);
              if (PASS == PLAIN_HYDRO) c[r] = __ldg(&a.jC[q]);
            }
          }
#pragma unroll
          for (int r = 0; r < kStage; ++r) {
            const float x = __fadd_rn(J[r].x, sx[r]), y = __fadd_rn(J[r].y, sy[r]), z = __fadd_rn(J[r].z, sz[r]);
            const float dx = fmaxf(fmaxf(bx0 - x, x - bx1), 0.f), dy = fmaxf(fmaxf(by0 - y, y - by1), 0.f),
                        dz = fmaxf(fmaxf(bz0 - z, z - bz1), 0.f);
            const bool in = k0 + 32 * r + lane < total && dx * dx + dy * dy + dz * dz < cull;
            const unsigned keep = __ballot_sync(full, in);
            if (in) {
              const int u = tn + __popc(keep & lt);
              tx[u] = x, ty[u] = y, tz[u] = z;
              if (PASS == PLAIN_HYDRO) S.b[u] = B[r], S.pc[u] = make_float2(J[r].w, c[r]);
              else if (shep) S.rho[u] = B[r].w;
            }
            tn += __popc(keep);
          }
        }
        const int tn32 = (tn + 31) & ~31;
        if (tn + lane < tn32) tx[tn + lane] = kFarTile, ty[tn + lane] = kFarTile, tz[tn + lane] = kFarTile;
        __syncwarp();
        int n = 0;  // this lane's candidates
        for (int u0 = 0; u0 < tn32; u0 += 32) {
          uint32_t m = 0;
#pragma unroll
          for (int u = 0; u < 32; u += 4) {
            const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(&tx[u0 + u]);
            const ulonglong2 Y = *reinterpret_cast<const ulonglong2*>(&ty[u0 + u]);
            const ulonglong2 Z = *reinterpret_cast<const ulonglong2*>(&tz[u0 + u]);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const f2 DX = sub2(IX, k ? X.y : X.x), DY = sub2(IY, k ? Y.y : Y.x), DZ = sub2(IZ, k ? Z.y : Z.x);
              const f2 T = add2(fma2(DZ, DZ, fma2(DY, DY, mul2(DX, DX))), NH2);  // negative exactly when r^2 < H^2
              m = __funnelshift_l(__float_as_uint(lo(T)), m, 1);
              m = __funnelshift_l(__float_as_uint(hi(T)), m, 1);
            }
          }
          S.mask[u0 >> 5][lane] = m;
          n += __popc(m);
        }
        const int nmax = __reduce_max_sync(full, n);
        uint32_t m = 0;
        int w = -1;
        auto next = [&]() {  // the lane's next candidate
          while (!m) m = S.mask[++w][lane];
          const int bit = __clz(m);
          m ^= 0x80000000u >> bit;
          return 32 * w + bit;
        };
        // two candidates' terms, then their additions in order
        for (int k = 0; k < nmax; k += 2) {
          if (k >= n) continue;
          const int u0 = next(), u1 = k + 1 < n ? next() : -1;
          if constexpr (PASS == PLAIN_DENSITY) {
            float w0 = 0.f, w1 = 0.f;
            const bool b0 = density_term(I, u0, S, iH, w0), b1 = u1 >= 0 && density_term(I, u1, S, iH, w1);
            if (b0) {
              sum += w0;
              if (shep) one += w0 / S.rho[u0];
            }
            if (b1) {
              sum += w1;
              if (shep) one += w1 / S.rho[u1];
            }
          } else {
            const PairTerms t = pair_terms(i2, S, u0, max(u1, 0));
            if (lo(t.R2) > 0.0f) {  // not the particle itself, nor any at its very place
              ++cnt;
              ax += lo(t.X), ay += lo(t.Y), az += lo(t.Z);
              ndsum = __fmaf_rn(lo(t.NG), lo(t.DRDV), ndsum);
              vsig = fmaxf(vsig, vs ? -lo(t.MU) : lo(t.MU));
            }
            if (u1 >= 0 && hi(t.R2) > 0.0f) {
              ++cnt;
              ax += hi(t.X), ay += hi(t.Y), az += hi(t.Z);
              ndsum = __fmaf_rn(hi(t.NG), hi(t.DRDV), ndsum);
              vsig = fmaxf(vsig, vs ? -hi(t.MU) : hi(t.MU));
            }
          }
        }
        __syncwarp();
      } while (k0 < total);
      if (PASS == PLAIN_DENSITY) {
        if (mine) a.rho_new[p] = shep ? sum / one : P.mass * P.Kw * sum;
      } else {
        float dt_cand = 0.0f;
        bool dt_valid = false;
        if (mine) {
          const uint32_t f = a.alt.flags[p];
          finish_hydro(a, p, P, inst, ph, f, ax, ay, az, -ndsum, vsig, cnt, dt_cand, dt_valid);
          if (!(f & kGhostBit)) pairs += cnt;  // pairs are counted for owned particles only
        }
        dt_min(a.dyn, inst, dt_cand, dt_valid);
      }
    }
  }
  if (PASS == PLAIN_HYDRO) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(full, pairs, o);
    if (lane == 0 && pairs) atomicAdd(a.pair_count, pairs);
  }
}

// Hydro pass (the plain FP32 path).  Restates force.h:38-57 for uniform h, m,
// nu within an instance:
//   a_i  = m sum_j [ -(P_i/rho_i^2 + P_j/rho_j^2 + Pi_ij) g + 4 nu g r^2 / ((rho_i+rho_j)(r^2+eps h^2)) dv ] ...
// with gradW = g dr; div v_i = -m/rho_i sum_j g (dr.dv); dt_i = C h / (c_i + v_sig).
// The epilogue adds gravity (Dam2.h:104-108), does the final kick
// (class.h:160-163), the density floor (Dam2.h:111), and folds the CFL limits
// of integral.h:2-12 into the instance's next dt.
__global__ void __launch_bounds__(32, 14) k_hydro_plain(const __grid_constant__ StepArgs a) {
  __shared__ PlainTile<PLAIN_HYDRO> S;
  cell_pass<PLAIN_HYDRO>(a, S);
  copy_dead(a);
}

// Summation rho_i = m sum_j W_ij (self included) or the Shepard filter of
// force.h:12-29, sum m W / sum (m/rho_j) W, from the pre-filter densities.
__global__ void __launch_bounds__(32, 12) k_density_plain(const __grid_constant__ StepArgs a) {
  if (a.dens_any && !*a.dens_any) return;  // no density pass in this launch
  __shared__ PlainTile<PLAIN_DENSITY> S;
  cell_pass<PLAIN_DENSITY>(a, S);
}

// The same passes with one thread per particle that walks the 27 cells itself:
// candidates are read from the caches, a warp's lanes diverge, but nothing is
// paid per cell.  Every term and addition is that of the cell passes, to the bit.
__global__ void __launch_bounds__(256) k_density_particle(const __grid_constant__ StepArgs a) {
  if (a.dens_any && !*a.dens_any) return;  // no density pass in this launch
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= *a.n_alive) return;
  const int inst = a.alt.flags[p] & kInstMask;
  const InstParams& P = a.params[inst];
  const int kind = density_kind(a, P, a.dyn[inst], a.phase[inst]);
  if (kind) search_density(a, P, p, kind);
}

__global__ void __launch_bounds__(256) k_hydro_particle(const __grid_constant__ StepArgs a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  int inst = 0;
  float dt_cand = 0.0f;
  bool dt_valid = false;
  unsigned cnt = 0;
  if (p < *a.n_alive) {
    const uint32_t f = a.alt.flags[p];
    inst = f & kInstMask;
    const InstParams& P = a.params[inst];
    const int ph = a.phase[inst];
    if (wants_force(P, a.dyn[inst], ph)) {
      const float4 I = a.jr[p].a, IB = a.jr[p].b;
      const float ci = a.jC[p];
      float ax = 0.f, ay = 0.f, az = 0.f, ndsum = -0.f, vsig = 0.f;
      const float nih = -P.inv_H, nkg = -P.Kg, eh2 = P.eh2, h = P.h, beta = P.beta, nah = -(P.alpha * 0.5f), nnu4 = -P.nu4;
      const int vs = P.vsig_mode;
      for_each_neighbor(a, P, I.x, I.y, I.z, [&](int q, const float4& J, float dx, float dy, float dz, float r2, uint32_t) {
        ++cnt;
        const float4 B = __ldg(&a.jr[q].b);
        const float cj = __ldg(&a.jC[q]);
        // pair_terms, operation by operation
        const float rinv = rsqrtf(r2), s = __fmul_rn(r2, rinv);
        const float A1 = fmaxf(__fmaf_rn(s, nih, 1.0f), 0.0f), B1 = fmaxf(__fmaf_rn(s, nih, 0.5f), 0.0f);
        const float F = __fmaf_rn(__fmul_rn(12.0f, B1), B1, __fmul_rn(__fmul_rn(-3.0f, A1), A1));
        const float ng = __fmul_rn(__fmul_rn(F, nkg), rinv);
        const float dvx = __fsub_rn(IB.x, B.x), dvy = __fsub_rn(IB.y, B.y), dvz = __fsub_rn(IB.z, B.z);
        const float drdv = __fmaf_rn(dz, dvz, __fmaf_rn(dx, dvx, __fmul_rn(dy, dvy)));
        const float rden = __frcp_rn(__fadd_rn(r2, eh2)), rs = __frcp_rn(__fadd_rn(IB.w, B.w));
        const float mu = drdv < 0.0f ? __fmul_rn(__fmul_rn(h, drdv), rden) : 0.0f;
        const float av = __fmul_rn(__fmul_rn(__fmaf_rn(beta, mu, __fmul_rn(nah, __fadd_rn(ci, cj))), mu), 2.0f);
        const float npg = __fmul_rn(__fmaf_rn(av, rs, __fadd_rn(I.w, J.w)), ng);
        const float visc = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(nnu4, ng), r2), rs), rden);
        ax = __fadd_rn(ax, __fmaf_rn(visc, dvx, __fmul_rn(npg, dx)));
        ay = __fadd_rn(ay, __fmaf_rn(visc, dvy, __fmul_rn(npg, dy)));
        az = __fadd_rn(az, __fmaf_rn(visc, dvz, __fmul_rn(npg, dz)));
        ndsum = __fmaf_rn(ng, drdv, ndsum);
        vsig = fmaxf(vsig, vs ? -mu : mu);
      });
      finish_hydro(a, p, P, inst, ph, f, ax, ay, az, -ndsum, vsig, cnt, dt_cand, dt_valid);
      if (f & kGhostBit) cnt = 0;  // pairs are counted for owned particles only
    } else {
      copy_state(a, p);
    }
  } else if (p < a.n_host) {
    copy_state(a, p);  // the dead tail
  }
  dt_min(a.dyn, inst, dt_cand, dt_valid);
  unsigned long long pairs = cnt;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
  if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(a.pair_count, pairs);
}

// Which of the two for n particles with `load` of them in a full cell (the cell's
// volume over a particle's, m / rho0).  A cell costs a warp 2 ns + 0.9 ns a particle
// of GPU time (hydro, large solvers), a thread's walk 0.3 ns + 0.07 ns x load, but at
// least 35 us + 8 us x load from end to end.  Hydro pass, us, cell / particle, by load
// 1.4, 4.5, 6, 9, 11, 14.5, 19 on jittered lattices:
//   64,000     159/46   92/80   92/86    79/113   84/128   82/161   88/197
//   125,000    300/52  180/111 153/111  136/136  144/172  151/221  160/258
//   512,000   1207/158 685/312 622/328  528/368  557/499  599/674  548/773
//   1,728,000 4329/465 2368/972 2083/1019 1829/1086 1883/1552 1966/2122 1946/2408
// Density pass:
//   64,000     105/45   69/77   70/81    62/96    73/108   73/129   75/154
//   512,000    738/112 453/207 428/210  384/218  406/290  425/372  385/433
//   1,728,000 2534/297 1527/590 1404/593 1273/590 1324/828 1376/1075 1348/1212
inline bool thread_per_particle(int pass, int n, float load) {
  return pass == PLAIN_HYDRO ? load <= 12.0f && n >= 12000.0f * load : load <= 16.0f + n / 4.0e5f && n >= 19000.0f * load;
}

template <int PASS>
inline int launch_plain(const StepArgs& a, int n, float load, cudaStream_t s) {
  if (thread_per_particle(PASS, n, load)) {
    auto kern = PASS == PLAIN_HYDRO ? k_hydro_particle : k_density_particle;
    kern<<<(n + 255) / 256, 256, 0, s>>>(a);
    WCSPH_CUDA(cudaGetLastError());
    return 0;
  }
  static TiledLaunch L[16];
  int dev = 0;
  WCSPH_CUDA(cudaGetDevice(&dev));
  TiledLaunch& T = L[dev & 15];
  auto kern = PASS == PLAIN_HYDRO ? k_hydro_plain : k_density_plain;
  if (T.device != dev) {
    int per_sm = 0, sms = 0;
    WCSPH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32, 0));
    WCSPH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    T.blocks = std::max(1, per_sm) * sms;
    T.device = dev;
  }
  kern<<<dim3(std::min(T.blocks, n), PASS == PLAIN_HYDRO ? kBatches : 1), 32, 0, s>>>(a);
  WCSPH_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace wcsph
