// Neighbour-list build: the scan that writes every particle's list row.
//
// One warp per non-empty cell, up to 32 of its particles at a time (lane l
// holds particle l of the batch):
//   1. The 27 neighbour cells are taken in the order of the cell search
//      (for_each_neighbor).  Of three cells along x two are neighbours in the
//      Morton order too, so that their particles are one run of slots: 18 runs
//      instead of 27 ranges.  The runs are laid end to end and read 64 candidates
//      at a time, each lane finding its candidate's run by bisection, so that
//      loads are full whatever a cell holds (run by run, short runs wait for one
//      another: cells of 2 particles 973 us a build, 414 so, of 6 328 and 248, of
//      18 and more the same; 512,000 particles).
//   2. A candidate is staged into the warp's shared-memory tile (SoA: x, y, z
//      shifted by the periodic image, and its list entry) only when it lies
//      within the list radius of the bounding box of the batch: about half
//      of the 27 cells' particles do (729 -> 370 on a lattice with cells of
//      2.3 h).
//   3. Every lane tests 32 staged candidates at a time against its own
//      particle (shared-memory broadcasts, packed f32x2 distances).  The sign
//      of r^2 - R^2 is shifted into a 32-bit mask: no predicates and no
//      divergent stores in the inner loop.
//   4. Every lane turns its masks into tile indices (in the shared memory of
//      the positions, which are done with) and writes its row from them in
//      16-byte groups of entries.
// The rows hold the candidates in the order of the cell search, whatever the
// block shape.
//
// Measured on a dam break under way (1.6M particles, 147M entries): 0.72-0.76 ms
// a build, 1.244 ms with a lane per particle walking all 27 cells' candidates
// and storing single words (32 separate sectors a store); periodic lattice of
// 1M: 0.625 against 0.942 ms; half2 lists of 0.5M: 0.322 against 0.429 ms.
// Bound by issue and latency: 54 % of the issue slots with 18 warps an SM, the
// L1 data pipe (shared memory) at 68 %.
#pragma once
#include "sim_tiled.cuh"

namespace wcsph {

constexpr float kFarAway = 1.0e30f;   // position of removed particles in the j-records
constexpr float kFarTile = -1.0e30f;  // padding of a tile: within no list radius of anything
constexpr float kFarLane = 3.0e30f;   // idle lanes of a warp

// Shared memory of one warp (10.9 KB: 20 warps an SM).  The row buffer (16-bit
// tile indices, one row a lane) takes the place of the positions once they are
// tested.  Most cells fill one tile and one row buffer (384 candidates and 64
// indices: 25 warps an SM but 1.27 times the instructions, 0.826 ms; 512 and
// 128: 16 warps, 0.846 ms).
constexpr int kScanTile = 448;  // candidates
struct alignas(16) ScanTile {
  static constexpr int kBuf = 112;  // indices per row
  union {
    float pos[3][kScanTile];
    uint16_t buf[32][kBuf + 2];  // + 2: the rows start in different banks
  };
  uint32_t e[kScanTile];
  uint32_t mask[kScanTile / 32][32];  // 32 candidates a word
};

// Low two bits of a particle's cell coordinates, one nibble per axis, as
// k_permute leaves them in x0[p].w (half2 entries name the neighbour cell).
__device__ __forceinline__ uint32_t cell_nibbles(int cx, int cy, int cz) {
  return (uint32_t)(cx & 3) | ((uint32_t)(cy & 3) << 4) | ((uint32_t)(cz & 3) << 8);
}

template <bool H16, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 20 / WARPS) k_list_scan(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const unsigned full = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ScanTile& S = reinterpret_cast<ScanTile*>(smem_raw)[warp];
  float *tx = S.pos[0], *ty = S.pos[1], *tz = S.pos[2];
  uint32_t* te = S.e;
  const unsigned lt = lanemask_lt();
  const int nrun = *a.run_count;
  const int L = a.list_max;
  const int ox = lane % 3 - 1, oy = (lane / 3) % 3 - 1, oz = lane / 9 - 1;  // neighbour cell of lane < 27
  const bool partial = a.inst_keep && a.list_flags[kLfPartial] != 0u;
  int longest = 0;
  const int stride = gridDim.x * WARPS;
  int c = blockIdx.x * WARPS + warp;
  int lin_next = c < nrun ? a.run_list[c] : 0;
  for (; c < nrun; c += stride) {
    const int lin = lin_next;
    if (c + stride < nrun) lin_next = a.run_list[c + stride];
    const int s = a.cell_start[lin], e = a.cell_end[lin];
    const int inst = a.alt.flags[s] & kInstMask;
    if (partial && a.inst_keep[inst]) continue;  // keeps its lists
    const InstParams& P = a.params[inst];
    // every active instance, idle or finished as it may be in this pass: the sort
    // has moved its particles, and later probes and steps read its rows
    if (!P.active) {
      for (int p = s + lane; p < e; p += 32) a.list_cnt[p] = 0;
      continue;
    }
    const int nx = P.ncell[0], ny = P.ncell[1];
    const int local = lin - P.cell_base;
    const int cx = local % nx, cy = (local / nx) % ny, cz = local / (nx * ny);

    // the neighbour cells, one per lane, and the runs they form
    int start = 0, end = 0;
    float shx = 0.f, shy = 0.f, shz = 0.f;
    uint32_t image = 13;
    if (lane < 27) {
      int x, y, z;
      if (neighbor_cell(P, 0, cx + ox, x, shx) && neighbor_cell(P, 1, cy + oy, y, shy) &&
          neighbor_cell(P, 2, cz + oz, z, shz)) {
        const int l2 = P.cell_base + (z * ny + y) * nx + x;
        start = a.cell_start[l2];
        end = a.cell_end[l2];
        image = (uint32_t)((shx > 0.f) - (shx < 0.f) + 1) + 3u * (uint32_t)((shy > 0.f) - (shy < 0.f) + 1) +
                9u * (uint32_t)((shz > 0.f) - (shz < 0.f) + 1);
      }
    }
    const unsigned some = __ballot_sync(full, end > start);  // non-empty cells
    const unsigned before = some & lt;
    const int prev = before ? 31 - __clz(before) : 0;
    const int prev_end = __shfl_sync(full, end, prev);
    const uint32_t prev_image = __shfl_sync(full, image, prev);
    const bool head = end > start && (!before || prev_end != start || prev_image != image);
    const unsigned heads = __ballot_sync(full, head);
    const unsigned later = lane < 31 ? heads >> (lane + 1) : 0u;
    const int next_head = later ? lane + __ffs(later) : 32;  // first lane of the next run
    const unsigned upto = next_head < 32 ? some & ((1u << next_head) - 1u) : some;
    const int run_end = __shfl_sync(full, end, upto ? 31 - __clz(upto) : 0);
    // candidate k of the search lies in the run of the last lane with first <= k, at slot k + its delta
    int first = head ? run_end - start : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(full, first, o);
      if (lane >= o) first += t;
    }
    const int total = __shfl_sync(full, first, 31);
    if (head) first -= run_end - start;  // lanes that head no run: first of the run after theirs
    const int delta = start - first;
    const int own_delta = __shfl_sync(full, delta, 31 - __clz(heads & 0x3fffu));  // of the run of the cell itself (lane 13)
    uint32_t meta = image;
    if (H16) {  // an axis on which the run wraps has one offset; elsewhere the cells' low bits give it
      meta |= ((shx != 0.f ? 0x003u : 0u) | (shy != 0.f ? 0x030u : 0u) | (shz != 0.f ? 0x300u : 0u)) << 5;
      meta |= ((shx > 0.f ? 0x002u : 0u) | (shy > 0.f ? 0x020u : 0u) | (shz > 0.f ? 0x200u : 0u)) << 15;
    }
    const uint32_t ci = cell_nibbles(cx, cy, cz);
    const float R2 = P.HL2, cull = P.HL2 * kCullMargin;
    const uint32_t hb = __float_as_uint(R2) - 1u;
    const f2 NR2 = dup(-R2);

    for (int ib = s; ib < e; ib += 32) {
      const int nbat = min(32, e - ib);
      const bool mine = lane < nbat;
      float4 I = make_float4(kFarLane, kFarLane, kFarLane, 0.f);
      if (mine) I = __ldg(&a.jr[ib + lane].a);
      // bounding box of the batch's live particles
      const bool live = mine && I.x < kFarAway;
      const float big = __int_as_float(0x7f800000);
      const float bx0 = warp_min_f(live ? I.x : big), bx1 = warp_max_f(live ? I.x : -big);
      const float by0 = warp_min_f(live ? I.y : big), by1 = warp_max_f(live ? I.y : -big);
      const float bz0 = warp_min_f(live ? I.z : big), bz1 = warp_max_f(live ? I.z : -big);
      const f2 IX = dup(I.x), IY = dup(I.y), IZ = dup(I.z);
      uint4* row = list_row(a, mine ? ib + lane : s);
      auto put = [&](int k, uint32_t ent) { reinterpret_cast<uint32_t*>(row + 32 * (k >> 2))[k & 3] = ent; };
      int len = 0;  // entries of this lane's row

      int k0 = 0;  // candidates staged or culled so far
      do {
        int tn = 0;                       // staged candidates
        int own0 = kScanTile, own1 = 0;   // tile indices that hold the cell's own particles
        for (; k0 < total && tn + 64 <= kScanTile; k0 += 64) {
          float4 J[2];
          uint32_t cj[2], mt[2];
          int qs[2];
          float sx[2], sy[2], sz[2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int k = k0 + 32 * r + lane;
            int run = 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
              if (__shfl_sync(full, first, run + o) <= k) run += o;
            qs[r] = k + __shfl_sync(full, delta, run);
            mt[r] = __shfl_sync(full, meta, run);
            sx[r] = __shfl_sync(full, shx, run), sy[r] = __shfl_sync(full, shy, run), sz[r] = __shfl_sync(full, shz, run);
            if (k < total) {
              J[r] = __ldg(&a.jr[qs[r]].a);
              if (H16) cj[r] = __float_as_uint(__ldg(&a.x0[qs[r]].w));
            }
          }
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int kr = k0 + 32 * r;
            const float x = __fadd_rn(J[r].x, sx[r]), y = __fadd_rn(J[r].y, sy[r]), z = __fadd_rn(J[r].z, sz[r]);
            const float dx = fmaxf(fmaxf(bx0 - x, x - bx1), 0.f), dy = fmaxf(fmaxf(by0 - y, y - by1), 0.f),
                        dz = fmaxf(fmaxf(bz0 - z, z - bz1), 0.f);
            const bool in = kr + lane < total && dx * dx + dy * dy + dz * dz < cull;
            const unsigned keep = __ballot_sync(full, in);
            if (in) {
              uint32_t ent = (uint32_t)qs[r] | (mt[r] << 27);
              if (H16) {
                uint32_t t = (cj[r] + 0x555u - ci) & 0x333u;  // offset + 1 per axis, no borrow between nibbles
                t = (t & ~((mt[r] >> 5) & 0x333u)) | (mt[r] >> 15);
                ent = (uint32_t)qs[r] |
                      (((t & 3u) | ((t >> 2) & 0xcu) | ((t >> 4) & 0x30u)) << kH16SlotBits);
              }
              const int u = tn + __popc(keep & lt);
              tx[u] = x, ty[u] = y, tz[u] = z, te[u] = ent;
            }
            if (kr + own_delta < e && kr + own_delta + 32 > s) own0 = min(own0, tn), own1 = tn + __popc(keep);
            tn += __popc(keep);
          }
        }
        const int tn32 = (tn + 31) & ~31;
        if (tn + lane < tn32) {
          tx[tn + lane] = kFarTile, ty[tn + lane] = kFarTile, tz[tn + lane] = kFarTile;
          te[tn + lane] = 0u;
        }
        __syncwarp();
        for (int u0 = 0; u0 < tn32; u0 += 32) {
          uint32_t m = 0;
          if (u0 + 32 <= own0 || u0 >= own1) {
#pragma unroll
            for (int u = 0; u < 32; u += 4) {
              const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(&tx[u0 + u]);
              const ulonglong2 Y = *reinterpret_cast<const ulonglong2*>(&ty[u0 + u]);
              const ulonglong2 Z = *reinterpret_cast<const ulonglong2*>(&tz[u0 + u]);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const f2 DX = sub2(IX, h ? X.y : X.x), DY = sub2(IY, h ? Y.y : Y.x), DZ = sub2(IZ, h ? Z.y : Z.x);
                // dist2 per half, then r^2 - R^2: negative exactly when r^2 < R^2
                const f2 T = add2(fma2(DZ, DZ, fma2(DY, DY, mul2(DX, DX))), NR2);
                m = __funnelshift_l(__float_as_uint(lo(T)), m, 1);
                m = __funnelshift_l(__float_as_uint(hi(T)), m, 1);
              }
            }
          } else {  // the cell's own particles: 0 < r^2 < R^2 (the particle itself, and any at its very place, out)
#pragma unroll 4
            for (int u = 0; u < 32; ++u) {
              const float r2 = dist2(I.x - tx[u0 + u], I.y - ty[u0 + u], I.z - tz[u0 + u]);
              m = 2u * m + (__float_as_uint(r2) - 1u < hb ? 1u : 0u);
            }
          }
          S.mask[u0 >> 5][lane] = m;  // bit 31 - u: candidate u0 + u is within the list radius
        }
        __syncwarp();
        const int words = tn32 >> 5;
        uint16_t* buf = S.buf[lane];
        for (int w = 0; w < words;) {
          // as many words as fit every lane's row buffer
          int n = 0;
          for (; w < words; ++w) {
            uint32_t m = S.mask[w][lane];
            if (__any_sync(full, n + __popc(m) > ScanTile::kBuf)) break;
            while (m) {
              const int u = __clz(m);
              m ^= 0x80000000u >> u;
              buf[n++] = (uint16_t)(32 * w + u);
            }
          }
          // up to an entry whose place in the row is a multiple of four, then whole groups, then the rest
          int g = 0;
          for (; g < n && ((len + g) & 3); ++g)
            if (len + g < L) put(len + g, te[buf[g]]);
          for (; g + 4 <= n; g += 4) {
            const uint4 ent = make_uint4(te[buf[g]], te[buf[g + 1]], te[buf[g + 2]], te[buf[g + 3]]);
            if (len + g + 4 <= L) row[8 * (len + g)] = ent;
          }
          for (; g < n; ++g)
            if (len + g < L) put(len + g, te[buf[g]]);
          len += n;
        }
        __syncwarp();
      } while (k0 < total);
      if (mine) {
        a.list_cnt[ib + lane] = len;
        if (len > L) {
          // the next step rebuilds (a finished instance's particles never move again)
          if (a.phase[inst] != PH_STEP || a.dyn[inst].dt_cur > 0.0f) a.list_flags[kLfOverflowPending] = 1u;
        } else {  // pad the row to a whole group of four (list_max is a multiple of four)
          for (int k = len; k < ((len + 3) & ~3); ++k) put(k, a.list_pad);
        }
        longest = max(longest, len);
      }
    }
  }
  longest = __reduce_max_sync(full, longest);
  if (lane == 0 && longest > 0) atomicMax(&a.list_flags[kLfLongest], (unsigned)longest);
}

template <bool H16, int WARPS>
inline int launch_list_scan_v(const StepArgs& a, cudaStream_t s) {
  static TiledLaunch L[16];
  int dev = 0;
  WCSPH_CUDA(cudaGetDevice(&dev));
  TiledLaunch& T = L[dev & 15];
  auto kern = k_list_scan<H16, WARPS>;
  const int bytes = (int)sizeof(ScanTile) * WARPS;
  if (T.device != dev) {
    WCSPH_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    int per_sm = 0, sms = 0;
    WCSPH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WARPS * 32, bytes));
    WCSPH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    T.blocks = std::max(1, per_sm) * sms;
    T.device = dev;
  }
  kern<<<T.blocks, WARPS * 32, bytes, s>>>(a);
  WCSPH_CUDA(cudaGetLastError());
  return 0;
}

// Shapes of the list build's scan: warps per block.  3 and 5 repeat shape 0,
// 4 and 6 shape 2.  All build the same lists.
constexpr int kBuildShapes = 7;
constexpr int kBuildShapesTimed = 3;

template <bool H16>
inline int launch_list_scan(const StepArgs& a, int n, cudaStream_t s, int shape = 0) {
  if (n > kMaxTiledParticles) {
    set_error("the tiled path holds at most %d particles per solver (got %d)", kMaxTiledParticles, n);
    return WCSPH_E_CAPACITY;
  }
  switch (shape) {
    case 1: return launch_list_scan_v<H16, 2>(a, s);
    case 2: case 4: case 6: return launch_list_scan_v<H16, 8>(a, s);
    default: return launch_list_scan_v<H16, 4>(a, s);
  }
}

}  // namespace wcsph
