// Reading an instance back in its original particle order.
//
// The state lies sorted by cell, so that a host loop over it writes every
// field at a random place, and copies into pageable memory run at a fraction
// of the link.  Here the device undoes the sort: k_read_index notes, for every
// original index, the slot that holds it; k_read_state / k_read_diag gather the
// caller's arrays, packed as the caller holds them, into buffers that are free
// between passes.  They then cross the link piece by piece into a ring of
// blocks, each copied out by a few host threads while the next ones are
// in flight.  1.25 M particles (56 MB): 70 -> 6.7 ms, 65,000: 1.43 -> 0.4, 12,600: 0.36 -> 0.12;
// a probe of 1.25 M 35 -> 6 ms.  Bound by the host's first touch of the caller's
// arrays.
#pragma once
#include <omp.h>
#include <sys/mman.h>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "sim_kernels.cuh"

namespace wcsph {

// Slots that may hold particles of the instance: its range [range_lo, range_hi)
// and, with tail set, the dead slots behind the live ones.  idx[i] becomes 1 +
// the last such slot of particle i (0: none).
__global__ void k_read_index(SimArrays A, const InstDyn* __restrict__ dyn, const int* __restrict__ n_alive, int n_host,
                             int slot, int n, int tail, unsigned* __restrict__ idx) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n_host) return;
  const int lo = dyn[slot].range_lo, hi = dyn[slot].range_hi;
  if (!(q >= lo && q < hi) && !(tail && q >= *n_alive)) return;
  if (tail) {  // ghosts: their owner reports them
    const uint32_t f = A.flags[q];
    if ((int)(f & kInstMask) != slot || (f & kGhostBit)) return;
  }
  const int i = A.pid[q];
  if (i >= 0 && i < n) atomicMax(&idx[i], (unsigned)q + 1u);
}

// What idx says of particle i: cover 0 (no slot holds it), 1 (dead) or 3, and
// the number of particles without a slot.
__device__ __forceinline__ int read_cover(const unsigned* idx, const uint32_t* flags, int i, bool in, uint8_t* cover,
                                          int* missing) {
  const int q = in ? (int)idx[i] - 1 : 0;
  const unsigned none = __ballot_sync(0xffffffffu, q < 0);
  if (none && (threadIdx.x & 31) == 0) atomicAdd(missing, __popc(none));
  if (in) cover[i] = q < 0 ? 0 : (flags[q] & kDeadBit) ? 1 : 3;
  return in ? q : -1;
}

__global__ void k_read_state(SimArrays A, const unsigned* __restrict__ idx, int n, float* __restrict__ pos3,
                             float* __restrict__ vel3, float* __restrict__ acc3, float* __restrict__ dens,
                             float* __restrict__ div_v, uint8_t* __restrict__ cover, int* __restrict__ missing) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = read_cover(idx, A.flags, i, i < n, cover, missing);
  if (q < 0) return;
  const float4 p = A.pos[q], v = A.vel[q], c = A.acc[q];
  const size_t k = 3 * (size_t)i;
  pos3[k] = p.x, pos3[k + 1] = p.y, pos3[k + 2] = p.z;
  vel3[k] = v.x, vel3[k + 1] = v.y, vel3[k + 2] = v.z;
  acc3[k] = c.x, acc3[k + 1] = c.y, acc3[k + 2] = c.z;
  dens[i] = p.w;
  div_v[i] = c.w;
}

__global__ void k_read_diag(const float4* __restrict__ acc, const float* __restrict__ dt, const float* __restrict__ rho,
                            const int* __restrict__ nbr, const uint32_t* __restrict__ flags,
                            const unsigned* __restrict__ idx, int n, float* __restrict__ acc3,
                            float* __restrict__ div_v, float* __restrict__ dt_i, float* __restrict__ dens,
                            int* __restrict__ n_nbr, uint8_t* __restrict__ cover, int* __restrict__ missing) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = read_cover(idx, flags, i, i < n, cover, missing);
  if (q < 0) return;
  const float4 c = acc[q];
  const size_t k = 3 * (size_t)i;
  acc3[k] = c.x, acc3[k + 1] = c.y, acc3[k + 2] = c.z;
  div_v[i] = c.w;
  dt_i[i] = dt[q];
  dens[i] = rho[q];
  n_nbr[i] = nbr[q];
}

// One of the caller's arrays: width 4-byte words a particle; src null: zeros.
struct ReadField {
  const void* src;
  void* dst;
  int width;
};

// Ring of host blocks the pieces of a read pass through, given back with the
// solver.  Its full size is for the largest read the solver can have, at most
// kBlockBytes a block (1.6 M particles, 72 MB: 4.6 ms with blocks of 8 MB, 7.3
// with 4), registered with the device.  That costs 0.4 to 2 ms once, at times more
// (12 MB of huge pages 0.8 ms; cudaMallocHost 5.6), and is done by the read with
// which the reads so far have brought a quarter of the ring's bytes: by the first
// one of a large instance, by the second where blocks are up to kSecondBytes
// (12,600 particles: 0.22 ms a read, 0.10 registered), late where a large solver is
// asked for a few particles (300 of 4 M: a first read of 2 ms and more with the
// full ring, 0.15 without).  Until then, where blocks are below kPinBytes, and where
// registering fails, ordinary memory of the read's own size serves; copies into it
// are synchronous.
class ReadRing {
 public:
  ~ReadRing() { release(); }

  // Copies the n (at most n_max in any read) particles' cover bytes and fields to the host: stream order
  // after the kernels that wrote them.  Particles without a slot keep the
  // caller's values.  alive (or null) becomes cover == 3.
  int copy_out(cudaStream_t s, int n, long long n_max, const uint8_t* cover, const int* missing, const ReadField* f, int nf,
               int32_t* alive) {
    struct Piece {
      int field, i0, i1;  // field -1: cover
      size_t off;
    };
    if (int rc = reserve(s, n, n_max)) return rc;
    // Pieces in order, cut into batches of one block each.
    std::vector<std::vector<Piece>> batch(1);
    size_t used = kHead;  // the first block starts with the count of missing particles
    auto add = [&](int field, size_t el) {
      for (int i = 0; i < n;) {
        size_t room = (bytes_ - used) / el / 16 * 16;  // pieces start 16-byte aligned
        if (room == 0) {
          batch.emplace_back();
          used = 0;
          room = bytes_ / el / 16 * 16;
        }
        const int m = (int)std::min<size_t>(room, (size_t)(n - i));
        batch.back().push_back({field, i, i + m, used});
        used = (used + el * m + 15) & ~(size_t)15;
        i += m;
      }
    };
    add(-1, 1);
    for (int k = 0; k < nf; ++k)
      if (f[k].dst && f[k].src) add(k, 4 * (size_t)f[k].width);
    auto enqueue = [&](size_t b) -> int {
      char* base = mem_ + (b % kBlocks) * bytes_;
      if (b == 0) WCSPH_CUDA(cudaMemcpyAsync(base, missing, sizeof(int), cudaMemcpyDeviceToHost, s));
      for (const Piece& p : batch[b]) {
        const size_t el = p.field < 0 ? 1 : 4 * (size_t)f[p.field].width;
        const char* src = p.field < 0 ? (const char*)cover : (const char*)f[p.field].src;
        WCSPH_CUDA(cudaMemcpyAsync(base + p.off, src + el * p.i0, el * (p.i1 - p.i0), cudaMemcpyDeviceToHost, s));
      }
      WCSPH_CUDA(cudaEventRecord(ev_[b % kBlocks], s));
      return 0;
    };
    for (size_t b = 0; b < batch.size() && b < kBlocks; ++b)
      if (int rc = enqueue(b)) return rc;
    int lost = 0;
    std::vector<uint8_t> have;  // cover, when some particles have no slot
    for (size_t b = 0; b < batch.size(); ++b) {
      WCSPH_CUDA(cudaEventSynchronize(ev_[b % kBlocks]));
      const char* base = mem_ + (b % kBlocks) * bytes_;
      if (b == 0) {
        memcpy(&lost, base, sizeof(int));
        if (lost) have.resize(n);
      }
      for (const Piece& p : batch[b]) {
        if (p.field < 0) {
          const uint8_t* c = (const uint8_t*)base + p.off - p.i0;
          if (lost) memcpy(have.data() + p.i0, c + p.i0, p.i1 - p.i0);
          if (alive) slices(p.i0, p.i1, 4, [&](int i0, int i1) {
            for (int i = i0; i < i1; ++i) alive[i] = c[i] == 3;
          });
        } else {
          const size_t el = 4 * (size_t)f[p.field].width;
          const char* src = base + p.off;
          char* dst = (char*)f[p.field].dst;
          slices(p.i0, p.i1, el, [&](int i0, int i1) {
            if (!lost) {
              memcpy(dst + el * i0, src + el * (i0 - p.i0), el * (i1 - i0));
              return;
            }
            for (int i = i0; i < i1; ++i)
              if (have[i]) memcpy(dst + el * i, src + el * (i - p.i0), el);
          });
        }
      }
      if (b + kBlocks < batch.size())
        if (int rc = enqueue(b + kBlocks)) return rc;
    }
    for (int k = 0; k < nf; ++k)
      if (f[k].dst && !f[k].src) {
        const size_t el = 4 * (size_t)f[k].width;
        char* dst = (char*)f[k].dst;
        slices(0, n, el, [&](int i0, int i1) {
          if (!lost) memset(dst + el * i0, 0, el * (i1 - i0));
          else
            for (int i = i0; i < i1; ++i)
              if (have[i]) memset(dst + el * i, 0, el);
        });
      }
    return 0;
  }

  void release() {
    drop();
    for (cudaEvent_t& e : ev_) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
  }

 private:
  static constexpr size_t kBlocks = 3, kBlockBytes = 8 << 20, kPinBytes = 128 << 10, kHead = 16;
  static constexpr size_t kSecondBytes = 1 << 20, kHuge = 2 << 20;
  static constexpr size_t kSlice = 128 << 10;  // bytes of a host thread's share, at least
  static constexpr int kThreads = 10;  // 309,000 particles: 0.8 ms, with 16 threads 1.3 (they share the cores with the caller)

  template <class Body>
  static void slices(int i0, int i1, size_t el, Body&& body) {
    const size_t bytes = el * (size_t)(i1 - i0);
    const int t = (int)std::min<size_t>(std::min(kThreads, omp_get_max_threads()), bytes / kSlice);
    if (t <= 1) return body(i0, i1);
#pragma omp parallel for num_threads(t) schedule(static)
    for (int k = 0; k < t; ++k)
      body(i0 + (int)((long long)(i1 - i0) * k / t), i0 + (int)((long long)(i1 - i0) * (k + 1) / t));
  }

  static size_t read_bytes(long long n) { return 48 * (size_t)n + 4096; }  // 45 a particle and a few pieces' alignment
  // A block of the ring for reads of n particles: a quarter of one, but 1 MB in one block.
  static size_t block_bytes(long long n) {
    const size_t whole = read_bytes(n);
    const size_t b = std::min<size_t>(kBlockBytes, std::max<size_t>(whole / 4, std::min<size_t>(whole, 1 << 20)));
    return (b + 4095) / 4096 * 4096;
  }

  int reserve(cudaStream_t s, int n, long long n_max) {
    for (cudaEvent_t& e : ev_)
      if (!e) WCSPH_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    if (full_) return 0;
    const size_t full = block_bytes(n_max);
    ++reads_;
    total_ += read_bytes(n);
    const bool now = full >= kPinBytes && 4 * total_ >= kBlocks * full && (full > kSecondBytes || reads_ > 1);
    const size_t want = now || full <= kSecondBytes ? full : block_bytes(n);
    if (bytes_ < want) {
      if (mem_) WCSPH_CUDA(cudaStreamSynchronize(s));  // a read that failed may have left copies in flight
      drop();
      const size_t all = (want * kBlocks + kHuge - 1) / kHuge * kHuge;
      mem_ = static_cast<char*>(now || want >= kPinBytes ? aligned_alloc(kHuge, all) : malloc(want * kBlocks));
      if (!mem_) {
        set_error("read: %zu bytes of host memory are not to be had", want * kBlocks);
        return WCSPH_E_NOMEM;
      }
      bytes_ = want;
    }
    if (now) {
      full_ = true;
      pin();
    }
    return 0;
  }

  void drop() {
    if (pinned_) cudaHostUnregister(mem_);
    free(mem_);
    mem_ = nullptr;
    pinned_ = full_ = false;
    bytes_ = 0;
  }

  void pin() {
    const size_t all = (bytes_ * kBlocks + kHuge - 1) / kHuge * kHuge;
    if (bytes_ > kSecondBytes) {
      madvise(mem_, all, MADV_HUGEPAGE);
      slices(0, (int)(all / kHuge), kHuge, [&](int i0, int i1) { memset(mem_ + kHuge * i0, 0, kHuge * (i1 - i0)); });
    }
    pinned_ = cudaHostRegister(mem_, bytes_ > kSecondBytes ? all : bytes_ * kBlocks, cudaHostRegisterDefault) == cudaSuccess;
    if (!pinned_) cudaGetLastError();
  }

  char* mem_ = nullptr;
  cudaEvent_t ev_[kBlocks] = {};
  size_t bytes_ = 0;      // per block
  size_t total_ = 0;      // bytes of the reads so far
  long long reads_ = 0;
  bool full_ = false;     // full size, and registered if it can be
  bool pinned_ = false;
};

}  // namespace wcsph
