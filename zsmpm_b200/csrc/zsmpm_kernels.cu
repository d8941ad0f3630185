// sm_100a kernels of the explicit MLS/APIC MPM substep.
//
// Pipeline of one substep (all launches have fixed shapes and read their sizes from
// device counters, so a substep can be captured in a CUDA graph):
//   activation  k_begin, k_insert_moved_blocks, k_insert_particle_blocks, k_enlarge,
//               k_bitmap_prepare, k_bitmap_set, scan(3), k_assign_ranks, k_neighbors
//   binning     k_bin_count, scan(3), k_cell_start, k_bin_scatter, k_bin_finalize, and the
//               incremental k_inc_* beside them
//               (scenes of up to 2^20 particles: activation and binning in one launch, k_prepare)
//   transfer    k_p2g, k_grid_update, k_grid_boundaries, k_g2p
// Reference operators replaced: SparsityOp.hpp:41-112 (activation), SparsityOp.hpp:115-196
// (binning), P2G.hpp:45-127, GridOp.hpp:54-164, G2P.hpp:43-84 (paths inside include/zensim).
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#include "zsmpm_device.cuh"
#include "zsmpm_internal.h"

namespace zsmpm {

namespace {

constexpr int kThreads = 256;
constexpr unsigned kFull = 0xffffffffu;
// Particle passes take kPass particles per thread per round: all loads first, so that several
// are in flight per thread (the passes are bound by load latency, not bandwidth).
constexpr int kPass = 4;

__device__ __forceinline__ void set_status(int *ctr, int bit) { atomicOr(&ctr[kCtrStatus], bit); }

__device__ __forceinline__ int grid_threads() { return gridDim.x * blockDim.x; }

// ----------------------------------------------------------------- hash table
// Insert with the reference's home slot and stride-127 linear probing
// (HashTable.hpp:356-374).  The slot is claimed by a 64-bit CAS on the packed key instead
// of the reference's per-slot spin lock, so no thread ever waits on another.
// Returns the insertion index when this call inserted the key, -1 when it existed, -2 when
// the table is full.
__device__ int table_insert(const scene_device &s, uint64_t key, int3 k, int *counter,
                            int index_base) {
  const int T = s.prm.table_size;
  int slot = home_slot(k.x, k.y, k.z, T);
  for (int probe = 0; probe < T; ++probe) {
    // most calls find their key already present (every warp of a block's particles asks):
    // a plain load settles those without a contended atomic
    unsigned long long prev = *reinterpret_cast<volatile unsigned long long *>(&s.pk[slot]);
    if (prev == (unsigned long long)key) return -1;
    if (prev == kEmptyKey)
      prev = atomicCAS((unsigned long long *)&s.pk[slot], (unsigned long long)kEmptyKey, (unsigned long long)key);
    if (prev == kEmptyKey) {
      const int idx = index_base + atomicAdd(counter, 1);
      s.tkeys[3 * slot + 0] = k.x;
      s.tkeys[3 * slot + 1] = k.y;
      s.tkeys[3 * slot + 2] = k.z;
      if (idx < s.prm.nb_cap) {
        s.ins_pk[idx] = key;
        s.ins_slot[idx] = slot;
        s.tidx[slot] = idx;
      } else {
        // beyond the block capacity: keep the key unqueryable so no kernel indexes past it
        set_status(s.ctr, kStatusCapacity);
        s.tidx[slot] = -1;
      }
      return idx;
    }
    if (prev == key) return -1;
    slot = (slot + 127) & (T - 1);
  }
  set_status(s.ctr, kStatusTableFull);
  return -2;
}

// HashTable::query (HashTable.hpp:444-456): index of the key or -1.
__device__ int table_query(const scene_device &s, uint64_t key, int3 k) {
  const int T = s.prm.table_size;
  int slot = home_slot(k.x, k.y, k.z, T);
  for (int probe = 0; probe < T; ++probe) {
    const uint64_t p = s.pk[slot];
    if (p == key) return s.tidx[slot];
    if (p == kEmptyKey) return -1;
    slot = (slot + 127) & (T - 1);
  }
  return -1;
}

// x / dx + 1/2, whose floor is the index bucket (one rounding, written out so that every kernel that
// asks for a particle's cell computes the same number)
__device__ __forceinline__ float bucket_of(const scene_params &p, float x) { return fmaf(x, p.inv_dx, 0.5f); }

// Stencil-origin cell and block of a position exactly as ComputeSparsity computes them
// (SparsityOp.hpp:70-77): c = floor(x * (1/dx) + 0.5) - 2, block = floor_div(c, 8).
// Returns false for NaN/Inf or positions beyond the packed key range.
__device__ __forceinline__ bool cell_of(const scene_params &p, float4 x, int3 &c, int3 &b) {
  const float fx = bucket_of(p, x.x), fy = bucket_of(p, x.y), fz = bucket_of(p, x.z);
  const float lim = (float)(kKeyLimit * 8);
  if (!(fabsf(fx) < lim && fabsf(fy) < lim && fabsf(fz) < lim)) return false;
  c = make_int3((int)floorf(fx) - 2, (int)floorf(fy) - 2, (int)floorf(fz) - 2);
  b = make_int3(block_of_cell(c.x), block_of_cell(c.y), block_of_cell(c.z));
  return true;
}

// x / dx for the particle's position in cells (P2G.hpp:62, G2P.hpp:56-58, G2P2G.hpp): the product
// with the rounded reciprocal and one correction by the remainder (Markstein 1990), which is
// the correctly rounded quotient but for rare last-place cases; where dx is a power of two the
// product is exact and the correction zero.
__device__ __forceinline__ float over_dx(const scene_params &p, float x) {
  const float q = x * p.inv_dx;
  return fmaf(fmaf(-q, p.dx, x), p.inv_dx, q);
}

// Batched scenes: the slot of a scene, the slot coordinate of a key component (keys of a
// scene lie in [32 slot - 4, 32 slot + 28)), and the scene-local block of a key.
__device__ __forceinline__ int3 slot_of_scene(int sc) { return make_int3(sc & 7, (sc >> 3) & 7, sc >> 6); }
__device__ __forceinline__ int slot_coord(int k) { return (k + kBatchMargin) / kBatchSlot; }
__device__ __forceinline__ int scene_of_key(int3 k) {
  return slot_coord(k.x) + 8 * slot_coord(k.y) + 64 * slot_coord(k.z);
}
__device__ __forceinline__ int3 local_block(const scene_params &p, int3 k) {
  if (!p.batch) return k;
  return make_int3(k.x - kBatchSlot * slot_coord(k.x), k.y - kBatchSlot * slot_coord(k.y),
                   k.z - kBatchSlot * slot_coord(k.z));
}

// Cell and block of particle i in the scene's key space: cell_of, then for batched scenes a
// check that the local block leaves room for the +1 enlargement inside the slot, and the
// slot offset.
// sid: the particle's scene (batched scenes only)
__device__ __forceinline__ bool particle_cell(const scene_device &s, int sid, float4 x, int3 &c, int3 &b) {
  if (!cell_of(s.prm, x, c, b)) return false;
  if (s.prm.batch) {
    const int hi = kBatchSlot - kBatchMargin - 1;
    if (b.x < -kBatchMargin || b.x >= hi || b.y < -kBatchMargin || b.y >= hi || b.z < -kBatchMargin || b.z >= hi)
      return false;
    const int3 o = slot_of_scene(sid);
    b = make_int3(b.x + kBatchSlot * o.x, b.y + kBatchSlot * o.y, b.z + kBatchSlot * o.z);
    c = make_int3(c.x + 8 * kBatchSlot * o.x, c.y + 8 * kBatchSlot * o.y, c.z + 8 * kBatchSlot * o.z);
  }
  return true;
}

// ----------------------------------------------------------------- CTA scan helpers
template <int NT>
__device__ __forceinline__ int cta_exclusive_scan(int v, int &total, int *smem /* >= NT/32 + 1 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < NT / 32 ? smem[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, w, o);
      if (lane >= o) w += y;
    }
    if (lane < NT / 32) smem[lane] = w;
    if (lane == NT / 32 - 1) smem[NT / 32] = w;
  }
  __syncthreads();
  const int incl = x + (warp > 0 ? smem[warp - 1] : 0);
  total = smem[NT / 32];
  __syncthreads();
  return incl - v;
}

// ----------------------------------------------------------------- device-wide scan
// Three-phase exclusive scan over n values produced by Load(i) (n read from device memory
// at *n_ptr), kScanCtas CTAs x kThreads.  out[n] receives the total.
struct load_popc {
  const uint32_t *w;
  __device__ int operator()(int i) const { return __popc(w[i]); }
};
struct load_int {
  const int *a;
  __device__ int operator()(int i) const { return a[i]; }
};

template <class Load>
__global__ void __launch_bounds__(kThreads) k_scan_reduce(Load ld, const int *n_ptr, int *part) {
  __shared__ int sm[kThreads / 32 + 1];
  const int n = *n_ptr;
  const int chunk = (n + gridDim.x - 1) / gridDim.x;
  const int lo = min(n, (int)blockIdx.x * chunk), hi = min(n, lo + chunk);
  int acc = 0;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) acc += ld(i);
  int total;
  cta_exclusive_scan<kThreads>(acc, total, sm);
  if (threadIdx.x == 0) part[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kThreads) k_scan_partials(int *part, int parts) {
  __shared__ int sm[kThreads / 32 + 1];
  const int v = threadIdx.x < parts ? part[threadIdx.x] : 0;
  int total;
  const int ex = cta_exclusive_scan<kThreads>(v, total, sm);
  if (threadIdx.x < parts) part[threadIdx.x] = ex;
  if (threadIdx.x == 0) part[parts] = total;
}

template <class Load>
__global__ void __launch_bounds__(kThreads) k_scan_down(Load ld, const int *n_ptr, const int *part,
                                                         int *out) {
  __shared__ int sm[kThreads / 32 + 1];
  const int n = *n_ptr;
  const int chunk = (n + gridDim.x - 1) / gridDim.x;
  const int lo = min(n, (int)blockIdx.x * chunk), hi = min(n, lo + chunk);
  int run = part[blockIdx.x];
  for (int base = lo; base < hi; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < hi ? ld(i) : 0;
    int total;
    const int ex = cta_exclusive_scan<kThreads>(v, total, sm);
    if (i < hi) out[i] = run + ex;
    run += total;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = part[gridDim.x];
}

template <class Load>
cudaError_t device_scan(Load ld, const int *n_ptr, int *part, int *out, cudaStream_t st) {
  k_scan_reduce<<<kScanCtas, kThreads, 0, st>>>(ld, n_ptr, part);
  k_scan_partials<<<1, kThreads, 0, st>>>(part, kScanCtas);
  k_scan_down<<<kScanCtas, kThreads, 0, st>>>(ld, n_ptr, part, out);
  return cudaGetLastError();
}

// ----------------------------------------------------------------- activation
// Resets the hash table (CleanSparsity, SparsityOp.hpp:41-55) and the per-substep counters.
__device__ __forceinline__ void do_begin(const scene_device &s) {
  const int T = s.prm.table_size;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < T; i += grid_threads()) {
    s.pk[i] = kEmptyKey;
    s.tkeys[3 * i + 0] = 0x7fffffff;
    s.tkeys[3 * i + 1] = 0x7fffffff;
    s.tkeys[3 * i + 2] = 0x7fffffff;
    s.tidx[i] = -1;
    s.tstatus[i] = -1;
  }
  if (blockIdx.x == 0 && threadIdx.x < kCtrCount) {
    const int t = threadIdx.x;
    // k_bitmap_prepare resets the two mask counters; the binning clears the mover count
    // the learned G2P's queue counters stay for a closure pass that runs beside this substep's
    // activation and binning (the learned G2P clears the queue before it fills it)
    if (t == kCtrStatus || t == kCtrMaskFrom || t == kCtrMaskBad || t == kCtrMovers || t == kCtrQueue ||
        t == kCtrQueueSubstep || t == kCtrBarrier || t == kCtrBarrierExit)
      return;
    if (t == kCtrUseMasks) {
      s.ctr[t] = s.ctr[kCtrMaskBad] == 0 ? s.ctr[kCtrMaskFrom] : 0;
      return;
    }
    if (t == kCtrIncBin) {
      // the move masks are valid exactly when the last G2P listed every particle that left
      // its cell, so the binning can merge those into the last binning's order
      s.ctr[t] = (s.ctr[kCtrMaskBad] == 0 && s.ctr[kCtrMaskFrom] > 0) ? 1 : 0;
      return;
    }
    if (t == kCtrSubstep) {
      s.ctr[t] += 1;
      return;
    }
    int v = 0;
    if (t >= kCtrBoxLo && t < kCtrBoxLo + 3) v = 0x7fffffff;
    if (t >= kCtrBoxHi && t < kCtrBoxHi + 3) v = -0x7fffffff;
    s.ctr[t] = v;
  }
}
__global__ void __launch_bounds__(kThreads) k_begin(scene_device s) { do_begin(s); }

// ComputeSparsity (SparsityOp.hpp:58-86): one insert per distinct block key of a warp.
__device__ __forceinline__ void do_insert_particle_blocks(const scene_device &s) {
  if (s.ctr[kCtrUseMasks] > 0) return;  // k_insert_moved_blocks inserts this substep's blocks
  const int lane = threadIdx.x & 31;
  const int n = s.prm.n;
  int3 lo = make_int3(0x7fffffff, 0x7fffffff, 0x7fffffff);
  int3 hi = make_int3(-0x7fffffff, -0x7fffffff, -0x7fffffff);
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int warps = grid_threads() >> 5;
  for (int base0 = warp_global * 32 * kPass; base0 < n; base0 += warps * 32 * kPass) {
    float4 xs[kPass];
    int sids[kPass];
#pragma unroll
    for (int u = 0; u < kPass; ++u) {
      const int i = base0 + u * 32 + lane;
      xs[u] = i < n ? s.cur.xm[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      sids[u] = (s.prm.batch && i < n) ? s.cur.sid[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < kPass; ++u) {
      const int i = base0 + u * 32 + lane;
      uint64_t key = kEmptyKey - 1 - lane;  // distinct per lane when invalid
      int3 c, b = make_int3(0, 0, 0);
      bool valid = false;
      if (i < n) {
        if (particle_cell(s, sids[u], xs[u], c, b)) {
          key = pack_key(b.x, b.y, b.z);
          valid = true;
        } else {
          set_status(s.ctr, kStatusOutOfDomain);
        }
      }
      const unsigned peers = __match_any_sync(kFull, key);
      if (valid && lane == __ffs(peers) - 1) {
        table_insert(s, key, b, &s.ctr[kCtrParticleBlocks], 0);
        lo = make_int3(min(lo.x, b.x), min(lo.y, b.y), min(lo.z, b.z));
        hi = make_int3(max(hi.x, b.x), max(hi.y, b.y), max(hi.z, b.z));
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo.x = min(lo.x, __shfl_xor_sync(kFull, lo.x, o));
    lo.y = min(lo.y, __shfl_xor_sync(kFull, lo.y, o));
    lo.z = min(lo.z, __shfl_xor_sync(kFull, lo.z, o));
    hi.x = max(hi.x, __shfl_xor_sync(kFull, hi.x, o));
    hi.y = max(hi.y, __shfl_xor_sync(kFull, hi.y, o));
    hi.z = max(hi.z, __shfl_xor_sync(kFull, hi.z, o));
  }
  if (lane == 0 && lo.x != 0x7fffffff) {
    atomicMin(&s.ctr[kCtrBoxLo + 0], lo.x);
    atomicMin(&s.ctr[kCtrBoxLo + 1], lo.y);
    atomicMin(&s.ctr[kCtrBoxLo + 2], lo.z);
    atomicMax(&s.ctr[kCtrBoxHi + 0], hi.x);
    atomicMax(&s.ctr[kCtrBoxHi + 1], hi.y);
    atomicMax(&s.ctr[kCtrBoxHi + 2], hi.z);
  }
}
__global__ void __launch_bounds__(kThreads) k_insert_particle_blocks(scene_device s) { do_insert_particle_blocks(s); }

// ComputeSparsity from the move masks the last G2P wrote: the blocks the particles of each
// previous block ended in (the same set of keys as the particle pass finds, since G2P computes
// each particle's block from the position it stores).  Runs instead of the particle pass
// after a G2P in which no particle left its block's 3^3 neighbourhood.
__device__ __forceinline__ void do_insert_moved_blocks(const scene_device &s) {
  const int nold = s.ctr[kCtrUseMasks];
  if (nold == 0) return;
  // the previous binning's block keys by their index then (k_assign_ranks renumbers blk_pk)
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nold; b += grid_threads()) s.old_pk[b] = s.blk_pk[b];
  int3 lo = make_int3(0x7fffffff, 0x7fffffff, 0x7fffffff);
  int3 hi = make_int3(-0x7fffffff, -0x7fffffff, -0x7fffffff);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nold * 27; t += grid_threads()) {
    const int b = t / 27, j = t % 27;
    if (!((s.bmask[b] >> j) & 1u)) continue;
    const int3 k = unpack_key(s.blk_pk[b]);
    const int3 nk = make_int3(k.x + j / 9 - 1, k.y + (j / 3) % 3 - 1, k.z + j % 3 - 1);
    table_insert(s, pack_key(nk.x, nk.y, nk.z), nk, &s.ctr[kCtrParticleBlocks], 0);
    lo = make_int3(min(lo.x, nk.x), min(lo.y, nk.y), min(lo.z, nk.z));
    hi = make_int3(max(hi.x, nk.x), max(hi.y, nk.y), max(hi.z, nk.z));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo.x = min(lo.x, __shfl_xor_sync(kFull, lo.x, o));
    lo.y = min(lo.y, __shfl_xor_sync(kFull, lo.y, o));
    lo.z = min(lo.z, __shfl_xor_sync(kFull, lo.z, o));
    hi.x = max(hi.x, __shfl_xor_sync(kFull, hi.x, o));
    hi.y = max(hi.y, __shfl_xor_sync(kFull, hi.y, o));
    hi.z = max(hi.z, __shfl_xor_sync(kFull, hi.z, o));
  }
  if ((threadIdx.x & 31) == 0 && lo.x != 0x7fffffff) {
    atomicMin(&s.ctr[kCtrBoxLo + 0], lo.x);
    atomicMin(&s.ctr[kCtrBoxLo + 1], lo.y);
    atomicMin(&s.ctr[kCtrBoxLo + 2], lo.z);
    atomicMax(&s.ctr[kCtrBoxHi + 0], hi.x);
    atomicMax(&s.ctr[kCtrBoxHi + 1], hi.y);
    atomicMax(&s.ctr[kCtrBoxHi + 2], hi.z);
  }
}
__global__ void __launch_bounds__(kThreads) k_insert_moved_blocks(scene_device s) { do_insert_moved_blocks(s); }

// EnlargeSparsity{lo=0, hi=2} (SparsityOp.hpp:88-112): the +{0,1}^3 neighbours of every
// particle block, so that the 3x3x3 stencil of every particle lands in active blocks.
__device__ __forceinline__ void do_enlarge(const scene_device &s) {
  const int npb = min(s.ctr[kCtrParticleBlocks], s.prm.nb_cap);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < npb * 7; t += grid_threads()) {
    const int i = t / 7, o = t % 7 + 1;
    const int3 k = unpack_key(s.ins_pk[i]);
    const int3 nk = make_int3(k.x + (o >> 2), k.y + ((o >> 1) & 1), k.z + (o & 1));
    table_insert(s, pack_key(nk.x, nk.y, nk.z), nk, &s.ctr[kCtrEnlarged], npb);
  }
}
__global__ void __launch_bounds__(kThreads) k_enlarge(scene_device s) { do_enlarge(s); }

// Total block count, capacity checks and the words of the dense bitmap over the blocks' bounding
// box, which ranks them in ascending (bx, by, bz) order.  `write`: the caller is the one thread
// that records them.
__device__ __forceinline__ void block_totals(const scene_device &s, bool write, int &blocks, int &words) {
  int nb = s.ctr[kCtrParticleBlocks] + s.ctr[kCtrEnlarged];
  int st = 0;
  // HashTable.hpp:369 flags an insertion index >= T - 20, i.e. more than T - 20 blocks
  if (nb > s.prm.table_size - 20) st |= kStatusTableFull;
  if (nb > s.prm.nb_cap) {
    st |= kStatusCapacity;
    nb = s.prm.nb_cap;
  }
  words = 0;
  if (nb > 0) {
    const long long ex = (long long)s.ctr[kCtrBoxHi + 0] - s.ctr[kCtrBoxLo + 0] + 2;
    const long long ey = (long long)s.ctr[kCtrBoxHi + 1] - s.ctr[kCtrBoxLo + 1] + 2;
    const long long ez = (long long)s.ctr[kCtrBoxHi + 2] - s.ctr[kCtrBoxLo + 2] + 2;
    const long long vol = ex * ey * ez;
    const long long w = (vol + 31) / 32;
    if (w > s.prm.bitmap_cap) {
      st |= kStatusBitmap;
      nb = 0;
    } else {
      words = (int)w;
    }
  }
  blocks = nb;
  if (!write) return;
  s.ctr[kCtrMaskFrom] = 0;  // the masks are spent: the ranks below renumber the blocks
  s.ctr[kCtrMaskBad] = 0;
  if (st) set_status(s.ctr, st);
  s.ctr[kCtrBlocks] = nb;
  *s.view_cnt = nb;
  s.ctr[kCtrWords] = words;
}

__global__ void k_bitmap_prepare(scene_device s) {
  int nb, words;
  if (threadIdx.x == 0) block_totals(s, true, nb, words);
}

__device__ __forceinline__ long long dense_id(const scene_device &s, int3 k) {
  const long long ey = (long long)s.ctr[kCtrBoxHi + 1] - s.ctr[kCtrBoxLo + 1] + 2;
  const long long ez = (long long)s.ctr[kCtrBoxHi + 2] - s.ctr[kCtrBoxLo + 2] + 2;
  return (((long long)k.x - s.ctr[kCtrBoxLo + 0]) * ey + ((long long)k.y - s.ctr[kCtrBoxLo + 1])) * ez +
         ((long long)k.z - s.ctr[kCtrBoxLo + 2]);
}

__device__ __forceinline__ void do_bitmap_set(const scene_device &s, int nb) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += grid_threads()) {
    const long long d = dense_id(s, unpack_key(s.ins_pk[i]));
    atomicOr(&s.bitmap[d >> 5], 1u << (d & 31));
  }
}
__global__ void __launch_bounds__(kThreads) k_bitmap_set(scene_device s) {
  do_bitmap_set(s, s.ctr[kCtrWords] > 0 ? s.ctr[kCtrBlocks] : 0);
}

// rank = number of active keys below this one; index == rank from here on
__device__ __forceinline__ void do_assign_ranks(const scene_device &s, int nb, const int *word_prefix) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += grid_threads()) {
    const uint64_t key = s.ins_pk[i];
    const int3 k = unpack_key(key);
    const long long d = dense_id(s, k);
    const uint32_t w = s.bitmap[d >> 5];
    const int rank = word_prefix[d >> 5] + __popc(w & ((1u << (d & 31)) - 1u));
    s.tidx[s.ins_slot[i]] = rank;
    s.blk_pk[rank] = key;
    s.active_keys[3 * rank + 0] = k.x;
    s.active_keys[3 * rank + 1] = k.y;
    s.active_keys[3 * rank + 2] = k.z;
  }
}
__global__ void __launch_bounds__(kThreads) k_assign_ranks(scene_device s) {
  do_assign_ranks(s, s.ctr[kCtrWords] > 0 ? s.ctr[kCtrBlocks] : 0, s.word_prefix);
}

// neighbour table b + {0,1}^3 (index dx*4 + dy*2 + dz); clears the bitmap for next time
__device__ __forceinline__ void do_neighbors(const scene_device &s) {
  const int nb = s.ctr[kCtrBlocks];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nb * 8; t += grid_threads()) {
    const int b = t >> 3, o = t & 7;
    const int3 k = unpack_key(s.blk_pk[b]);
    const int3 nk = make_int3(k.x + (o >> 2), k.y + ((o >> 1) & 1), k.z + (o & 1));
    s.nbr[t] = table_query(s, pack_key(nk.x, nk.y, nk.z), nk);
  }
  const int words = s.ctr[kCtrWords];
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += grid_threads()) s.bitmap[w] = 0u;
}
__global__ void __launch_bounds__(kThreads) k_neighbors(scene_device s) { do_neighbors(s); }

// ----------------------------------------------------------------- binning
// Per particle: its block index and stencil-origin cell; counts per cell (rank within the
// cell from the atomic) and per block (warp-aggregated).
__device__ __forceinline__ bool incremental_binning(const scene_device &s) {
  return s.ctr[kCtrIncBin] != 0 && !s.prm.bin_full;
}

__device__ __forceinline__ void do_bin_count(const scene_device &s) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    s.ctr[kCtrOrderFront] = 0;  // k_cell_start fills work_order
    s.ctr[kCtrOrderBack] = 0;
    // the persistent kernels of this binning and of the transfers after it start from their
    // first block (a second binning after one activation must not find them spent)
    s.ctr[kCtrWork + kWorkCellStart] = 0;
    s.ctr[kCtrWork + kWorkFinalize] = 0;
    s.ctr[kCtrWork + kWorkP2G] = 0;
    s.ctr[kCtrWork + kWorkG2P] = 0;
  }
  if (incremental_binning(s)) return;  // k_inc_stayers and k_inc_movers count this substep
  const int lane = threadIdx.x & 31;
  const int n = s.prm.n;
  const int nb = s.ctr[kCtrBlocks];
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int warps = grid_threads() >> 5;
  for (int base0 = warp_global * 32 * kPass; base0 < n; base0 += warps * 32 * kPass) {
   float4 xs[kPass];
   int sids[kPass];
#pragma unroll
   for (int u = 0; u < kPass; ++u) {
     const int i = base0 + u * 32 + lane;
     xs[u] = i < n ? s.cur.xm[i] : make_float4(0.f, 0.f, 0.f, 0.f);
     sids[u] = (s.prm.batch && i < n) ? s.cur.sid[i] : 0;
   }
#pragma unroll
   for (int u = 0; u < kPass; ++u) {
    const int i = base0 + u * 32 + lane;
    uint64_t key = kEmptyKey - 1 - lane;
    int3 c = make_int3(0, 0, 0), b = make_int3(0, 0, 0);
    bool valid = false;
    if (i < n && particle_cell(s, sids[u], xs[u], c, b)) {
      key = pack_key(b.x, b.y, b.z);
      valid = true;
    }
    const unsigned peers = __match_any_sync(kFull, key);
    const int leader = __ffs(peers) - 1;
    int blk = -1;
    if (valid && lane == leader) blk = table_query(s, key, b);
    blk = __shfl_sync(kFull, blk, leader);
    if (valid && (blk < 0 || blk >= nb)) set_status(s.ctr, kStatusMissingBlock);
    const bool ok = valid && blk >= 0 && blk < nb;
    // block counts, one atomic per distinct block of the warp
    const unsigned bpeers = __match_any_sync(kFull, ok ? blk : -1 - lane);
    if (ok && lane == __ffs(bpeers) - 1) atomicAdd(&s.block_count[blk], __popc(bpeers));
    // cell counts, one atomic per distinct cell of the warp (particles arrive in the previous
    // binning's order, so a warp spans a few cells); ranks within the warp follow lane order
    const int cell = ((c.x - 8 * b.x) << 6) | ((c.y - 8 * b.y) << 3) | (c.z - 8 * b.z);
    const uint32_t k32 = ok ? (uint32_t)blk * 512u + (uint32_t)cell : 0xffffffffu - (uint32_t)lane;
    const unsigned cpeers = __match_any_sync(kFull, k32);
    const int cleader = __ffs(cpeers) - 1;
    int cbase = 0;
    if (ok && lane == cleader) {
      cbase = atomicAdd(&s.cell_count[k32], __popc(cpeers));
      // cell counts share their word with the incremental binning's arrival count (high 16 bits)
      if (cbase + __popc(cpeers) > 0xffff) set_status(s.ctr, kStatusCapacity);
    }
    cbase = __shfl_sync(kFull, cbase, cleader);
    if (i < n) {
      s.key32[i] = ok ? k32 : 0xffffffffu;
      s.rnk[i] = ok ? cbase + __popc(cpeers & lanemask_lt()) : 0;
    }
   }
  }
}
__global__ void __launch_bounds__(kThreads) k_bin_count(scene_device s) {
  // (k_prepare, where the movers are counted beside this, has it from do_begin)
  if (blockIdx.x == 0 && threadIdx.x == 0) s.ctr[kCtrDirty] = 0;
  do_bin_count(s);
}

// The blocks that hold particles, in the order the per-block kernels take them: work_order holds
// those of kBigBlock particles or more from the front and the others from the back.
__device__ __forceinline__ int work_blocks(const scene_device &s) {
  return s.ctr[kCtrOrderFront] + s.ctr[kCtrOrderBack];
}
__device__ __forceinline__ int work_block(const scene_device &s, int front, int nb, int w) {
  return s.work_order[w < front ? w : nb - 1 - (w - front)];
}

// G2P's items: parts of a block's slots (each loads the block's velocity halo again, so a block is
// split only where the blocks alone would leave SMs idle: measured with one split less or more,
// 490 k particles 0.0645 / 0.0553 / 0.0557 ms, 3.7 M 0.245 / 0.236 / 0.26 ms.
__device__ __forceinline__ int slot_parts(int nb, int ctas) {
  return nb >= 4 * ctas ? 1 : nb * 2 >= 4 * ctas ? 2 : nb * 4 >= 4 * ctas ? 4 : 8;
}

// Persistent per-block CTA loop helper.
__device__ __forceinline__ int grab_block(int *counter, int *s_b) {
  __syncthreads();
  if (threadIdx.x == 0) *s_b = atomicAdd(counter, 1);
  __syncthreads();
  return *s_b;
}

// cell-major offsets of every cell's particle list
__global__ void __launch_bounds__(512) k_cell_start(scene_device s) {
  __shared__ int sm[512 / 32 + 1];
  __shared__ int s_b;
  const int nb = s.ctr[kCtrBlocks];
  for (;;) {
    const int b = grab_block(&s.ctr[kCtrWork + kWorkCellStart], &s_b);
    if (b >= nb) break;
    // low 16 bits: particles counted in place (every particle of a full binning, the stayers of
    // an incremental one); high 16 bits: the incremental binning's arrivals
    const int craw = s.cell_count[b * 512 + threadIdx.x];
    const int c = (craw & 0xffff) + (craw >> 16);
    int total;
    const int ex = cta_exclusive_scan<512>(c, total, sm);
    s.cell_start[b * 512 + threadIdx.x] = s.block_start[b] + ex;
    // the per-block kernels take the big blocks first, so that they end on small ones
    if (threadIdx.x == 0) {
      s.bmask[b] = 0u;  // (G2P's items add to it)
      if (total >= kBigBlock)
        s.work_order[atomicAdd(&s.ctr[kCtrOrderFront], 1)] = b;
      else if (total > 0)
        s.work_order[nb - 1 - atomicAdd(&s.ctr[kCtrOrderBack], 1)] = b;
    }
  }
}

__device__ __forceinline__ void do_bin_scatter(const scene_device &s) {
  if (incremental_binning(s)) return;
  const int n = s.prm.n;
  const int stride = grid_threads();
  for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += kPass * stride) {
    uint32_t k[kPass];
    int r[kPass], cs[kPass];
#pragma unroll
    for (int u = 0; u < kPass; ++u) {
      const int i = i0 + u * stride;
      k[u] = i < n ? s.key32[i] : 0xffffffffu;
      r[u] = i < n ? s.rnk[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < kPass; ++u) cs[u] = k[u] != 0xffffffffu ? s.cell_start[k[u]] : 0;
#pragma unroll
    for (int u = 0; u < kPass; ++u)
      if (k[u] != 0xffffffffu) s.tmp[cs[u] + r[u]] = i0 + u * stride;
  }
}
__global__ void __launch_bounds__(kThreads) k_bin_scatter(scene_device s) { do_bin_scatter(s); }

// Orders the list of one cell (indices into cur) by upload id, from `in` into `out` (which may
// be the same array).  Lists of up to 12 entries are sorted in registers (every index known at
// compile time): two rounds of independent loads (the list, then the ids), then an insertion
// sort of (id << 32 | index) entries; ids are unique, so this orders the cell by id.  Longer
// lists (strongly compressed cells) take an insertion sort in place in global memory.
__device__ __forceinline__ void sort_cell_by_id(const scene_device &s, const int *in, int *out, int cs, int c) {
  constexpr int kMaxList = 12;
  if (c <= kMaxList) {
    unsigned long long e[kMaxList];
#pragma unroll
    for (int r = 0; r < kMaxList; ++r) e[r] = r < c ? (unsigned long long)(uint32_t)in[cs + r] : ~0ull;
#pragma unroll
    for (int r = 0; r < kMaxList; ++r)
      if (r < c) e[r] |= (unsigned long long)(uint32_t)s.cur.id[(int)(uint32_t)e[r]] << 32;
#pragma unroll
    for (int r = 1; r < kMaxList; ++r)
      if (r < c) {
#pragma unroll
        for (int q = r; q > 0; --q) {
          const unsigned long long lo = e[q - 1], hi = e[q];
          const bool sw = lo > hi;
          e[q - 1] = sw ? hi : lo;
          e[q] = sw ? lo : hi;
        }
      }
#pragma unroll
    for (int r = 0; r < kMaxList; ++r)
      if (r < c) out[cs + r] = (int)(uint32_t)e[r];
  } else {
    int *w = const_cast<int *>(in);
    for (int r = 1; r < c; ++r) {
      const int i = w[cs + r];
      const int id = s.cur.id[i];
      int q = r;
      while (q > 0 && s.cur.id[w[cs + q - 1]] > id) {
        w[cs + q] = w[cs + q - 1];
        --q;
      }
      w[cs + q] = i;
    }
    if (out != in)
      for (int r = 0; r < c; ++r) out[cs + r] = w[cs + r];
  }
}

// Final particle order of a block (full binning): cells ascending, the particles of a cell in
// increasing upload index (a stable sort by (block, cell)).  Also zeroes the block's grid and
// the counts for the next substep.  The register sort caps the kernel at 3 CTAs of 512
// threads per SM (binning 0.71 -> 0.62 ms on the 30 M-particle sand scene against a sort in
// local memory at 4 CTAs).
__global__ void __launch_bounds__(512, 3) k_bin_finalize(scene_device s) {
  if (incremental_binning(s)) return;
  __shared__ int s_b;
  const int nb = s.ctr[kCtrBlocks];
  const int t = threadIdx.x;
  if (blockIdx.x == 0 && t == 0) {
    s.ctr[kCtrMovers] = 0;  // the next G2P lists its movers afresh
    s.ctr[kCtrBinInfo] = -1;
  }
  for (;;) {
    const int b = grab_block(&s.ctr[kCtrWork + kWorkFinalize], &s_b);
    if (b >= nb) break;
    const int c = s.cell_count[b * 512 + t];
    const int cs = s.cell_start[b * 512 + t];
    s.cell_count[b * 512 + t] = 0;
    sort_cell_by_id(s, s.tmp, s.src, cs, c);
    float4 *g = reinterpret_cast<float4 *>(s.grid + (size_t)b * kGridChannels * 512);
    g[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t == 0) s.block_count[b] = 0;
  }
}

// ----------------------------------------------------------------- incremental binning
// After a G2P whose particles all stayed within their block's 3^3 neighbourhood, the particles
// are stored in the last binning's slot order, and G2P has flagged each slot whose particle
// left its cell (moved[]) and listed those slots (movers[]).  The particles that stayed
// (typically 98-99%) keep their relative order: it is already (cell, upload id) within their
// cell, and the block order is ascending keys both times.  So the new order is the stayers of
// every old cell, placed in order at the start of the same cell's new range, with the movers
// appended behind them and only the cells that received movers sorted again by id.  The result
// equals the full binning's order bit for bit.
//   k_inc_map            per old block: its index in the new activation
//   k_inc_stayers        per old cell: its stayers -> cell_count (low 16 bits) of the cell in
//                        the block's new index, and the block's total
//   k_inc_movers         per mover: its new cell, arrival rank (high 16 bits of cell_count)
//   (scan, k_cell_start) as in the full binning
//   k_inc_place_stayers  per old cell: src of its stayers
//   k_inc_place_movers   per mover: src behind the stayers of its cell
//   k_inc_sort           per cell that received movers: sorted by id
//   k_inc_finalize       per new cell: counts and grid zeroed

// the new index of every old block (one query per block, before the per-block passes)
__global__ void __launch_bounds__(kThreads) k_inc_map(scene_device s) {
  if (!incremental_binning(s)) return;
  const int nold = s.ctr[kCtrUseMasks];
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nold; b += grid_threads()) {
    const uint64_t key = s.old_pk[b];
    s.new_of_old[b] = table_query(s, key, unpack_key(key));
  }
}

// The stayers of one old cell j = b * 512 + c: its slot range in the previous binning and the
// number of its particles that did not move out (the flags of a cell are a few adjacent bytes)
__device__ __forceinline__ int2 prev_cell_range(const scene_device &s, int j) {
  const int b = j >> 9, c = j & 511;
  const int cs = s.cell_start_prev[j];
  const int ce = c < 511 ? s.cell_start_prev[j + 1] : s.block_start_prev[b + 1];
  return make_int2(cs, ce);
}

// kFused: within the fused kernel, where the movers are counted in the same phase (the counts are
// added, not stored) and the new block indices are found here
template <bool kFused>
__device__ __forceinline__ void do_inc_stayers(const scene_device &s) {
  if (!incremental_binning(s)) return;
  const int nold = s.ctr[kCtrUseMasks], nb = s.ctr[kCtrBlocks];
  const long long cells = (long long)nold * 512;  // a warp covers 32 cells of one block
  const int lane = threadIdx.x & 31;
  for (long long j0 = blockIdx.x * (long long)blockDim.x; j0 < cells; j0 += grid_threads()) {
    const long long j = j0 + threadIdx.x;
    const bool in = j < cells;
    int stay = 0, nbi = -1;
    if (kFused && j0 + (threadIdx.x & ~31) < cells) {  // (a warp's cells are of one block)
      const int b = (int)((j0 + (threadIdx.x & ~31)) >> 9);
      if (lane == 0) {
        const uint64_t key = s.old_pk[b];
        nbi = table_query(s, key, unpack_key(key));
        if (((j0 + threadIdx.x) & 511) == 0) s.new_of_old[b] = nbi;
      }
      nbi = __shfl_sync(kFull, nbi, 0);
    }
    if (in) {
      const int2 r = prev_cell_range(s, (int)j);
      int slot = r.x;
      for (; slot + 4 <= r.y; slot += 4) {
        const uint8_t a = s.moved[slot], b1 = s.moved[slot + 1], c = s.moved[slot + 2], d = s.moved[slot + 3];
        stay += (a == 0) + (b1 == 0) + (c == 0) + (d == 0);
      }
      for (; slot < r.y; ++slot) stay += s.moved[slot] == 0;
      if (!kFused) nbi = s.new_of_old[(int)(j >> 9)];
      if (stay > 0xffff) set_status(s.ctr, kStatusCapacity);  // shares its word with the arrivals
      if (nbi >= 0 && nbi < nb) {
        if (!kFused)
          s.cell_count[nbi * 512 + (int)(j & 511)] = stay;
        else if (stay > 0)
          atomicAdd(&s.cell_count[nbi * 512 + (int)(j & 511)], stay);
      } else if (stay > 0)
        set_status(s.ctr, kStatusMissingBlock);
    }
    const int wsum = __reduce_add_sync(kFull, stay);
    if (lane == 0 && wsum > 0 && nbi >= 0 && nbi < nb) atomicAdd(&s.block_count[nbi], wsum);
  }
}
__global__ void __launch_bounds__(kThreads) k_inc_stayers(scene_device s) { do_inc_stayers<false>(s); }

__device__ __forceinline__ void do_inc_movers(const scene_device &s) {
  if (!incremental_binning(s)) return;
  const int nmov = min(s.ctr[kCtrMovers], s.prm.mover_cap);
  const int nb = s.ctr[kCtrBlocks];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nmov; k += grid_threads()) {
    const int slot = s.movers[k];
    int3 c, b;
    int2 pos = make_int2(-1, 0);
    if (particle_cell(s, s.prm.batch ? s.cur.sid[slot] : 0, s.cur.xm[slot], c, b)) {
      const int blk = table_query(s, pack_key(b.x, b.y, b.z), b);
      if (blk >= 0 && blk < nb) {
        const int k32 = blk * 512 + (((c.x - 8 * b.x) << 6) | ((c.y - 8 * b.y) << 3) | (c.z - 8 * b.z));
        const int old = atomicAdd(&s.cell_count[k32], 1 << 16);
        atomicAdd(&s.block_count[blk], 1);
        pos = make_int2(k32, old >> 16);
        if ((old >> 16) >= 0x7fff) set_status(s.ctr, kStatusCapacity);
        // the first arrival lists the cell for k_inc_sort (at most one entry per mover)
        if ((old >> 16) == 0) s.dirty[atomicAdd(&s.ctr[kCtrDirty], 1)] = k32;
      }
    }
    if (pos.x < 0) set_status(s.ctr, kStatusMissingBlock);
    s.mover_pos[k] = pos;
  }
}
__global__ void __launch_bounds__(kThreads) k_inc_movers(scene_device s) { do_inc_movers(s); }

__device__ __forceinline__ void do_inc_place_stayers(const scene_device &s) {
  if (!incremental_binning(s)) return;
  const int nold = s.ctr[kCtrUseMasks], nb = s.ctr[kCtrBlocks];
  const long long cells = (long long)nold * 512;
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < cells; j += grid_threads()) {
    const int nbi = s.new_of_old[(int)(j >> 9)];
    if (nbi < 0 || nbi >= nb) continue;
    const int2 r = prev_cell_range(s, (int)j);
    int dst = s.cell_start[nbi * 512 + (int)(j & 511)];
    // four flags loaded together per round (a cell holds a few adjacent slots)
    for (int slot = r.x; slot < r.y; slot += 4) {
      uint8_t f[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) f[u] = slot + u < r.y ? s.moved[slot + u] : (uint8_t)1;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (f[u] == 0) s.src[dst++] = slot + u;
    }
  }
}
__global__ void __launch_bounds__(kThreads) k_inc_place_stayers(scene_device s) { do_inc_place_stayers(s); }

__device__ __forceinline__ void do_inc_place_movers(const scene_device &s) {
  if (!incremental_binning(s)) return;
  const int nmov = min(s.ctr[kCtrMovers], s.prm.mover_cap);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nmov; k += grid_threads()) {
    const int2 pos = s.mover_pos[k];
    if (pos.x < 0) continue;
    s.src[s.cell_start[pos.x] + (s.cell_count[pos.x] & 0xffff) + pos.y] = s.movers[k];
  }
}
__global__ void __launch_bounds__(kThreads) k_inc_place_movers(scene_device s) { do_inc_place_movers(s); }

// the cells that received movers, in upload-id order (stayers and arrivals merged)
__global__ void __launch_bounds__(kThreads) k_inc_sort(scene_device s) {
  if (!incremental_binning(s)) return;
  const int nd = min(s.ctr[kCtrDirty], s.prm.mover_cap);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nd; k += grid_threads()) {
    const int j = s.dirty[k];
    const int craw = s.cell_count[j];
    const int c = (craw & 0xffff) + (craw >> 16);
    if (c > 1) sort_cell_by_id(s, s.src, s.src, s.cell_start[j], c);
  }
}

__global__ void __launch_bounds__(kThreads) k_inc_finalize(scene_device s) {
  if (!incremental_binning(s)) return;
  const int nb = s.ctr[kCtrBlocks];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    s.ctr[kCtrBinInfo] = min(s.ctr[kCtrMovers], s.prm.mover_cap);
    s.ctr[kCtrMovers] = 0;  // the next G2P lists its movers afresh (k_inc_place_movers has read them)
  }
  const long long cells = (long long)nb * 512;
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < cells; j += grid_threads()) {
    s.cell_count[j] = 0;
    const int b = (int)(j >> 9), cell = (int)(j & 511);
#pragma unroll
    for (int ch = 0; ch < kGridChannels; ++ch) s.grid[((size_t)b * kGridChannels + ch) * 512 + cell] = 0.f;
    if (cell == 0) s.block_count[b] = 0;
  }
}

// ----------------------------------------------------------------- activation and binning in one launch
// The same passes as above in one cooperative kernel, with grid barriers in place of the kernel
// boundaries: eight of them instead of 25 launches.  Scans over few entries (the bitmap's words,
// the blocks) are done by every CTA for itself.  A launch boundary costs about 2.5 us here, a
// grid barrier about 2 us and a cluster barrier a fraction of one, so this is the path wherever the
// passes are short (fused_prepare).
//   kCluster: one cluster of 16 CTAs of 1,024 threads, synchronised by the hardware's cluster barrier;
//   else a cooperative grid of 512-thread CTAs with a barrier in memory.
constexpr int kPrepScan = 4096;  // entries a CTA scans by itself
constexpr int kPrepCluster = 16;
template <bool kCluster>
struct prep_shape {
  static constexpr int kThreads = kCluster ? 1024 : 512;
};

// All CTAs of the (cooperative) grid arrive; false when the wait gave up (kStatusTimeout is set and the
// caller leaves).  `target` counts the arrivals up to and with this barrier.
template <bool kCluster>
__device__ __forceinline__ bool prep_barrier(const scene_device &s, int &target, int *ok) {
  if (kCluster) {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
    return true;
  }
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&s.ctr[kCtrBarrier], 1);
    int seen = 0;
    for (int i = 0; i < (1 << 21); ++i) {
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(&s.ctr[kCtrBarrier]) : "memory");
      if (seen >= target) break;
    }
    __threadfence();
    *ok = seen >= target;
    if (seen < target) set_status(s.ctr, kStatusTimeout);
  }
  __syncthreads();
  return *ok != 0;
}

// Exclusive scan of load(0 .. n) by this CTA into out[0 .. n] (shared memory, n <= kPrepScan)
template <int kPrepThreads, class Load>
__device__ __forceinline__ void prep_scan_local(Load load, int n, int *out, int *sm) {
  const int per = (n + kPrepThreads - 1) / kPrepThreads, lo = min(n, (int)threadIdx.x * per), hi = min(n, lo + per);
  int sum = 0;
  for (int i = lo; i < hi; ++i) sum += load(i);
  int total, run = cta_exclusive_scan<kPrepThreads>(sum, total, sm);
  for (int i = lo; i < hi; ++i) {
    out[i] = run;
    run += load(i);
  }
  if (threadIdx.x == 0) out[n] = total;
  __syncthreads();
}

// The same over many entries, with the whole grid, into out[0 .. n] in global memory (two barriers)
template <bool kCluster, class Load>
__device__ __forceinline__ bool prep_scan_grid(const scene_device &s, Load load, int n, int *out, int *sm, int &target,
                                               int *ok) {
  constexpr int kPrepThreads = prep_shape<kCluster>::kThreads;
  const int chunk = (n + gridDim.x - 1) / gridDim.x;
  const int lo = min(n, (int)blockIdx.x * chunk), hi = min(n, lo + chunk);
  int acc = 0, total;
  for (int i = lo + threadIdx.x; i < hi; i += kPrepThreads) acc += load(i);
  cta_exclusive_scan<kPrepThreads>(acc, total, sm);
  if (threadIdx.x == 0) s.scan_part[blockIdx.x] = total;
  if (!prep_barrier<kCluster>(s, target, ok)) return false;
  int before = 0, run;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += kPrepThreads) before += s.scan_part[i];
  cta_exclusive_scan<kPrepThreads>(before, run, sm);
  for (int base = lo; base < hi; base += kPrepThreads) {
    const int i = base + threadIdx.x;
    const int ex = cta_exclusive_scan<kPrepThreads>(i < hi ? load(i) : 0, total, sm);
    if (i < hi) out[i] = run + ex;
    run += total;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = run;
  return prep_barrier<kCluster>(s, target, ok);
}

// cell starts, a warp per block (16 consecutive cells a lane), and the work order
__device__ __forceinline__ void prep_cell_start(const scene_device &s, int nb, const int *block_start) {
  const int lane = threadIdx.x & 31;
  for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nb; b += grid_threads() >> 5) {
    const int4 *in = reinterpret_cast<const int4 *>(s.cell_count + (size_t)b * 512) + 4 * lane;
    int c[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int4 v = in[q];
      c[4 * q] = v.x, c[4 * q + 1] = v.y, c[4 * q + 2] = v.z, c[4 * q + 3] = v.w;
    }
    int sum = 0;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int n = (c[q] & 0xffff) + (c[q] >> 16);  // counted in place + arrivals (k_cell_start)
      c[q] = sum;
      sum += n;
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, x, o);
      if (lane >= o) x += y;
    }
    const int total = __shfl_sync(kFull, x, 31), base = block_start[b] + x - sum;
    int4 *out = reinterpret_cast<int4 *>(s.cell_start + (size_t)b * 512) + 4 * lane;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      out[q] = make_int4(base + c[4 * q], base + c[4 * q + 1], base + c[4 * q + 2], base + c[4 * q + 3]);
    if (lane == 0) {
      s.bmask[b] = 0u;  // (G2P's items add to it)
      if (total >= kBigBlock)
        s.work_order[atomicAdd(&s.ctr[kCtrOrderFront], 1)] = b;
      else if (total > 0)
        s.work_order[nb - 1 - atomicAdd(&s.ctr[kCtrOrderBack], 1)] = b;
    }
  }
}

template <bool kCluster>
__global__ void __launch_bounds__(prep_shape<kCluster>::kThreads, kCluster ? 1 : 2)
    k_prepare(scene_device s, int activate, int bin) {
  constexpr int kPrepThreads = prep_shape<kCluster>::kThreads;
  __shared__ int sm[kPrepThreads / 32 + 1];
  __shared__ int s_ok;
  __shared__ int s_scan[kPrepScan + 1];
  int target = 0;
  // (a wait that gives up leaves through the end, where the barrier counters are cleared)
  do {
    if (activate) {
      do_begin(s);
      if (!prep_barrier<kCluster>(s, target, &s_ok)) break;
      do_insert_particle_blocks(s);
      do_insert_moved_blocks(s);
      if (!prep_barrier<kCluster>(s, target, &s_ok)) break;
      do_enlarge(s);
      if (!prep_barrier<kCluster>(s, target, &s_ok)) break;
      int nb, words;
      block_totals(s, blockIdx.x == 0 && threadIdx.x == 0, nb, words);
      do_bitmap_set(s, words > 0 ? nb : 0);
      if (!prep_barrier<kCluster>(s, target, &s_ok)) break;
      const load_popc popc{s.bitmap};
      if (words <= kPrepScan) {
        prep_scan_local<kPrepThreads>(popc, words, s_scan, sm);
        do_assign_ranks(s, words > 0 ? nb : 0, s_scan);
      } else {
        if (!prep_scan_grid<kCluster>(s, popc, words, s.word_prefix, sm, target, &s_ok)) break;
        do_assign_ranks(s, nb, s.word_prefix);
      }
      if (!prep_barrier<kCluster>(s, target, &s_ok)) break;
      do_neighbors(s);
    }
    if (bin) {
      // (the neighbours above and the counts below both only need the ranks)
      do_bin_count(s);
      do_inc_stayers<true>(s);
      do_inc_movers(s);
      if (!prep_barrier<kCluster>(s, target, &s_ok)) break;
      const int nb = s.ctr[kCtrBlocks];
      const load_int count{s.block_count};
      if (nb < kPrepScan) {
        prep_scan_local<kPrepThreads>(count, nb, s_scan, sm);
        if (blockIdx.x == 0)
          for (int i = threadIdx.x; i <= nb; i += kPrepThreads) s.block_start[i] = s_scan[i];
        prep_cell_start(s, nb, s_scan);
      } else {
        if (!prep_scan_grid<kCluster>(s, count, nb, s.block_start, sm, target, &s_ok)) break;
        prep_cell_start(s, nb, s.block_start);
      }
      if (!prep_barrier<kCluster>(s, target, &s_ok)) break;
      const bool inc = incremental_binning(s);
      do_bin_scatter(s);
      do_inc_place_stayers(s);
      do_inc_place_movers(s);
      // the grid starts zeroed
      const long long quads = (long long)nb * (kGridChannels * 512 / 4);
      for (long long q = blockIdx.x * (long long)kPrepThreads + threadIdx.x; q < quads; q += grid_threads())
        reinterpret_cast<float4 *>(s.grid)[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!prep_barrier<kCluster>(s, target, &s_ok)) break;
      // the cells' lists by upload id (incremental: those that received movers), and the counts
      // zeroed for the next binning; a cell's length from the starts
      auto cell_len = [&](int j) {
        return ((j & 511) < 511 ? s.cell_start[j + 1] : s.block_start[(j >> 9) + 1]) - s.cell_start[j];
      };
      const int t0 = blockIdx.x * kPrepThreads + threadIdx.x;
      if (inc) {
        const int nd = min(s.ctr[kCtrDirty], s.prm.mover_cap);
        for (int k = t0; k < nd; k += grid_threads()) {
          const int j = s.dirty[k], c = cell_len(j);
          if (c > 1) sort_cell_by_id(s, s.src, s.src, s.cell_start[j], c);
        }
      }
      const long long cells = (long long)nb * 512;
      for (long long j = t0; j < cells; j += grid_threads()) {
        if (!inc) sort_cell_by_id(s, s.tmp, s.src, s.cell_start[j], cell_len((int)j));
        s.cell_count[j] = 0;
        if ((j & 511) == 0) s.block_count[j >> 9] = 0;
      }
      if (t0 == 0) {
        s.ctr[kCtrBinInfo] = inc ? min(s.ctr[kCtrMovers], s.prm.mover_cap) : -1;
        s.ctr[kCtrMovers] = 0;  // the next G2P lists its movers afresh
      }
    }
  } while (false);
  if (kCluster) return;
  // the last CTA to leave clears the barrier for the next launch
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&s.ctr[kCtrBarrierExit], 1) == (int)gridDim.x - 1) {
      s.ctr[kCtrBarrier] = 0;
      s.ctr[kCtrBarrierExit] = 0;
    }
  }
}

// ----------------------------------------------------------------- P2G
// Work items are (block, range of x planes); a CTA of four warps takes one at a time.  Warp w
// owns the 16 cells y in {2w, 2w + 1}, z in 0..7 of every plane, two lanes per cell: one sums
// the channels (m, p_x), the other (p_y, p_z); the nodes' values are packed pairs.  All particles of
// a cell share its 27 stencil nodes, so a lane keeps 27 pair sums in registers; it walks the
// cells of its (y, z) column along x and the sums slide with it: after each plane the nine
// leading nodes are complete for this column and go to the node plane in shared memory (shared
// atomics), and the other eighteen carry over.  A cell thus adds 9 nodes instead of 27, and the
// node plane, two deep, replaces a halo of the whole block.  Grid channels: m and
// p = sum W (m v + A (x_i - x_p)), the reference's mv + rhs (P2G.hpp:108-125) with
// A = m C - (4 dt/dx^2) tau precomputed by G2P.
//
// The particles come through a ring of S windows per warp: a window holds four ranks of the
// warp's 16 cells, 64 bytes a particle (x|m and the three rows v_d, A_d0..2), fetched with
// 16-byte cp.async in the order of the slot map, so that neighbouring lanes read neighbouring
// particles.  The slot-map entries are loaded one window ahead of the copies.  Warps depend on
// each other only in the node planes (one barrier per plane).
//
// A particle binned in cell c of the block has its stencil origin at c + 1 (SparsityOp.hpp:72-77
// against P2G.hpp:62-66).  Where rounding puts x / dx on the other side of a cell boundary
// (dx not a power of two) its weights are evaluated at f just outside [0.5, 1.5): the quadratic
// B-spline is C1 there, so the difference is of second order in that rounding.
//
// What bounds it: the FMA pipe and instruction issue together, about 300 thread instructions a
// particle (27 nodes x 4 channels x 2 operations in pairs, 108; weights, staging and emission the
// rest); the 68 bytes a particle are 0.31 ms of a 30 M-particle launch.  That launch takes 0.918 ms
// (0.59 of it without the arithmetic of the nodes, 0.17 for the flush).
constexpr int kP2GThreads = 128;
constexpr int kP2GRanksDefault = 8;  // ranks in flight per cell unless tuned: windows of 4, 2 deep
constexpr int kP2GWin = 4;            // ranks per window
constexpr int kP2GRow = 17;           // float4 row of 16 cells, padded (copies of one cell's ranks hit other banks)
constexpr int kP2GField = kP2GWin * kP2GRow;  // float4 of one field of a window
constexpr int kP2GStage = 4 * kP2GField;      // float4 of a window
constexpr int kP2GUnit = kP2GField + kP2GRow; // the mass channel's rows, read one rank past the end
// A warp's share of a node plane: [channel][4 y][12 z] floats (z from 8b; rows 2w .. 2w + 3 of the
// block's ten), the channels padded so that a warp's stores of two channels fall on distinct banks.
// Node planes are kept four deep (two barriers apart).
constexpr int kP2GPlaneRow = 12, kP2GPlaneCh = 4 * kP2GPlaneRow + 4, kP2GPlane = 4 * kP2GPlaneCh;

constexpr size_t p2g_smem_bytes(int ranks) {
  return sizeof(float4) * ((size_t)4 * (ranks / kP2GWin) * kP2GStage + kP2GUnit) + sizeof(float) * 4 * 4 * kP2GPlane +
         sizeof(int) * 2 * 528;
}

// cp.async (sm_80 and later): copies that land in shared memory while the warp computes
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(a), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { cp_async_wait<0>(); }

__device__ __forceinline__ float2 shfl_up2(float2 a, int d) {
  return make_float2(__shfl_up_sync(kFull, a.x, d), __shfl_up_sync(kFull, a.y, d));
}
__device__ __forceinline__ float2 shfl_down2(float2 a, int d) {
  return make_float2(__shfl_down_sync(kFull, a.x, d), __shfl_down_sync(kFull, a.y, d));
}
__device__ __forceinline__ float2 shfl_xor2(float2 a, int d) {
  return make_float2(__shfl_xor_sync(kFull, a.x, d), __shfl_xor_sync(kFull, a.y, d));
}
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// acc + w v as two scalar operations
__device__ __forceinline__ float2 add_scaled(float2 acc, float w, float2 v) {
  return make_float2(fmaf(w, v.x, acc.x), fmaf(w, v.y, acc.y));
}

// Twice the quadratic B-spline weights (InterpolationKernel.hpp:93-130) of the nodes 0, 1, 2 of a
// stencil for nh = 1 - f, the distance from the particle to the middle node in cells.  (The factor
// two drops the halvings; it is a power of two, so the products of three such weights with data
// scaled by 1/8 round as the plain ones do.)
__device__ __forceinline__ void bspline_weights(float nh, float *w) {
  const float t = nh + 0.5f, g = 0.5f - nh;
  w[0] = t * t;
  w[1] = fmaf(-2.f * nh, nh, 1.5f);
  w[2] = g * g;
}

// Twice the node weights of the cell-centric pair (P2C2GTransfer): a particle's tent weights to
// the centers of its two cells per axis, 1/2 - fx and 1/2 + fx with fx = x/dx - floor(x/dx + 1/2),
// each passed half to either corner, over the nodes base .. base + 2 (base = floor(x/dx + 1/2)
// - 1, fx = -nh).
__device__ __forceinline__ void cell_weights(float nh, float *w) {
  w[0] = nh + 0.5f;
  w[1] = 1.f;
  w[2] = 0.5f - nh;
}

// Parts a block's eight x planes are split into (work items of 8 / parts planes each): one where
// the blocks alone fill the chip several times over, more where they do not (a block's particles
// would otherwise be one CTA's serial work while other SMs idle).
__device__ __forceinline__ int plane_parts(int nb, int ctas) {
  return nb >= 4 * ctas ? 1 : nb * 2 >= 4 * ctas ? 2 : nb * 4 >= 4 * ctas ? 4 : 8;
}

// kCell: P2C2GTransfer of the cell-centric pair (below) with the pair's node weights and affine
// term; `rows` holds v and the affine term (A = m C - (4 dt/dx^2) tau for APIC), with_mass = 0
// leaves the mass channel and the m v term out.  S windows in the ring (the staging depth of the
// tuner: 8, 12 or 16 ranks).  kDof: the second half of G2P2G (below), which adds the three vector
// channels to the node-major dof vector fout (ndofs entries).
template <bool kCell, int S, bool kDof = false>
__global__ void __launch_bounds__(kP2GThreads, 4)
    k_p2g(scene_device s, const float4 *rows, int with_mass, float *fout, long long ndofs, const int *skip) {
  extern __shared__ __align__(16) float4 p2g_smem[];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  float4 *const ring = p2g_smem + w * S * kP2GStage;
  float4 *const unit = p2g_smem + 4 * S * kP2GStage;  // (1, 0, 0, 0): the mass channel's row
  float *const plane = reinterpret_cast<float *>(unit + kP2GUnit);
  // per item parity: the block's 512 cell starts and its end, its neighbours and its key
  int *const meta = reinterpret_cast<int *>(plane + 16 * kP2GPlane);
  constexpr int kMeta = 528, kMetaEnd = 512, kMetaKey = 514, kMetaNbr = 516;
  __shared__ int s_item[2];
  __shared__ unsigned char s_hot[4][4];  // [node plane][warp]: the warp added to it
  const scene_params &prm = s.prm;
  const int nb = s.ctr[kCtrBlocks], front = s.ctr[kCtrOrderFront], nwork = work_blocks(s);
  if (kDof && ((skip && *skip) || (long long)nb * 1536 > ndofs)) return;  // (k_force_rows sets the status)
  const int parts = plane_parts(nwork, gridDim.x), nx = 8 / parts, items = nwork * parts;
  int *const counter = &s.ctr[kCtrWork + (kDof ? kWorkForceScatter : kWorkP2G)];
  for (int q = t; q < kP2GUnit; q += kP2GThreads) unit[q] = make_float4(1.f, 0.f, 0.f, 0.f);
  for (int q = t; q < 16 * kP2GPlane; q += kP2GThreads) plane[q] = 0.f;

  auto fetch_meta = [&](int *m, int b) {
    cp_async16(m + 4 * t, s.cell_start + (size_t)b * 512 + 4 * t);
    if (t == 0) cp_async4(m + kMetaEnd, s.block_start + b + 1);
    if (t < 2) {
      cp_async16(m + kMetaNbr + 4 * t, s.nbr + (size_t)b * 8 + 4 * t);
      cp_async4(m + kMetaKey + t, reinterpret_cast<const int *>(s.blk_pk + b) + t);
    }
    cp_async_commit();
  };

  int ahead = 0;  // thread 0: the item after next
  if (t == 0) {
    s_item[0] = atomicAdd(counter, 1);
    ahead = atomicAdd(counter, 1);
  }
  __syncthreads();
  int item = s_item[0];
  if (item < items) fetch_meta(meta, work_block(s, front, nb, item / parts));
  // the lane's cell column, channels and constants
  const int cell16 = lane & 15, pair = lane >> 4;
  const int ly = 2 * w + (cell16 >> 3), lz = cell16 & 7;
  // the weights below are twice the stencil's, so the data carry 1/8
  const float2 dx8 = dup2(0.125f * prm.dx);
  const float mscale = with_mass ? 0.125f : 0.f;
  // where the lane stores the node sums it ends up with: row 2 (ly & 1), node z = lz + 1 from 8b
  float *const emit0 = plane + w * kP2GPlane + 2 * pair * kP2GPlaneCh + 2 * (ly & 1) * kP2GPlaneRow + lz + 1;
  // the copies of a window: ranks lane & 3 of the cells lane >> 2 and (lane >> 2) + 8
  const int cp_cell = lane >> 2, cp_rank = lane & 3;
  float4 *const cp_dst = ring + cp_rank * kP2GRow + cp_cell;

  for (int par = 0; item < items; par ^= 1) {
    if (t == 0) {
      s_item[par ^ 1] = ahead;
      ahead = atomicAdd(counter, 1);
    }
    cp_async_wait_all();
    __syncthreads();  // this item's starts are in place; the last item is done with the other set
    const int *const cs = meta + par * kMeta;
    const int next = s_item[par ^ 1];
    const int next_b = next < items ? work_block(s, front, nb, next / parts) : -1;
    const int x0 = item % parts * nx, x1 = x0 + nx;
    if (cs[x0 * 64] == cs[x1 * 64]) {  // (cs[512] is the block's end)
      if (next_b >= 0) fetch_meta(meta + (par ^ 1) * kMeta, next_b);
      item = next;
      continue;
    }
    const uint64_t key = (uint64_t)(uint32_t)cs[kMetaKey] | ((uint64_t)(uint32_t)cs[kMetaKey + 1] << 32);
    const int3 bk = local_block(prm, unpack_key(key));
    // the stencils' middle nodes
    const float by = (float)(bk.y * 8 + ly + 2), bz = (float)(bk.z * 8 + lz + 2);

    // ---- the ring's producers: slot-map entries (one window ahead), then the copies
    int lx = x0 - 1, lrank = 0, lmax = 0;  // the window whose slot-map entries are loaded next
    int src0 = -1, src1 = -1;
    int fill = 0;  // ring stage the next copies go to
    const int *const mycells = cs + 16 * w;
    auto load_src = [&]() {
      while (lrank >= lmax && lx < x1) {  // next plane with particles in the warp's cells
        lrank = 0;
        lmax = 0;
        if (++lx < x1) {
          const int c = lx * 64 + cell16;
          lmax = __reduce_max_sync(kFull, mycells[c + 1] - mycells[c]);
        }
      }
      src0 = src1 = -1;
      if (lx < x1) {
        const int c = lx * 64 + cp_cell;
        const int a = mycells[c] + lrank + cp_rank, b = mycells[c + 8] + lrank + cp_rank;
        if (a < mycells[c + 1]) src0 = s.src[a];
        if (b < mycells[c + 9]) src1 = s.src[b];
        lrank += kP2GWin;
      }
    };
    auto copy = [&]() {
      float4 *const d = cp_dst + fill * kP2GStage;
      if (src0 >= 0) {
        const float4 *const r = rows + row_at(0, src0);
        cp_async16(d, s.cur.xm + src0);
        cp_async16(d + kP2GField, r);
        cp_async16(d + 2 * kP2GField, r + 32);
        cp_async16(d + 3 * kP2GField, r + 64);
      }
      if (src1 >= 0) {
        const float4 *const r = rows + row_at(0, src1);
        cp_async16(d + 8, s.cur.xm + src1);
        cp_async16(d + 8 + kP2GField, r);
        cp_async16(d + 8 + 2 * kP2GField, r + 32);
        cp_async16(d + 8 + 3 * kP2GField, r + 64);
      }
      cp_async_commit();
      fill = fill + 1 == S ? 0 : fill + 1;
    };
    load_src();
#pragma unroll
    for (int k = 0; k < S - 1; ++k) {
      copy();
      load_src();
    }

    float2 acc[27];
#pragma unroll
    for (int n = 0; n < 27; ++n) acc[n] = make_float2(0.f, 0.f);
    int hot = 0;    // planes until the carried sums are all zero
    int drain = 0;  // ring stage consumed next
    // planes go two at a time: one barrier, and a warp may run ahead of the others within them
#pragma unroll 1
    for (int p0 = 0; p0 < nx + 2; p0 += 2) {
      const float *const pl0 = plane + (p0 & 2) * 4 * kP2GPlane;
      if (p0 == 2 && next_b >= 0) fetch_meta(meta + (par ^ 1) * kMeta, next_b);
#pragma unroll 1
      for (int p = p0; p < min(p0 + 2, nx + 2); ++p) {
        if (p < nx) {
          const int c = (x0 + p) * 64 + cell16;
          const int cnt = mycells[c + 1] - mycells[c];
          const int maxc = __reduce_max_sync(kFull, cnt);
          const float bx = (float)(bk.x * 8 + x0 + p + 2);
          if (maxc > 0) hot = 3;
#pragma unroll 1
          for (int r0 = 0; r0 < maxc; r0 += kP2GWin) {
            cp_async_wait<S - 2>();
            __syncwarp();  // the window has landed for every lane, the stage before it is free
            copy();
            load_src();
            const float4 *const st = ring + drain * kP2GStage + cell16;
            const float4 *const pa = pair ? st + 2 * kP2GField : unit;
            const float4 *const pb = pair ? st + 3 * kP2GField : st + kP2GField;
            drain = drain + 1 == S ? 0 : drain + 1;
            const int rn = min(cnt - r0, kP2GWin);
            float4 xm = st[0], ra = pa[0], rb = pb[0];
#pragma unroll 1
            for (int r = 0; r < rn; ++r) {
              // the next rank's data load while this one is summed (the row behind the last is
              // the next field's, read and not used)
              const float4 xm_n = st[(r + 1) * kP2GRow], ra_n = pa[(r + 1) * kP2GRow], rb_n = pb[(r + 1) * kP2GRow];
              float X[3];
              if (kCell) {  // the index bucket floor(x * (1/dx) + 1/2) as the binning keys it
                X[0] = xm.x * prm.inv_dx, X[1] = xm.y * prm.inv_dx, X[2] = xm.z * prm.inv_dx;
              } else {
                X[0] = over_dx(prm, xm.x), X[1] = over_dx(prm, xm.y), X[2] = over_dx(prm, xm.z);
              }
              const float hx = bx - X[0], hy = by - X[1], hz = bz - X[2];
              // W (qm + (ii - 1) ax + (jj - 1) ay + (kk - 1) az): qm the momentum the middle node
              // would take, a the affine terms of one cell
              const float2 ax = mul2(make_float2(ra.y, rb.y), dx8), ay = mul2(make_float2(ra.z, rb.z), dx8),
                           az = mul2(make_float2(ra.w, rb.w), dx8);
              float2 q = mul2(dup2(xm.w * mscale), make_float2(ra.x, rb.x));
              q = fma2(ax, dup2(hx), q);
              q = fma2(ay, dup2(hy), q);
              q = fma2(az, dup2(hz), q);
              // A packed operation takes the FMA pipe 2.6 cycles a warp, a scalar one 1.0 to 1.5
              // (measured): packing saves issue slots and costs pipe time.  The balance: the weights, the
              // channels' common factor, and the sums as scalars, the nodes' values in pairs (30 M
              // particles: all in pairs 0.996 ms, scalar weights 0.947, scalar sums too 0.918, all scalar
              // 0.928).
              float wx[3], wy[3], w2[3];
              if (kCell) {
                cell_weights(hx, wx);
                cell_weights(hy, wy);
                cell_weights(hz, w2);
              } else {
                bspline_weights(hx, wx);
                bspline_weights(hy, wy);
                bspline_weights(hz, w2);
              }
              const float2 wz[3] = {dup2(w2[0]), dup2(w2[1]), dup2(w2[2])};
              const float2 minus = dup2(-1.f);
              const float2 c0 = mul2(mul2(wz[0], az), minus), c2 = mul2(wz[2], az);
#pragma unroll
              for (int ii = 0; ii < 3; ++ii) {
                const float2 qi = ii == 0 ? fma2(ax, minus, q) : ii == 1 ? q : add2(q, ax);
#pragma unroll
                for (int jj = 0; jj < 3; ++jj) {
                  const float2 qij = jj == 0 ? fma2(ay, minus, qi) : jj == 1 ? qi : add2(qi, ay);
                  const float wij = wx[ii] * wy[jj];
                  const int n = (ii * 3 + jj) * 3;
                  acc[n] = add_scaled(acc[n], wij, fma2(wz[0], qij, c0));
                  acc[n + 1] = add_scaled(acc[n + 1], wij, mul2(wz[1], qij));
                  acc[n + 2] = add_scaled(acc[n + 2], wij, fma2(wz[2], qij, c2));
                }
              }
              xm = xm_n, ra = ra_n, rb = rb_n;
            }
          }
        }
        // ---- the plane's leading nodes (x0 + p + 1 from 8b) are complete for this column: the
        // warp adds its lanes' 3 x 3 sums up into its 4 rows of 10 nodes by shuffles and stores
        // them (every entry has one writer, so no atomics and nothing to clear)
        if (lane == 0) s_hot[(p0 & 2) + (p & 1)][w] = hot > 0;
        if (hot > 0) {
          --hot;
          float2 lo[3], hi[3];  // of row y + jj: node z + kk summed over the lanes at z; nodes 8 and 9 past lanes 6, 7
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) {
            const float2 a0 = acc[3 * jj], a1 = acc[3 * jj + 1], a2 = acc[3 * jj + 2];
            const float2 u1 = shfl_up2(a1, 1), u2 = shfl_up2(a2, 2), d1 = shfl_down2(a1, 1);
            lo[jj] = a0;
            if (lz >= 1) lo[jj] = add2(lo[jj], u1);
            if (lz >= 2) lo[jj] = add2(lo[jj], u2);
            hi[jj] = lz == 6 ? add2(a2, d1) : a2;  // used by lanes 6 and 7
          }
          // the two y rows of the warp: lanes of the first end with rows 0 and 1, of the second 2 and 3
          const bool second = (ly & 1) != 0;
          const float2 xl = shfl_xor2(second ? lo[0] : lo[2], 8), xh = shfl_xor2(second ? hi[0] : hi[2], 8);
          const float2 r0 = second ? add2(lo[1], xl) : lo[0], r1 = second ? lo[2] : add2(lo[1], xl);
          const float2 h0 = second ? add2(hi[1], xh) : hi[0], h1 = second ? hi[2] : add2(hi[1], xh);
          float *const e = emit0 + ((p0 & 2) + (p & 1)) * 4 * kP2GPlane;
          e[0] = r0.x;
          e[kP2GPlaneCh] = r0.y;
          e[kP2GPlaneRow] = r1.x;
          e[kP2GPlaneCh + kP2GPlaneRow] = r1.y;
          if (lz >= 6) {
            e[2] = h0.x;
            e[kP2GPlaneCh + 2] = h0.y;
            e[kP2GPlaneRow + 2] = h1.x;
            e[kP2GPlaneCh + kP2GPlaneRow + 2] = h1.y;
          }
#pragma unroll
          for (int n = 0; n < 18; ++n) acc[n] = acc[n + 9];
#pragma unroll
          for (int n = 18; n < 27; ++n) acc[n] = make_float2(0.f, 0.f);
        }
      }
      __syncthreads();
      // ---- flush the two planes: each 4 channels x 10 y x 3 quads of z, a row summed over the two
      // warps that share it, by 16-byte reductions into the blocks b + {0,1}^3; the next two planes
      // go to the other buffers, so one barrier is enough
      // (kDof: 10 y x 3 quads, the three vector channels of a quad's nodes as three of them)
      constexpr int kItems = kDof ? 30 : 120;
      for (int it = t; it < kItems * min(2, nx + 2 - p0); it += kP2GThreads) {
        const int p = it < kItems ? 0 : 1, u = it - kItems * p;
        const int hy = u % 30 / 3, quad = u % 3, v = hy >> 1, row = hy & 1;
        const bool lo = v < 4 && s_hot[(p0 & 2) + p][v], hi = v > 0 && s_hot[(p0 & 2) + p][v - 1];
        auto quad_sum = [&](int ch) {
          const float *const at = pl0 + p * 4 * kP2GPlane + ch * kP2GPlaneCh + quad * 4;
          float4 q4 = make_float4(0.f, 0.f, 0.f, 0.f);
          if (lo) q4 = *reinterpret_cast<const float4 *>(at + v * kP2GPlane + row * kP2GPlaneRow);
          if (hi) {
            const float4 o = *reinterpret_cast<const float4 *>(at + (v - 1) * kP2GPlane + (row + 2) * kP2GPlaneRow);
            q4.x += o.x, q4.y += o.y, q4.z += o.z, q4.w += o.w;
          }
          return q4;
        };
        auto nonzero = [](float4 q) { return q.x != 0.f || q.y != 0.f || q.z != 0.f || q.w != 0.f; };
        const int X = x0 + p0 + p + 1, Y = hy + 1;
        const int cell = ((X & 7) << 6) | ((Y & 7) << 3) | ((quad * 4) & 7);
        const int *const to = cs + kMetaNbr + ((X >= 8 ? 4 : 0) | (Y >= 8 ? 2 : 0) | (quad == 2 ? 1 : 0));
        if (kDof) {
          const float4 fx = quad_sum(1), fy = quad_sum(2), fz = quad_sum(3);
          if (nonzero(fx) || nonzero(fy) || nonzero(fz)) {
            if (*to < 0) {
              set_status(s.ctr, kStatusMissingBlock);
            } else {
              float *const dst = fout + ((size_t)*to * 512 + cell) * 3;
              red_add_v4(dst, fx.x, fy.x, fz.x, fx.y);
              red_add_v4(dst + 4, fy.y, fz.y, fx.z, fy.z);
              red_add_v4(dst + 8, fz.z, fx.w, fy.w, fz.w);
            }
          }
        } else {
          const int ch = u / 30;
          const float4 q4 = quad_sum(ch);
          if (nonzero(q4)) {
            if (*to < 0)
              set_status(s.ctr, kStatusMissingBlock);
            else
              red_add_v4(s.grid + ((size_t)*to * kGridChannels + ch) * 512 + cell, q4.x, q4.y, q4.z, q4.w);
          }
        }
      }
    }
    item = next;
  }
}

// ----------------------------------------------------------------- the cell-centric pair
// P2C2GTransfer (simulation/transfer/P2C2G.hpp:27-189) and G2C2PTransfer with its Pre and Post
// passes (G2C2P.hpp:36-278), the fixed-corotated branch.  Both go through the grid cells: the
// particles within dx of a cell's center x_c (per axis) carry the tent weight
// W = prod (1 - |x_c - x_p| / dx), and a cell passes its sums to its 8 corner nodes (and takes
// its velocity from them) with weight 1/8.  A particle's cells are those of the index buckets
// floor(x / dx + 0.5) in {c, c + 1}^3 around it.  The cells are linear stages between the
// particles and the nodes, so each node receives sum_p w_p (m v + A (x_i - x_p)) with the
// composed node weights of cell_weights, and each particle takes sum_i w_i v_i: P2C2G runs as
// the staged P2G kernel with those weights (k_p2g<true>) and G2C2P as a variant of the G2P
// kernel (k_g2p<..., true>), both without per-particle atomics.  (A literal cell-gather P2C2G,
// one thread per cell walking its 8 buckets, measured 5.1 ms against 1.5 ms for P2G on 30 M
// particles: its loads are dependent and scattered.)
//
// Per particle the pair carries x, m, v, F and B (the reference's C attribute) and, written at
// the end of G2C2P for the next P2C2G, the affine term
//   A = (m B - dt V0 P(F) F^T) Dinv,   Dinv_k = 2 / (dx^2 - 2 r_k^2),  r = x - dx round(x / dx),
// columns k scaled (P2C2G.hpp:86-146); it is the same array the APIC path keeps its affine
// momentum in.

// Dinv of one position component, as P2C2G.hpp:87-91 and PostG2C2PTransfer compute it
__device__ __forceinline__ float cell_dinv(const scene_params &p, float x) {
  const float r = x - floorf(x * p.inv_dx + 0.5f) * p.dx;
  return 2.f / (p.dx * p.dx - 2.f * r * r);
}

// The pair's per-particle affine term A of the stored state, in the particle order of cur:
// part 0 the whole term (P2C2GTransfer; the cell-scheme counterpart of k_prime), 1 the momentum
// part m B Dinv (P2C2GTransferMomentum), 2 the force part -dt V0 P F^T Dinv (P2C2GTransferForce).
__global__ void __launch_bounds__(kThreads) k_cell_affine(scene_device s, int part, float4 *out) {
  if (part == 0 && blockIdx.x == 0 && threadIdx.x == 0) s.ctr[kCtrMaskFrom] = 0;
  const scene_params &p = s.prm;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += grid_threads()) {
    const float4 xm = s.cur.xm[i];
    const float dinv[3] = {cell_dinv(p, xm.x), cell_dinv(p, xm.y), cell_dinv(p, xm.z)};
    float F[9], tau[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) F[k] = s.cur.F[mat_at(k, i)];
    float pl = 0.f;
    if (part != 1) constitutive_update<false, true>(p.mat, F, pl, tau);
    float A[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const float mB = part == 2 ? 0.f : xm.w * s.cur.C[mat_at(k, i)];
      const float f = part == 1 ? 0.f : p.dt * tau[k];
      A[k] = (mB - f) * dinv[k / 3];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
      out[row_at(d, i)] = make_float4(s.cur.row[row_at(d, i)].x, A[d], A[3 + d], A[6 + d]);
  }
}

// ----------------------------------------------------------------- grid update
// ComputeGridBlockVelocity with the rhs term (v = (mv + rhs)/m + g dt; GridOp.hpp:93-99
// restated) and ApplyBoundaryConditionOnGridBlocks with six planes wall_cells*dx inside
// the unit box (GridOp.hpp:136-161, Collider.h:98-105).
__device__ __forceinline__ void apply_walls(const scene_params &p, const float pos[3], float v[3]) {
  if (p.wall_type == 3) return;
  const float lo = (float)p.wall_cells * p.dx, hi = 1.f - (float)p.wall_cells * p.dx;
#pragma unroll
  for (int w = 0; w < 6; ++w) {
    const int axis = w >> 1;
    const float sgn = (w & 1) ? -1.f : 1.f;
    const float sd = sgn * (pos[axis] - ((w & 1) ? hi : lo));
    if (!(sd < 0.f)) continue;
    if (p.wall_type == 0) {
      v[0] = v[1] = v[2] = 0.f;
    } else {
      const float proj = sgn * v[axis];
      if (p.wall_type == 1 || proj < 0.f) v[axis] = v[axis] - proj * sgn;
    }
  }
}

// the scene's colliders after its walls, then its sparse level sets, each in list order
__device__ __forceinline__ void apply_colliders(const scene_params &p, int count, int nls, const float pos[3],
                                             float v[3]) {
  for (int k = 0; k < count; ++k) collider_resolve(p.colliders[k], pos, v);
  for (int k = 0; k < nls; ++k) levelset_resolve(p.levelsets[k], pos, v);
}

__global__ void __launch_bounds__(kThreads) k_grid_update(scene_device s) {
  const scene_params &p = s.prm;
  const int nb = s.ctr[kCtrBlocks];
  const long long total = (long long)nb * 512;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += grid_threads()) {
    const int b = (int)(t >> 9), cell = (int)(t & 511);
    float *g = s.grid + (size_t)b * kGridChannels * 512 + cell;
    const float m = g[0];
    if (m == 0.f) continue;
    const float inv = 1.f / m;
    float v[3] = {g[512] * inv + p.gravity[0] * p.dt, g[1024] * inv + p.gravity[1] * p.dt,
                  g[1536] * inv + p.gravity[2] * p.dt};
    if (m > 0.f) {
      const int3 k = local_block(p, unpack_key(s.blk_pk[b]));
      const float pos[3] = {((float)k.x * 8.f + (float)(cell >> 6)) * p.dx,
                            ((float)k.y * 8.f + (float)((cell >> 3) & 7)) * p.dx,
                            ((float)k.z * 8.f + (float)(cell & 7)) * p.dx};
      apply_walls(p, pos, v);
    }
    g[512] = v[0];
    g[1024] = v[1];
    g[1536] = v[2];
  }
}

// The scene's colliders and level sets, after the walls of k_grid_update, on every node with
// positive mass (their own launch, so that k_grid_update keeps its registers; without colliders
// every CTA returns at once).
__global__ void __launch_bounds__(kThreads) k_grid_boundaries(scene_device s) {
  const scene_params &p = s.prm;
  const int ncol = p.ncolliders ? min(*p.ncolliders, kMaxColliders) : 0;
  const int nls = p.nlevelsets ? min(*p.nlevelsets, kMaxLevelsets) : 0;
  if (ncol + nls == 0) return;
  const long long total = (long long)s.ctr[kCtrBlocks] * 512;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += grid_threads()) {
    const int b = (int)(t >> 9), cell = (int)(t & 511);
    float *g = s.grid + (size_t)b * kGridChannels * 512 + cell;
    if (!(g[0] > 0.f)) continue;
    const int3 k = local_block(p, unpack_key(s.blk_pk[b]));
    const float pos[3] = {((float)k.x * 8.f + (float)(cell >> 6)) * p.dx,
                          ((float)k.y * 8.f + (float)((cell >> 3) & 7)) * p.dx,
                          ((float)k.z * 8.f + (float)(cell & 7)) * p.dx};
    float v[3] = {g[512], g[1024], g[1536]};
    apply_colliders(p, ncol, nls, pos, v);
    g[512] = v[0];
    g[1024] = v[1];
    g[1536] = v[2];
  }
}

// ----------------------------------------------------------------- G2P
// One CTA per block (persistent): stage the 12^3 halo of grid velocities in shared memory,
// then per particle gather v and C (G2P.hpp:56-66), advect, update F = (I + dt C) F
// (G2P.hpp:76-78), run the constitutive update and write the particle to its binned slot
// in the next buffer set, so that storage order follows the binning of this substep.
// Particles are taken 32 per warp and the whole warp steps together (lanes past the block's
// end run on a copy of its first particle and write nothing): the SVD's early exit is a
// warp-wide vote, and the learned closure's tensor-core MLP runs across the warp.  While a
// warp computes one batch, cp.async copies its next batch's state (x|m, F, plastic, id) into
// the warp's other prefetch buffer, and the slot map entry of the batch after that is loaded,
// so the gathers of the particle state wait on no load (1.86 -> 1.72 ms on the 30 M-particle
// sand scene).

// trial-state features of the closure: log singular values and the model's three
// material/state features
__device__ __forceinline__ void closure_features(const material_dev &mat, const float *S, float plastic,
                                                 float *feat) {
#pragma unroll
  for (int i = 0; i < 3; ++i) feat[i] = logf(fmaxf(fabsf(S[i]), 1e-4f));
  if (mat.model == 1) {
    feat[3] = mat.friction_deg;
    feat[4] = mat.cohesion;
    feat[5] = plastic;
  } else {
    feat[3] = mat.theta_c;
    feat[4] = mat.theta_s;
    feat[5] = logf(plastic);
  }
}

__device__ __forceinline__ principal_result plain_principal(const material_dev &mat, const float *S,
                                                            const float *l, float plastic) {
  if (mat.model == 1)
    return dp_principal(mat.mu, mat.lambda, mat.cohesion, mat.beta, mat.volume_correction, mat.yield_surface, l,
                        plastic);
  return snow_principal(mat.mu, mat.lambda, mat.hardening, mat.theta_c, mat.theta_s, S, plastic);
}

// columns i and j of (log S, S, U, V) by descending singular value
__device__ __forceinline__ void sort_columns(float *l, float *S, float *U, float *V, int i, int j) {
  if (S[i] >= S[j]) return;
  float t = S[i];
  S[i] = S[j];
  S[j] = t;
  t = l[i];
  l[i] = l[j];
  l[j] = t;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    t = U[3 * i + r];
    U[3 * i + r] = U[3 * j + r];
    U[3 * j + r] = t;
    t = V[3 * i + r];
    V[3 * i + r] = V[3 * j + r];
    V[3 * j + r] = t;
  }
}

// The learned constitutive update (committed ordering), G2P's part.
//
// The network replaces the return-mapping branch, i.e. the projection of a trial state that
// lies outside the yield surface.  Which branch a trial state takes is decided here exactly,
// by the tests of the plain map: Drucker-Prager (compute_stress_sand) projects to the tip when
// tr >= 0 and onto the cone when tr < 0 and dgamma > 0, and is elastic otherwise; snow clamps
// the singular values that leave [1 - theta_c, 1 + theta_s].  Elastic states keep their strain
// and the tip takes its closed form, here.  A projection inside the network's training hull is
// queued (raw features, U, V, S, the plastic state and the binned slot): after G2P the
// tcgen05 kernel runs the network over the queue in 128-row tiles, and k_closure_finish forms
// the projected state, its stress by the model's own formula (Hencky for Drucker-Prager,
// hardened fixed corotated for snow) and writes F, the affine momentum and the plastic state.
// Projections outside the hull, or beyond the queue's capacity, take the plain map here.
// Returns true when the particle was queued (its F, A and plastic state are then not written
// by G2P).
__device__ __forceinline__ bool learned_update(const scene_device &s, const material_dev &mat, const closure_dev &cd,
                                               float *F, float &plastic, float *tau, bool active, int slot, int sid,
                                               int id, float m, const float *Cm, unsigned &all_updates) {
  float U[9], S[3], V[9];
  bool columns = false;
  if (mat.model == 1) columns = svd3_columns<true>(F, U, S, V);
  const unsigned rest = __ballot_sync(kFull, !columns);
  if (!columns) svd3<true>(F, U, S, V, rest);
  float feat[6];
  closure_features(mat, S, plastic, feat);
  bool project = false;
  float H[3], pl_new = plastic;
  if (mat.model == 1) {
    float eps[3], eh[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) eps[i] = feat[i] - mat.cohesion;
    const float sum_eps = eps[0] + eps[1] + eps[2];
    const float tr = sum_eps + plastic;
#pragma unroll
    for (int i = 0; i < 3; ++i) eh[i] = eps[i] - tr / 3.f;
    const float ehn = sqrtf(eh[0] * eh[0] + eh[1] * eh[1] + eh[2] * eh[2]);
    const float smu = 2.f * mat.mu;
    if (tr >= 0.f) {
#pragma unroll
      for (int i = 0; i < 3; ++i) H[i] = mat.cohesion;
      if (mat.volume_correction) pl_new = mat.beta * sum_eps + plastic;
    } else {
      pl_new = 0.f;
      const float dg = ehn + (3.f * mat.lambda + smu) / smu * tr * mat.yield_surface;
      project = dg > 0.f;
#pragma unroll
      for (int i = 0; i < 3; ++i) H[i] = feat[i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      project = project || S[i] < 1.f - mat.theta_c || S[i] > 1.f + mat.theta_s;
      H[i] = feat[i];
    }
  }
  // the network takes the log singular values in descending order, as svd3 sorts them
  if (project && columns) {
    sort_columns(feat, S, U, V, 0, 1);
    sort_columns(feat, S, U, V, 0, 2);
    sort_columns(feat, S, U, V, 1, 2);
  }
  bool in_hull = true;
#pragma unroll
  for (int k = 0; k < kMlpIn; ++k) in_hull = in_hull && feat[k] >= cd.in_min[k] && feat[k] <= cd.in_max[k];
  bool queued = false;
  const bool want = active && project && in_hull;
  const unsigned wq = __ballot_sync(kFull, want);
  all_updates += __popc(__ballot_sync(kFull, active));
  if (wq) {
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == __ffs(wq) - 1) base = atomicAdd(&s.ctr[kCtrQueue], __popc(wq));
    base = __shfl_sync(0xffffffffu, base, __ffs(wq) - 1);
    if (want) {
      const long long k = base + __popc(wq & lanemask_lt());
      if (k < s.aux.qcap) {
        float *fr = s.aux.q_feat + 6 * k;
#pragma unroll
        for (int i = 0; i < 6; ++i) fr[i] = feat[i];
        float *u = s.aux.q_uvs + queue_at(0, k);  // entry e at u[32 e]
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          u[32 * i] = U[i];
          u[32 * (9 + i)] = V[i];
        }
        u[32 * 18] = S[0];
        u[32 * 19] = S[1];
        u[32 * 20] = S[2];
        u[32 * 21] = plastic;
        // the particle's mass and C, for the affine momentum (so that the finish reads only the
        // queue)
        u[32 * 22] = m;
#pragma unroll
        for (int i = 0; i < 9; ++i) u[32 * (23 + i)] = Cm[i];
        s.aux.q_slot[k] = make_int2(slot, sid);
        s.aux.q_id[k] = id;
        queued = true;
      }
    }
  }
  if (queued) return true;
  float Ns[3], tp[3];
  if (active && project) {
    // outside the hull (or a full queue): the plain map
    const principal_result r = plain_principal(mat, S, feat, plastic);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      tp[i] = r.tau[i];
      Ns[i] = r.Ns[i];
    }
    pl_new = r.plastic;
    atomicAdd(&cd.audit[5], 1.0);
  } else if (mat.model == 1) {
#pragma unroll
    for (int i = 0; i < 3; ++i) Ns[i] = expf(H[i]);
    const float trl = H[0] + H[1] + H[2];
#pragma unroll
    for (int i = 0; i < 3; ++i) tp[i] = 2.f * mat.mu * H[i] + mat.lambda * trl;
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i) Ns[i] = S[i];  // inside the clamp box: no projection, Jp unchanged
    const float e = expf(mat.hardening * (1.f - plastic));
    float Ph[3];
    fc_principal(mat.mu * e, mat.lambda * e, Ns, Ph);
#pragma unroll
    for (int i = 0; i < 3; ++i) tp[i] = Ph[i] * Ns[i];
  }
  plastic = pl_new;
  const float d[3] = {tp[0] * mat.volume, tp[1] * mat.volume, tp[2] * mat.volume};
  mul_diag_t(tau, U, d, U);
  mul_diag_t(F, U, Ns, V);
  return false;
}

// The learned update's second part, for the projections the network has given (after the
// tcgen05 pass over the queue): projected state, its stress, F, the affine momentum and the
// plastic state written to the particle's binned slot; one projection in audit_period is
// checked against the plain map (double accumulators).
__global__ void __launch_bounds__(kThreads) k_closure_finish(scene_device s) {
  const closure_dev &cd = s.aux.cd;
  const int nq = (int)min((long long)s.ctr[kCtrQueue], s.aux.qcap);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (nq > 0) atomicAdd(&cd.audit[6], (double)nq);
    // a bounded tensor-core wait of the network pass that gave up is the scene's error too
    if (cd.tc_status && *cd.tc_status) set_status(s.ctr, kStatusTimeout);
  }
  const int substep = s.ctr[kCtrQueueSubstep];  // of the G2P that queued the rows
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nq; k += grid_threads()) {
    const int2 sl = s.aux.q_slot[k];
    const int slot = sl.x;
    const material_dev mat = s.prm.batch ? s.prm.mats[sl.y] : s.prm.mat;
    const float *u = s.aux.q_uvs + queue_at(0, k);
    float U[9], V[9], S[3], feat[6], y[6];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      U[i] = u[32 * i];
      V[i] = u[32 * (9 + i)];
    }
    S[0] = u[32 * 18];
    S[1] = u[32 * 19];
    S[2] = u[32 * 20];
    const float plastic = u[32 * 21];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      feat[i] = s.aux.q_feat[6 * (size_t)k + i];
      y[i] = s.aux.q_out[6 * (size_t)k + i];
    }
    float H[3], Ns[3], tp[3], pl_new;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      H[i] = feat[i] + y[i];
      Ns[i] = expf(H[i]);
    }
    if (mat.model == 1) {
      pl_new = 0.f;  // the cone branch (tr < 0) resets logJp, as compute_stress_sand does
      const float trl = H[0] + H[1] + H[2];
#pragma unroll
      for (int i = 0; i < 3; ++i) tp[i] = 2.f * mat.mu * H[i] + mat.lambda * trl;
    } else {
      pl_new = plastic * (S[0] * S[1] * S[2] / fmaxf(Ns[0] * Ns[1] * Ns[2], 1e-6f));
      const float e = expf(mat.hardening * (1.f - pl_new));
      float Ph[3];
      fc_principal(mat.mu * e, mat.lambda * e, Ns, Ph);
#pragma unroll
      for (int i = 0; i < 3; ++i) tp[i] = Ph[i] * Ns[i];
    }
    const int id = s.aux.q_id[k];
    if (cd.audit_period > 0 &&
        ((unsigned)id * 2654435761u + (unsigned)substep * 40503u) % (unsigned)cd.audit_period == 0u) {
      const principal_result r = plain_principal(mat, S, feat, plastic);
      float d2 = 0.f, t2 = 0.f;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        d2 += (tp[i] - r.tau[i]) * (tp[i] - r.tau[i]);
        t2 += r.tau[i] * r.tau[i];
      }
      const float floor_stress = 1e-4f * (3.f * mat.lambda + 2.f * mat.mu);
      const float rel = sqrtf(d2) / (sqrtf(t2) + floor_stress);
      // non-negative doubles order like their bit patterns, so the max is an integer max
      atomicAdd(&cd.audit[0], 1.0);
      atomicAdd(&cd.audit[1], (double)rel);
      atomicMax(reinterpret_cast<unsigned long long *>(&cd.audit[2]),
                (unsigned long long)__double_as_longlong((double)rel));
      atomicAdd(&cd.audit[3], (double)d2);
      atomicAdd(&cd.audit[4], (double)t2);
    }
    const float dd[3] = {tp[0] * mat.volume, tp[1] * mat.volume, tp[2] * mat.volume};
    float tau[9], Fn[9];
    mul_diag_t(tau, U, dd, U);
    mul_diag_t(Fn, U, Ns, V);
    const float m = u[32 * 22];
#pragma unroll
    for (int c = 0; c < 9; ++c) s.nxt.F[mat_at(c, slot)] = Fn[c];
#pragma unroll
    for (int d = 0; d < 3; ++d) {  // (the row's first entry is the velocity, which G2P wrote)
      float *const r = &s.nxt.row[row_at(d, slot)].x;
#pragma unroll
      for (int c = 0; c < 3; ++c) r[1 + c] = m * u[32 * (23 + 3 * c + d)] - s.prm.kappa * tau[3 * c + d];
    }
    if (s.nxt.plastic) s.nxt.plastic[slot] = pl_new;
  }
}

// Grid to particle: v = sum W v_i and B = sum W v_i (node - f)^T over the stencil whose first node is
// svf[row], by separable sums, z first: per axis the weighted end nodes a, c give the sum a + c + w v
// and the first moment about the middle node c - a, and the moments move to the particle at the
// end (B = M + (1 - f) v).  240 operations; moments about the particle throughout took 300, in pairs
// (fma.rn.f32x2) where x and y allow it (G2P of 30 M particles 1.657 -> 1.608 ms, ten iterations of the
// implicit solve at 3.7 M 4.01 -> 3.92).
__device__ __forceinline__ void gather_velocity(const float4 *svf, int row, const float w[3][3], const float f[3],
                                                float v[3], float B[9]) {
  float mx[3], my[3], mz[3];
#pragma unroll
  for (int ii = 0; ii < 3; ++ii) {
    float t[3], ty[3], tz[3];  // of the plane ii: the sum and the y and z moments
#pragma unroll
    for (int jj = 0; jj < 3; ++jj) {
      const float4 *const n = svf + row + (ii * kHalo + jj) * kHalo;
      const float4 n0 = n[0], n1 = n[1], n2 = n[2];
      const float v0[3] = {n0.x, n0.y, n0.z}, v1[3] = {n1.x, n1.y, n1.z}, v2[3] = {n2.x, n2.y, n2.z};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float a = w[2][0] * v0[d], c = w[2][2] * v2[d];
        const float sum = fmaf(w[2][1], v1[d], a + c), m = c - a;
        if (jj == 0) {
          t[d] = w[1][0] * sum;
          tz[d] = w[1][0] * m;
        } else if (jj == 1) {
          ty[d] = -t[d];
          t[d] = fmaf(w[1][1], sum, t[d]);
          tz[d] = fmaf(w[1][1], m, tz[d]);
        } else {
          ty[d] = fmaf(w[1][2], sum, ty[d]);
          t[d] = fmaf(w[1][2], sum, t[d]);
          tz[d] = fmaf(w[1][2], m, tz[d]);
        }
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (ii == 0) {
        v[d] = w[0][0] * t[d];
        my[d] = w[0][0] * ty[d];
        mz[d] = w[0][0] * tz[d];
      } else {
        if (ii == 1) mx[d] = -v[d];
        else mx[d] = fmaf(w[0][2], t[d], mx[d]);
        v[d] = fmaf(w[0][ii], t[d], v[d]);
        my[d] = fmaf(w[0][ii], ty[d], my[d]);
        mz[d] = fmaf(w[0][ii], tz[d], mz[d]);
      }
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    B[d] = fmaf(1.f - f[0], v[d], mx[d]);
    B[3 + d] = fmaf(1.f - f[1], v[d], my[d]);
    B[6 + d] = fmaf(1.f - f[2], v[d], mz[d]);
  }
}

// Shared memory of k_g2p: the velocity halo, one float4 (vx, vy, vz, 0) per node so that a
// node is one 16-byte load; then per warp
// two prefetch buffers of 32 particles, each laid out as x|m float4[32], F[9][32],
// plastic[32], id[32] (kG2PPrefetch floats).
constexpr int kG2PPrefetch = 4 * 32 + 9 * 32 + 32 + 32;
constexpr size_t g2p_smem_bytes(int nt) {
  return sizeof(float4) * kHaloCells + sizeof(float) * 2 * kG2PPrefetch * (size_t)(nt / 32);
}

// kLearned: the closure's network gives the return map's projections (queued for the tcgen05
// pass, 256 threads only); kBatch: batched scenes (per-block scene material, scene-local block
// origin); NT threads per CTA.  The variants are register-capped for 3 (256 threads) or 5 (128
// threads) resident CTAs per SM: the kernel is issue- and latency-bound, and the extra warps
// hide more latency than the cap costs (2.41 -> 2.09 ms on the 30 M-particle sand scene, no
// spills).
// kCell: G2C2PTransfer with PreG2C2PTransfer and PostG2C2PTransfer (the cell-centric pair,
// fixed corotated), gathered per particle: a particle takes sum_c W_c/8 v_i over the 8 corners i
// of its cells c, i.e. the node weights (3/4 - f/2, 1/2, f/2 - 1/4) per axis over the same three
// nodes as the quadratic stencil (f = x/dx - base, base = floor(x/dx + 1/2) - 1), and
// B = sum W v_i (x_i - x_p)^T; then F <- (I + dt B Dinv) F, x += v dt, and the affine term A of
// the next P2C2G from the new state.
template <bool kLearned, bool kBatch, int NT, bool kCell = false>
__global__ void __launch_bounds__(NT, NT == 256 ? 3 : 5) k_g2p(scene_device s) {
  static_assert(!kLearned || NT == kThreads, "learned G2P runs at 256 threads");
  static_assert(!kCell || (!kLearned && !kBatch), "the cell-centric pair runs on single fixed-corotated scenes");
  extern __shared__ __align__(16) float g2p_smem[];
  float4 *svf = reinterpret_cast<float4 *>(g2p_smem);
  __shared__ int s_b;
  __shared__ material_dev s_mat;
  __shared__ unsigned s_moved;  // the block's move mask
  const scene_params &p = s.prm;
  const int nb = s.ctr[kCtrBlocks], front = s.ctr[kCtrOrderFront], nwork = work_blocks(s);
  const int parts = slot_parts(nwork, gridDim.x);
  const int substep = s.ctr[kCtrSubstep];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    s.ctr[kCtrMaskFrom] = nb;
    if (kLearned) s.ctr[kCtrQueueSubstep] = substep;  // for the closure pass's audit sampling
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float *const pf = g2p_smem + 4 * kHaloCells + warp * 2 * kG2PPrefetch;
  unsigned all_updates = 0;  // learned closure: particle updates of this warp
  // the lane's particle of a batch into prefetch buffer `buf` (lanes past the block's end copy
  // the block's first particle)
  auto prefetch = [&](int buf, int i) {
    float *b = pf + buf * kG2PPrefetch;
    cp_async16(b + 4 * lane, &s.cur.xm[i]);
#pragma unroll
    for (int k = 0; k < 9; ++k) cp_async4(b + 128 + 32 * k + lane, &s.cur.F[mat_at(k, i)]);
    if (s.cur.plastic) cp_async4(b + 416 + lane, &s.cur.plastic[i]);
    cp_async4(b + 448 + lane, &s.cur.id[i]);
    cp_async_commit();
  };
  for (;;) {
    const int w = grab_block(&s.ctr[kCtrWork + kWorkG2P], &s_b);
    if (w >= nwork * parts) break;
    const int b = work_block(s, front, nb, w / parts);
    // this item's part of the block's slots
    const int first = s.block_start[b], last = s.block_start[b + 1];
    const int len = (last - first + 32 * parts - 1) / (32 * parts) * 32;
    const int start = first + w % parts * len, end = min(last, start + len);
    if (start >= end) continue;
    const int3 gk = unpack_key(s.blk_pk[b]);
    if (kBatch && threadIdx.x == 0) s_mat = p.mats[scene_of_key(gk)];
    if (threadIdx.x == 0) s_moved = 0u;
    // halo load: items (hx, hy, quad) over 12 x 12 x 3; each reads four consecutive cells of
    // the three velocity channels (16-byte loads) and writes four float4 nodes
    for (int it = threadIdx.x; it < kHalo * kHalo * 3; it += NT) {
      const int quad = it % 3, hy = (it / 3) % kHalo, hx = it / (3 * kHalo);
      const int t = (hx >= 8 ? 4 : 0) | (hy >= 8 ? 2 : 0) | (quad == 2 ? 1 : 0);
      const int tb = s.nbr[b * 8 + t];
      float4 vx = make_float4(0.f, 0.f, 0.f, 0.f), vy = vx, vz = vx;
      if (tb >= 0) {
        const int cell = ((hx & 7) << 6) | ((hy & 7) << 3) | ((quad * 4) & 7);
        const float *g = s.grid + ((size_t)tb * kGridChannels + 1) * 512 + cell;
        vx = *reinterpret_cast<const float4 *>(g);
        vy = *reinterpret_cast<const float4 *>(g + 512);
        vz = *reinterpret_cast<const float4 *>(g + 1024);
      }
      float4 *dst = svf + (hx * kHalo + hy) * kHalo + quad * 4;
      dst[0] = make_float4(vx.x, vy.x, vz.x, 0.f);
      dst[1] = make_float4(vx.y, vy.y, vz.y, 0.f);
      dst[2] = make_float4(vx.z, vy.z, vz.z, 0.f);
      dst[3] = make_float4(vx.w, vy.w, vz.w, 0.f);
    }
    __syncthreads();
    const int3 bk = kBatch ? local_block(p, gk) : gk;
    const int org[3] = {bk.x * 8, bk.y * 8, bk.z * 8};
    // each warp takes batches of 32 slots; the next batch's particles are copied into the
    // warp's other prefetch buffer while this batch computes
    int buf = 0;
    int i = 0, inext = 0;  // the particle of this batch and of the next
    const int base0 = start + warp * 32;
    if (base0 < end) {
      i = s.src[base0 + lane < end ? base0 + lane : start];
      prefetch(0, i);
      if (base0 + NT < end) inext = s.src[base0 + NT + lane < end ? base0 + NT + lane : start];
    }
    for (int base = start + warp * 32; base < end; base += NT) {
      const int slot = base + lane;
      // every lane of the warp stays in the loop (lanes past the block's end work on a copy of
      // its first particle and store nothing): the SVD's early exit is a warp-wide vote
      const bool active = slot < end;
      const bool more = base + NT < end;  // warp-uniform
      // the batch after next: its slot map load has a whole batch to land
      const int nslot2 = base + 2 * NT + lane;
      const int inext2 = base + 2 * NT < end ? s.src[nslot2 < end ? nslot2 : start] : 0;
      cp_async_wait_all();  // this batch's copies (the only group in flight)
      const float *pb = pf + buf * kG2PPrefetch;
      float4 xm = reinterpret_cast<const float4 *>(pb)[lane];
      const int icur = i;
      if (more) prefetch(buf ^ 1, inext);
      buf ^= 1;
      i = inext;
      inext = inext2;
      int hb[3];
      float w[3][3], f[3];
      if (kCell) {
        // the index bucket floor(x / dx + 1/2) as the binning computes it; its cells are
        // bucket - 1 and bucket, their corners the nodes bucket - 1 .. bucket + 1
        const float X[3] = {xm.x * p.inv_dx, xm.y * p.inv_dx, xm.z * p.inv_dx};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float bs = floorf(X[d] + 0.5f) - 1.f;
          f[d] = X[d] - bs;
          hb[d] = (int)bs - org[d];
          w[d][0] = 0.75f - 0.5f * f[d];
          w[d][1] = 0.5f;
          w[d][2] = 0.5f * f[d] - 0.25f;
        }
      } else {
        const float X[3] = {over_dx(p, xm.x), over_dx(p, xm.y), over_dx(p, xm.z)};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float bs = floorf(X[d] - 0.5f);
          f[d] = X[d] - bs;
          hb[d] = (int)bs - org[d];
          w[d][0] = 0.5f * (1.5f - f[d]) * (1.5f - f[d]);
          const float f1 = f[d] - 1.f;
          w[d][1] = 0.75f - f1 * f1;
          const float f2 = 0.5f + f1;
          w[d][2] = 0.5f * f2 * f2;
        }
      }
      const bool inside = hb[0] >= 0 && hb[0] <= kHalo - 3 && hb[1] >= 0 && hb[1] <= kHalo - 3 &&
                          hb[2] >= 0 && hb[2] <= kHalo - 3;
      if (active && !inside) set_status(s.ctr, kStatusMissingBlock);
      // the cell this slot was binned in, as the binning computed it from the same position
      const int sid = kBatch ? s.cur.sid[icur] : 0;
      const float cold[3] = {floorf(bucket_of(p, xm.x)), floorf(bucket_of(p, xm.y)), floorf(bucket_of(p, xm.z))};
      float vel[3] = {0.f, 0.f, 0.f};
      float B[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // sum W v (node - f)^T
      if (inside) {
        gather_velocity(svf, (hb[0] * kHalo + hb[1]) * kHalo + hb[2], w, f, vel, B);
      }
      float C[9];  // APIC: C = (4/dx^2) sum W v (x_i - x_p)^T; the cell pair: B = sum W v (x_i - x_p)^T
#pragma unroll
      for (int k = 0; k < 9; ++k) C[k] = B[k] * (kCell ? p.dx : p.four_over_dx);
      // the cell pair updates F with B Dinv at the position before the move
      // (PostG2C2PTransfer); APIC with C
      float Cs[9];
      if (kCell) {
        const float dold[3] = {cell_dinv(p, xm.x), cell_dinv(p, xm.y), cell_dinv(p, xm.z)};
#pragma unroll
        for (int k = 0; k < 9; ++k) Cs[k] = C[k] * dold[k / 3];
      } else {
#pragma unroll
        for (int k = 0; k < 9; ++k) Cs[k] = C[k];
      }
      xm.x += vel[0] * p.dt;
      xm.y += vel[1] * p.dt;
      xm.z += vel[2] * p.dt;
      {
        // the block of the new position, as the next activation computes it from the stored
        // x, recorded relative to this block for k_insert_moved_blocks; and whether the
        // particle left the cell it was binned in, for the next (incremental) binning
        // (most particles stay in their cell, where the block is this one)
        unsigned bit = active ? 1u << 13 : 0u;
        bool moved_far = false;
        const bool left_cell = active && !(floorf(bucket_of(p, xm.x)) == cold[0] &&
                                           floorf(bucket_of(p, xm.y)) == cold[1] &&
                                           floorf(bucket_of(p, xm.z)) == cold[2]);
        if (left_cell) {
          int3 c2, b2;
          bit = 0u;
          moved_far = true;
          if (particle_cell(s, sid, xm, c2, b2)) {
            const int ox = b2.x - gk.x, oy = b2.y - gk.y, oz = b2.z - gk.z;
            if (ox >= -1 && ox <= 1 && oy >= -1 && oy <= 1 && oz >= -1 && oz <= 1) {
              bit = 1u << ((ox + 1) * 9 + (oy + 1) * 3 + (oz + 1));
              moved_far = false;
            }
          }  // (else the particle pass of the next activation reports it)
        }
        if (active) s.moved[slot] = (uint8_t)left_cell;
        const unsigned wbits = __reduce_or_sync(kFull, bit);
        if (lane == 0 && wbits) atomicOr(&s_moved, wbits);
        bool bad = moved_far;
        const unsigned leavers = __ballot_sync(kFull, left_cell && !moved_far);
        if (leavers) {
          int base = 0;
          if (lane == 0) base = atomicAdd(&s.ctr[kCtrMovers], __popc(leavers));
          base = __shfl_sync(kFull, base, 0);
          if ((leavers >> lane) & 1u) {
            const int k = base + __popc(leavers & lanemask_lt());
            if (k < p.mover_cap)
              s.movers[k] = slot;
            else
              bad = true;  // list full: the next substep bins every particle
          }
        }
        if (__any_sync(kFull, bad) && lane == 0) s.ctr[kCtrMaskBad] = 1;
      }
      // F, the plastic state and the id from the prefetch buffer, read after the gather so
      // that they take no registers during it (the buffer is next written by the prefetch of
      // the following batch)
      float F[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) F[k] = pb[128 + 32 * k + lane];
      float pl = s.cur.plastic ? pb[416 + lane] : 0.f;
      const int id = __float_as_int(pb[448 + lane]);
      // F <- (I + dt C) F
      float Fn[9];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r)
          Fn[3 * c + r] = F[3 * c + r] + p.dt * (Cs[r] * F[3 * c] + Cs[3 + r] * F[3 * c + 1] + Cs[6 + r] * F[3 * c + 2]);
      // trial-state log for the closure's training set
      if (!kBatch && s.aux.log_period > 0 && active && p.mat.model != 0 &&
          ((unsigned)id + (unsigned)substep) % (unsigned)s.aux.log_period == 0u) {
        float U[9], S[3], V[9], feat[6];
        svd3(Fn, U, S, V);
        closure_features(p.mat, S, pl, feat);
        const unsigned long long k = atomicAdd(s.aux.log_count, 1ull);
        if ((long long)k < s.aux.log_cap)
          for (int q = 0; q < 6; ++q) s.aux.log_buf[6 * k + q] = feat[q];
      }
      float tau[9];
      // in a batch the closure serves the scenes of its material model (uniform over a CTA: a
      // block belongs to one scene); a queued projection's F, A and plastic state are written
      // by k_closure_finish
      bool queued = false;
      if (kLearned && (!kBatch || s_mat.model == s.aux.cd.model))
        queued = learned_update(s, kBatch ? s_mat : p.mat, s.aux.cd, Fn, pl, tau, active, slot, sid, id, xm.w, C,
                                all_updates);
      else
        constitutive_update<true, true>(kBatch ? s_mat : p.mat, Fn, pl, tau);
      if (!active) continue;
      s.nxt.xm[slot] = xm;
      if (p.store_c) {
#pragma unroll
        for (int k = 0; k < 9; ++k) s.nxt.C[mat_at(k, slot)] = C[k];
      }
      if (kCell) {
        // the affine term of the next P2C2G, from the new position and F (P2C2G.hpp:86-146)
        const float dnew[3] = {cell_dinv(p, xm.x), cell_dinv(p, xm.y), cell_dinv(p, xm.z)};
#pragma unroll
        for (int d = 0; d < 3; ++d)
          s.nxt.row[row_at(d, slot)] = make_float4(vel[d], (xm.w * C[d] - p.dt * tau[d]) * dnew[0],
                                                   (xm.w * C[3 + d] - p.dt * tau[3 + d]) * dnew[1],
                                                   (xm.w * C[6 + d] - p.dt * tau[6 + d]) * dnew[2]);
      } else if (!queued) {
#pragma unroll
        for (int d = 0; d < 3; ++d)
          s.nxt.row[row_at(d, slot)] =
              make_float4(vel[d], xm.w * C[d] - p.kappa * tau[d], xm.w * C[3 + d] - p.kappa * tau[3 + d],
                          xm.w * C[6 + d] - p.kappa * tau[6 + d]);
      } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) s.nxt.row[row_at(d, slot)].x = vel[d];
      }
      if (!queued) {
#pragma unroll
        for (int k = 0; k < 9; ++k) s.nxt.F[mat_at(k, slot)] = Fn[k];
        if (s.nxt.plastic) s.nxt.plastic[slot] = pl;
      }
      s.nxt.id[slot] = id;
      if (kBatch) s.nxt.sid[slot] = sid;
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_moved) atomicOr(&s.bmask[b], s_moved);
  }
  if (kLearned && lane == 0 && all_updates) atomicAdd(&s.aux.cd.audit[7], (double)all_updates);
}

// ----------------------------------------------------------------- G2P2G and the implicit system
// G2P2GTransfer (simulation/transfer/G2P2G.hpp:49-142), the force operator of the implicit
// solve (simulation/mpm/ImplicitMPM.hpp:34-61), in two launches:
//  1. k_force_rows: per particle, gather C from the velocity vector, form the trial
//     F = (I + dt C) F, evaluate the stress on a copy of the state (the particle's own is not
//     written) and store (4/dx^2) tau as the particle's affine rows (in the next buffer, which the
//     next G2P overwrites);
//  2. k_p2g<kDof> scatters them, f(node) += W (4/dx^2) tau (x_i - x_p), as P2G does the affine
//     momentum, into the force vector.
// v and f are node-major over the active blocks in canonical order, v[(block*512 + cell)*3 + d]:
// the layout of a dof_view<space, 3> over a Vector (types/View.h:77-168).
//
// One kernel that gathered a chunk of 64 cells, staged its particles in shared memory and added
// their sums to a halo of forces there kept its two halves waiting for each other at 16 barriers a
// block, and used one CTA a block however few there were; the rows cost 96 bytes a particle and
// free both halves of that (ten iterations of the solve: 3.7 M particles 5.12 -> 4.02 ms, 50 k 1.04 ->
// 0.56).  What bounds k_force_rows is instruction issue, as in k_g2p: the gather and the SVD.
__global__ void __launch_bounds__(kThreads, 3)
    k_force_rows(scene_device s, const float *__restrict__ vin, long long ndofs, float dt, const int *skip,
                 float4 *rows) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) float force_smem[];
  float4 *const svf = reinterpret_cast<float4 *>(force_smem);
  __shared__ int s_b;
  const scene_params &p = s.prm;
  const int nb = s.ctr[kCtrBlocks], front = s.ctr[kCtrOrderFront], nwork = work_blocks(s);
  if ((long long)nb * 1536 > ndofs) {
    if (blockIdx.x == 0 && threadIdx.x == 0) set_status(s.ctr, kStatusCapacity);
    return;
  }
  const int parts = slot_parts(nwork, gridDim.x);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float scale = p.four_over_dx * p.inv_dx;
  float *const pf = force_smem + 4 * kHaloCells + warp * 2 * kG2PPrefetch;
  auto prefetch = [&](int buf, int i) {
    float *b = pf + buf * kG2PPrefetch;
    cp_async16(b + 4 * lane, &s.cur.xm[i]);
#pragma unroll
    for (int k = 0; k < 9; ++k) cp_async4(b + 128 + 32 * k + lane, &s.cur.F[mat_at(k, i)]);
    if (s.cur.plastic) cp_async4(b + 416 + lane, &s.cur.plastic[i]);
    cp_async_commit();
  };
  for (;;) {
    const int w = grab_block(&s.ctr[kCtrWork + kWorkForceRows], &s_b);
    if (w >= nwork * parts) break;
    const int b = work_block(s, front, nb, w / parts);
    const int first = s.block_start[b], last = s.block_start[b + 1];
    const int len = (last - first + 32 * parts - 1) / (32 * parts) * 32;
    const int start = first + w % parts * len, end = min(last, start + len);
    if (start >= end) continue;
    // velocity halo: items (hx, hy, quad) over 12 x 12 x 3; four consecutive nodes are 12
    // consecutive floats (three 16-byte loads)
    for (int it = threadIdx.x; it < kHalo * kHalo * 3; it += kThreads) {
      const int quad = it % 3, hy = (it / 3) % kHalo, hx = it / (3 * kHalo);
      const int tb = s.nbr[b * 8 + ((hx >= 8 ? 4 : 0) | (hy >= 8 ? 2 : 0) | (quad == 2 ? 1 : 0))];
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f), c = a, d = a;
      if (tb >= 0) {
        const int cell = ((hx & 7) << 6) | ((hy & 7) << 3) | ((quad * 4) & 7);
        const float4 *g = reinterpret_cast<const float4 *>(vin + ((size_t)tb * 512 + cell) * 3);
        a = g[0];
        c = g[1];
        d = g[2];
      }
      float4 *dst = svf + (hx * kHalo + hy) * kHalo + quad * 4;
      dst[0] = make_float4(a.x, a.y, a.z, 0.f);
      dst[1] = make_float4(a.w, c.x, c.y, 0.f);
      dst[2] = make_float4(c.z, c.w, d.x, 0.f);
      dst[3] = make_float4(d.y, d.z, d.w, 0.f);
    }
    __syncthreads();
    const int3 bk = unpack_key(s.blk_pk[b]);
    const int org[3] = {bk.x * 8, bk.y * 8, bk.z * 8};
    // batches of 32 slots a warp, the next batch's particles copied meanwhile (as in k_g2p); lanes
    // past the end work on a copy of the part's first particle, as the SVD's early exit is a warp vote
    int buf = 0, i = 0, inext = 0;
    const int base0 = start + warp * 32;
    if (base0 < end) {
      i = s.src[base0 + lane < end ? base0 + lane : start];
      prefetch(0, i);
      if (base0 + kThreads < end) inext = s.src[base0 + kThreads + lane < end ? base0 + kThreads + lane : start];
    }
    for (int base = base0; base < end; base += kThreads) {
      const bool active = base + lane < end;
      const int nslot2 = base + 2 * kThreads + lane;
      const int inext2 = base + 2 * kThreads < end ? s.src[nslot2 < end ? nslot2 : start] : 0;
      cp_async_wait_all();
      const float *const pb = pf + buf * kG2PPrefetch;
      const float4 xm = reinterpret_cast<const float4 *>(pb)[lane];
      const int icur = i;
      if (base + kThreads < end) prefetch(buf ^ 1, inext);
      buf ^= 1;
      i = inext;
      inext = inext2;
      const float X[3] = {over_dx(p, xm.x), over_dx(p, xm.y), over_dx(p, xm.z)};
      int hb[3];
      float wt[3][3], f[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float bs = floorf(X[d] - 0.5f);
        f[d] = X[d] - bs;
        hb[d] = (int)bs - org[d];
        wt[d][0] = 0.5f * (1.5f - f[d]) * (1.5f - f[d]);
        const float f1 = f[d] - 1.f;
        wt[d][1] = 0.75f - f1 * f1;
        const float f2 = 0.5f + f1;
        wt[d][2] = 0.5f * f2 * f2;
      }
      const bool inside = hb[0] >= 0 && hb[0] <= kHalo - 3 && hb[1] >= 0 && hb[1] <= kHalo - 3 && hb[2] >= 0 &&
                          hb[2] <= kHalo - 3;
      if (active && !inside) set_status(s.ctr, kStatusMissingBlock);
      float B[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // sum W v (node - f)^T
      if (inside) {
        float vel[3];
        gather_velocity(svf, (hb[0] * kHalo + hb[1]) * kHalo + hb[2], wt, f, vel, B);
      }
      // trial F = (I + dt C) F (G2P2G.hpp:103-105), C = B 4/dx
      float F[9], Fn[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) F[k] = pb[128 + 32 * k + lane];
      float pl = s.cur.plastic ? pb[416 + lane] : 0.f;
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r)
          Fn[3 * c + r] = F[3 * c + r] + dt * p.four_over_dx *
                                             (B[r] * F[3 * c] + B[3 + r] * F[3 * c + 1] + B[6 + r] * F[3 * c + 2]);
      float tau[9];
      constitutive_update<true, false>(p.mat, Fn, pl, tau);
      if (!active) continue;
      // (a particle outside the halo scatters nothing)
#pragma unroll
      for (int d = 0; d < 3; ++d)
        rows[row_at(d, icur)] = inside ? make_float4(0.f, scale * tau[d], scale * tau[3 + d], scale * tau[6 + d])
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// dof entries of the active blocks (nb * 512 * 3), or 0 with the capacity status when the
// caller's vectors are shorter
__device__ __forceinline__ long long dof_count(const scene_device &s, long long ndofs) {
  const long long total = (long long)s.ctr[kCtrBlocks] * 1536;
  if (total <= ndofs) return total;
  if (blockIdx.x == 0 && threadIdx.x == 0) set_status(s.ctr, kStatusCapacity);
  return 0;
}

// mass of the node t = block * 512 + cell
__device__ __forceinline__ float node_mass(const scene_device &s, long long t) {
  return s.grid[(t >> 9) * kGridChannels * 512 + (t & 511)];
}
// the collision response of the scene's walls, colliders and level sets at a node
struct node_boundaries {
  const scene_params &p;
  int ncol, nls;
  __device__ __forceinline__ explicit node_boundaries(const scene_params &prm)
      : p(prm),
        ncol(prm.ncolliders ? min(*prm.ncolliders, kMaxColliders) : 0),
        nls(prm.nlevelsets ? min(*prm.nlevelsets, kMaxLevelsets) : 0) {}
  __device__ __forceinline__ void apply(const scene_device &s, long long t, float v[3]) const {
    const int cell = (int)(t & 511);
    const int3 k = unpack_key(s.blk_pk[t >> 9]);
    const float pos[3] = {((float)k.x * 8.f + (float)(cell >> 6)) * p.dx,
                          ((float)k.y * 8.f + (float)((cell >> 3) & 7)) * p.dx,
                          ((float)k.z * 8.f + (float)(cell & 7)) * p.dx};
    apply_walls(p, pos, v);
    if (ncol + nls > 0) apply_colliders(p, ncol, nls, pos, v);
  }
};

// ImplicitMPMSystem::ForceDtSqrPlusMass (ImplicitMPM.hpp:17-33): where the grid mass of the
// node is positive, out = (f dt^2 + m) dv, with f = out on entry.
__global__ void __launch_bounds__(kThreads) k_implicit_mass(scene_device s, const float *__restrict__ dv,
                                                             float *__restrict__ out, float dt, long long ndofs) {
  const long long total = dof_count(s, ndofs);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += grid_threads()) {
    const long long node = i / 3;
    const float m = s.grid[(node >> 9) * kGridChannels * 512 + (node & 511)];
    if (m > 0.f) out[i] = (out[i] * dt * dt + m) * dv[i];
  }
}

// ImplicitMPMSystem::Projector (ImplicitMPM.hpp:63-97) with the scene's six walls: nodes with
// positive mass get the walls' collision response, all others are zeroed.
__global__ void __launch_bounds__(kThreads) k_implicit_project(scene_device s, float *__restrict__ dof,
                                                                long long ndofs) {
  const node_boundaries bc(s.prm);
  const long long total = dof_count(s, ndofs) / 3;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += grid_threads()) {
    float *v = dof + t * 3;
    if (node_mass(s, t) > 0.f) {
      float vel[3] = {v[0], v[1], v[2]};
      bc.apply(s, t, vel);
      v[0] = vel[0];
      v[1] = vel[1];
      v[2] = vel[2];
    } else {
      v[0] = v[1] = v[2] = 0.f;
    }
  }
}

// ImplicitMPMSystem::DivPernodeMass (ImplicitMPM.hpp:126-137): out = in / m where the grid
// mass is positive; other entries of out are left as they are.
__global__ void __launch_bounds__(kThreads) k_implicit_precondition(scene_device s, const float *__restrict__ in,
                                                                     float *__restrict__ out, long long ndofs) {
  const long long total = dof_count(s, ndofs);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += grid_threads()) {
    const long long node = i / 3;
    const float m = s.grid[(node >> 9) * kGridChannels * 512 + (node & 511)];
    if (m > 0.f) out[i] = in[i] / m;
  }
}

// ConjugateGradient::solve (math/linear/ConjugateGradient.hpp:69-172) on the device.  The
// scalars (r.q, alpha, beta, the stopping test) live in a cg_state in device memory, so no
// step needs the host: every kernel of an iteration returns at once when the solve is finished.
//
// An iteration is four launches: the force operator, and three passes over the nodes that do
// between two dot products all that needs no other node (mass, boundaries and p.Ap; the updates of
// x and r, the preconditioner and r.q; the new direction and a zeroed A p).  The CTA that arrives
// last at a dot product takes its scalars.  The vectors stay in L2 (7 MB each for 3.7 M particles),
// so a pass costs mostly its launch and the reduction: ten iterations and the start, force operator
// included, take 5.11 ms where launches of one operation each took 5.97 (50 k: 1.03 and 1.56; with the fused force operator of the time).
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Adds the CTA's products (floats per thread and warp, doubles from there on) to the dot product;
// true in thread 0 of the CTA that arrives last, with the sum in out and the accumulator cleared.
__device__ __forceinline__ bool cg_dot(float acc, cg_state *cs, double &out) {
  __shared__ double s_sum[kThreads / 32];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = (double)acc;
  __syncthreads();
  if (threadIdx.x != 0) return false;
  double sum = 0.0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) sum += s_sum[w];
  if (sum != 0.0) atomicAdd(&cs->acc, sum);
  __threadfence();
  if (atomicAdd(&cs->arrived, 1u) != gridDim.x - 1) return false;
  __threadfence();
  out = atomicAdd(&cs->acc, 0.0);
  cs->acc = 0.0;
  cs->arrived = 0;
  return true;
}

// the loop head (:118-122): stop at the tolerance or after max_iters iterations
__device__ __forceinline__ void cg_check(cg_state *cs, int max_iters) {
  if (cs->iter >= max_iters || cs->norm <= cs->local_tol) cs->done = 1;
}

// ForceDtSqrPlusMass and Projector on one node: v = the constrained (f dt^2 + m) d, zero off the mass
__device__ __forceinline__ void cg_operator(const scene_device &s, const node_boundaries &bc, long long t, float m,
                                            const float *f, const float *d, float dt, float v[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = (f[3 * t + k] * dt * dt + m) * d[3 * t + k];
  bc.apply(s, t, v);
}

// The solve's start from A x's forces in ap: r = P(b - A x), p = M r, zTrk = r.p, and the tolerance
// min(relTol * norm, tol) (:97-117); A p zeroed for the first iteration's forces.
__global__ void __launch_bounds__(kThreads) k_cg_start(scene_device s, const float *__restrict__ x,
                                                        const float *__restrict__ b, cg_vectors v, long long ndofs,
                                                        float dt, cg_state *cs, float tol, float rel_tol,
                                                        int max_iters) {
  const node_boundaries bc(s.prm);
  const long long total = dof_count(s, ndofs) / 3;
  float acc = 0.f;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += grid_threads()) {
    const float m = node_mass(s, t);
    float r[3] = {0.f, 0.f, 0.f}, q[3] = {0.f, 0.f, 0.f};
    if (m > 0.f) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float ax = (v.ap[3 * t + k] * dt * dt + m) * x[3 * t + k];
        r[k] = b[3 * t + k] - ax;
      }
      bc.apply(s, t, r);
#pragma unroll
      for (int k = 0; k < 3; ++k) q[k] = r[k] / m;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      v.r[3 * t + k] = r[k];
      v.p[3 * t + k] = q[k];
      v.ap[3 * t + k] = 0.f;
      acc += r[k] * q[k];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < 2) s.ctr[kCtrWork + kWorkForceRows + threadIdx.x] = 0;
  double dot;
  if (cg_dot(acc, cs, dot)) {
    const float z = (float)dot;
    cs->ztrk = z;
    cs->norm = sqrtf(z);
    cs->local_tol = fminf(rel_tol * cs->norm, tol);
    cg_check(cs, max_iters);
  }
}

// A p from its forces, and alpha = zTrk / (Ap . p) (:129-134)
__global__ void __launch_bounds__(kThreads) k_cg_apply(scene_device s, cg_vectors v, long long ndofs, float dt,
                                                        cg_state *cs) {
  if (cs->done) return;
  const node_boundaries bc(s.prm);
  const long long total = dof_count(s, ndofs) / 3;
  float acc = 0.f;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += grid_threads()) {
    const float m = node_mass(s, t);
    if (!(m > 0.f)) continue;  // p, r and A p are zero there
    float a[3];
    cg_operator(s, bc, t, m, v.ap, v.p, dt, a);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      v.ap[3 * t + k] = a[k];
      acc += a[k] * v.p[3 * t + k];
    }
  }
  double dot;
  if (cg_dot(acc, cs, dot)) cs->alpha = cs->ztrk / (float)dot;
}

// x = alpha p + x, r = -alpha Ap + r, zTrk = r . M r, beta = zTrk / zTrkLast, norm = sqrt(zTrk),
// one iteration done (:137-170)
__global__ void __launch_bounds__(kThreads) k_cg_update(scene_device s, float *__restrict__ x, cg_vectors v,
                                                         long long ndofs, cg_state *cs, int max_iters) {
  if (cs->done) return;
  const float alpha = cs->alpha;
  const long long total = dof_count(s, ndofs) / 3;
  float acc = 0.f;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += grid_threads()) {
    const float m = node_mass(s, t);
    if (!(m > 0.f)) continue;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const long long i = 3 * t + k;
      x[i] = alpha * v.p[i] + x[i];
      const float r = -alpha * v.ap[i] + v.r[i];
      v.r[i] = r;
      acc += r / m * r;
    }
  }
  double dot;
  if (cg_dot(acc, cs, dot)) {
    const float last = cs->ztrk;
    cs->ztrk = (float)dot;
    cs->beta = cs->ztrk / last;
    cs->norm = sqrtf(cs->ztrk);
    cs->iter += 1;
    cg_check(cs, max_iters);
  }
}

// p = beta p + M r (:163), and the next iteration's A p zeroed
__global__ void __launch_bounds__(kThreads) k_cg_direction(scene_device s, cg_vectors v, long long ndofs,
                                                            const cg_state *cs) {
  if (cs->done) return;
  const float beta = cs->beta;
  const long long total = dof_count(s, ndofs) / 3;
  if (blockIdx.x == 0 && threadIdx.x < 2) s.ctr[kCtrWork + kWorkForceRows + threadIdx.x] = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += grid_threads()) {
    const float m = node_mass(s, t);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const long long i = 3 * t + k;
      if (m > 0.f) v.p[i] = beta * v.p[i] + v.r[i] / m;
      v.ap[i] = 0.f;
    }
  }
}

// ----------------------------------------------------------------- import / export
// scene of upload index i: the last scene whose start is <= i
__device__ __forceinline__ int scene_of_index(const scene_params &p, int i) {
  int lo = 0, hi = p.nscenes;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (p.scene_start[mid] <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}

// The affine term P2G takes of a particle's state, as rows: m C - kappa tau, or the cell pair's
__device__ __forceinline__ void store_rows(const scene_params &p, float4 *row, size_t i, float4 xm, const float *v,
                                           const float *C, const float *tau) {
  float A[9];
  if (p.transfer == kTransferCell) {
    const float dinv[3] = {cell_dinv(p, xm.x), cell_dinv(p, xm.y), cell_dinv(p, xm.z)};
#pragma unroll
    for (int k = 0; k < 9; ++k) A[k] = (xm.w * C[k] - p.dt * tau[k]) * dinv[k / 3];
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) A[k] = xm.w * C[k] - p.kappa * tau[k];
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) row[row_at(d, i)] = make_float4(v[d], A[d], A[3 + d], A[6 + d]);
}

// Arrays with N floats a particle (x, v: 3, C, F: 9) cross between the caller's layout and a warp's
// registers through shared memory, so that consecutive lanes touch consecutive floats: with one
// particle a lane each load or store of a 9-float row spread over 32 sectors (30 M particles:
// upload 4.1 ms, download 2.9 ms).
constexpr int kMoveThreads = 256;
template <int N>
__device__ __forceinline__ void warp_read(const float *src, size_t i0, int cnt, float *buf, float *out) {
  const int lane = threadIdx.x & 31;
  float v[N];
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = 32 * k + lane < N * cnt ? src[N * i0 + 32 * k + lane] : 0.f;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < N; ++k) buf[32 * k + lane] = v[k];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < N; ++k) out[k] = buf[N * lane + k];
}
// particle p of the warp goes to row ids[p]
template <int N>
__device__ __forceinline__ void warp_write(float *dst, const int *ids, int cnt, float *buf, const float *in) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < N; ++k) buf[N * lane + k] = in[k];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int e = 32 * k + lane, p = e / N;
    if (p < cnt) dst[N * (size_t)ids[p] + (e - N * p)] = buf[e];
  }
}

// The caller's arrays into the scene (v, C, F, plastic optional), with the stress of the uploaded
// state: its projected F and plastic state, and the affine term for the first P2G.
__global__ void __launch_bounds__(kMoveThreads) k_import(scene_device s, const float *m, const float *x, const float *v,
                                                         const float *C, const float *F, const float *pl, int n) {
  __shared__ float s_buf[kMoveThreads / 32][9 * 32];
  if (blockIdx.x == 0 && threadIdx.x == 0) s.ctr[kCtrMaskFrom] = 0;  // new particles: no move masks
  const int lane = threadIdx.x & 31;
  float *const buf = s_buf[threadIdx.x >> 5];
  for (int i0 = (blockIdx.x * kMoveThreads + threadIdx.x) & ~31; i0 < n; i0 += grid_threads()) {
    const int cnt = min(32, n - i0), i = i0 + lane;
    const bool active = lane < cnt;
    float xp[3], vp[3] = {0.f, 0.f, 0.f}, Cp[9], Fp[9], tau[9];
    warp_read<3>(x, i0, cnt, buf, xp);
    if (v) warp_read<3>(v, i0, cnt, buf, vp);
#pragma unroll
    for (int k = 0; k < 9; ++k) Cp[k] = 0.f;
    if (C) warp_read<9>(C, i0, cnt, buf, Cp);
    if (F) warp_read<9>(F, i0, cnt, buf, Fp);
    if (!F || !active) {
#pragma unroll
      for (int k = 0; k < 9; ++k) Fp[k] = (k & 3) == 0 ? 1.f : 0.f;
    }
    const int sc = s.prm.batch ? scene_of_index(s.prm, min(i, n - 1)) : 0;
    const material_dev mat = s.prm.batch ? s.prm.mats[sc] : s.prm.mat;
    float plastic = 0.f;
    if (s.cur.plastic) plastic = pl ? (active ? pl[i] : 0.f) : (mat.model == 2 ? 1.f : 0.f);
    // (the lanes of a warp may hold particles of scenes with different models)
    constitutive_update<false, true>(mat, Fp, plastic, tau);
    if (!active) continue;
    const float4 xm = make_float4(xp[0], xp[1], xp[2], m[i]);
    s.cur.xm[i] = xm;
    store_rows(s.prm, s.cur.row, i, xm, vp, Cp, tau);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      s.cur.C[mat_at(k, i)] = Cp[k];
      s.cur.F[mat_at(k, i)] = Fp[k];
    }
    if (s.cur.plastic) s.cur.plastic[i] = plastic;
    s.cur.id[i] = i;
    if (s.prm.batch) s.cur.sid[i] = sc;
  }
}

__global__ void k_import_tv(scene_device s, const float *base, int nchn, int om, int ox, int ov,
                            int oC, int oF, int opl, int n) {
  const float plastic_default = s.prm.mat.model == 2 ? 1.f : 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += grid_threads()) {
    const size_t tile = (size_t)(i / 32) * nchn * 32 + (i % 32);
    auto at = [&](int chn) { return base[tile + (size_t)chn * 32]; };
    s.cur.xm[i] = make_float4(at(ox), at(ox + 1), at(ox + 2), at(om));
#pragma unroll
    for (int d = 0; d < 3; ++d) s.cur.row[row_at(d, i)] = make_float4(ov >= 0 ? at(ov + d) : 0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      s.cur.C[mat_at(k, i)] = oC >= 0 ? at(oC + k) : 0.f;
      s.cur.F[mat_at(k, i)] = oF >= 0 ? at(oF + k) : ((k & 3) == 0 ? 1.f : 0.f);
    }
    if (s.cur.plastic) s.cur.plastic[i] = opl >= 0 ? at(opl) : plastic_default;
    s.cur.id[i] = i;
  }
}

// stress of the stored state; A = m C - kappa tau (what the previous G2P would have written)
__global__ void k_prime(scene_device s) {
  if (blockIdx.x == 0 && threadIdx.x == 0) s.ctr[kCtrMaskFrom] = 0;  // new particles: no move masks
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.prm.n; i += grid_threads()) {
    float F[9], tau[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) F[k] = s.cur.F[mat_at(k, i)];
    float pl = s.cur.plastic ? s.cur.plastic[i] : 0.f;
    if (s.prm.batch)
      constitutive_update<false, true>(s.prm.mats[s.cur.sid[i]], F, pl, tau);
    else
      constitutive_update<false, true>(s.prm.mat, F, pl, tau);
    const float m = s.cur.xm[i].w;
    float A[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      s.cur.F[mat_at(k, i)] = F[k];
      A[k] = m * s.cur.C[mat_at(k, i)] - s.prm.kappa * tau[k];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
      s.cur.row[row_at(d, i)] = make_float4(s.cur.row[row_at(d, i)].x, A[d], A[3 + d], A[6 + d]);
    if (s.cur.plastic) s.cur.plastic[i] = pl;
  }
}

__global__ void __launch_bounds__(kMoveThreads) k_export(scene_device s, float *m, float *x, float *v, float *C,
                                                         float *F, float *pl) {
  __shared__ float s_buf[kMoveThreads / 32][9 * 32];
  __shared__ int s_id[kMoveThreads / 32][32];
  const int n = s.prm.n, lane = threadIdx.x & 31;
  float *const buf = s_buf[threadIdx.x >> 5];
  int *const ids = s_id[threadIdx.x >> 5];
  for (int i0 = (blockIdx.x * kMoveThreads + threadIdx.x) & ~31; i0 < n; i0 += grid_threads()) {
    const int cnt = min(32, n - i0), i = min(i0 + lane, n - 1);
    const int o = s.cur.id[i];
    const float4 xm = s.cur.xm[i];
    float vp[3], Mp[9], Np[9];
#pragma unroll
    for (int d = 0; d < 3; ++d) vp[d] = v ? s.cur.row[row_at(d, i)].x : 0.f;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      Mp[k] = C ? s.cur.C[mat_at(k, i)] : 0.f;
      Np[k] = F ? s.cur.F[mat_at(k, i)] : 0.f;
    }
    __syncwarp();
    ids[lane] = o;
    const float xp[3] = {xm.x, xm.y, xm.z};
    if (x) warp_write<3>(x, ids, cnt, buf, xp);
    if (v) warp_write<3>(v, ids, cnt, buf, vp);
    if (C) warp_write<9>(C, ids, cnt, buf, Mp);
    if (F) warp_write<9>(F, ids, cnt, buf, Np);
    if (lane < cnt) {
      if (m) m[o] = xm.w;
      if (pl) pl[o] = s.cur.plastic ? s.cur.plastic[i] : 0.f;
    }
  }
}

__global__ void k_export_tv(scene_device s, float *base, int nchn, int om, int ox, int ov, int oC,
                            int oF, int opl) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.prm.n; i += grid_threads()) {
    const int o = s.cur.id[i];
    const size_t tile = (size_t)(o / 32) * nchn * 32 + (o % 32);
    auto at = [&](int chn) -> float & { return base[tile + (size_t)chn * 32]; };
    const float4 xm = s.cur.xm[i];
    const float vv[3] = {s.cur.row[row_at(0, i)].x, s.cur.row[row_at(1, i)].x, s.cur.row[row_at(2, i)].x};
    if (om >= 0) at(om) = xm.w;
    if (ox >= 0) {
      at(ox) = xm.x;
      at(ox + 1) = xm.y;
      at(ox + 2) = xm.z;
    }
    if (ov >= 0) {
      at(ov) = vv[0];
      at(ov + 1) = vv[1];
      at(ov + 2) = vv[2];
    }
    for (int k = 0; k < 9; ++k) {
      if (oC >= 0) at(oC + k) = s.cur.C[mat_at(k, i)];
      if (oF >= 0) at(oF + k) = s.cur.F[mat_at(k, i)];
    }
    if (opl >= 0) at(opl) = s.cur.plastic ? s.cur.plastic[i] : 0.f;
  }
}

__global__ void k_export_order(scene_device s, int *order) {
  // order[slot] = upload id of the particle that the binning placed in `slot`
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < s.prm.n; t += grid_threads())
    order[t] = s.cur.id[s.src[t]];
}

__global__ void k_svd_batch(const float *A, float *U, float *S, float *V, long long count) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += grid_threads()) {
    float a[9], u[9], sg[3], v[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) a[k] = A[9 * i + k];
    svd3(a, u, sg, v);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      U[9 * i + k] = u[k];
      V[9 * i + k] = v[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) S[3 * i + k] = sg[k];
  }
}

__global__ void k_constitutive_batch(material_dev mat, float *F, float *pl, float *tau, long long count) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += grid_threads()) {
    float f[9], t[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) f[k] = F[9 * i + k];
    float p = pl ? pl[i] : 0.f;
    constitutive(mat, f, p, t);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      F[9 * i + k] = f[k];
      tau[9 * i + k] = t[k];
    }
    if (pl) pl[i] = p;
  }
}

// ----------------------------------------------------------------- allocation-free activation
// Kernels used only by zsmpm_activate_blocks_noalloc (zsmpm_static.cu): particle positions
// come as the reference's Particles "x" layout (3 floats per particle) instead of the
// scene's float4 buffer, and the result is copied out to the caller's arrays.

// Zeroes the bitmap and the status word of the static scratch before a call.
__global__ void __launch_bounds__(kThreads) k_static_reset(scene_device s) {
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < s.prm.bitmap_cap; w += grid_threads())
    s.bitmap[w] = 0u;
  if (blockIdx.x == 0 && threadIdx.x == 0) s.ctr[kCtrStatus] = 0;
}

// ComputeSparsity over AoS positions, one insert per distinct block key of a warp.
__global__ void __launch_bounds__(kThreads) k_insert_aos(scene_device s, const float *x) {
  const int lane = threadIdx.x & 31;
  const int n = s.prm.n;
  int3 lo = make_int3(0x7fffffff, 0x7fffffff, 0x7fffffff);
  int3 hi = make_int3(-0x7fffffff, -0x7fffffff, -0x7fffffff);
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int warps = grid_threads() >> 5;
  for (int base = warp_global * 32; base < n; base += warps * 32) {
    const int i = base + lane;
    uint64_t key = kEmptyKey - 1 - lane;
    int3 c, b = make_int3(0, 0, 0);
    bool valid = false;
    if (i < n) {
      const float4 pos = make_float4(x[3 * (size_t)i], x[3 * (size_t)i + 1], x[3 * (size_t)i + 2], 0.f);
      if (cell_of(s.prm, pos, c, b)) {
        key = pack_key(b.x, b.y, b.z);
        valid = true;
      } else {
        set_status(s.ctr, kStatusOutOfDomain);
      }
    }
    const unsigned peers = __match_any_sync(kFull, key);
    if (valid && lane == __ffs(peers) - 1) {
      table_insert(s, key, b, &s.ctr[kCtrParticleBlocks], 0);
      lo = make_int3(min(lo.x, b.x), min(lo.y, b.y), min(lo.z, b.z));
      hi = make_int3(max(hi.x, b.x), max(hi.y, b.y), max(hi.z, b.z));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo.x = min(lo.x, __shfl_xor_sync(kFull, lo.x, o));
    lo.y = min(lo.y, __shfl_xor_sync(kFull, lo.y, o));
    lo.z = min(lo.z, __shfl_xor_sync(kFull, lo.z, o));
    hi.x = max(hi.x, __shfl_xor_sync(kFull, hi.x, o));
    hi.y = max(hi.y, __shfl_xor_sync(kFull, hi.y, o));
    hi.z = max(hi.z, __shfl_xor_sync(kFull, hi.z, o));
  }
  if (lane == 0 && lo.x != 0x7fffffff) {
    atomicMin(&s.ctr[kCtrBoxLo + 0], lo.x);
    atomicMin(&s.ctr[kCtrBoxLo + 1], lo.y);
    atomicMin(&s.ctr[kCtrBoxLo + 2], lo.z);
    atomicMax(&s.ctr[kCtrBoxHi + 0], hi.x);
    atomicMax(&s.ctr[kCtrBoxHi + 1], hi.y);
    atomicMax(&s.ctr[kCtrBoxHi + 2], hi.z);
  }
}

// Copies the sorted keys out; count_out = block count, or -1 (table full / capacity /
// bounding box), -2 (more blocks than cap), -3 (a position was NaN/Inf or out of range).
__global__ void __launch_bounds__(kThreads) k_export_keys(scene_device s, int *keys_out, int cap,
                                                           int *count_out) {
  const int st = s.ctr[kCtrStatus];
  const int nb = s.ctr[kCtrBlocks];
  int code = nb;
  if (st & kStatusOutOfDomain) code = -3;
  else if (st & (kStatusTableFull | kStatusCapacity | kStatusBitmap)) code = -1;
  else if (nb > cap) code = -2;
  if (blockIdx.x == 0 && threadIdx.x == 0) *count_out = code;
  if (code < 0) return;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 3 * nb; t += grid_threads())
    keys_out[t] = s.active_keys[t];
}

// SM count of the current device, looked up once per device ordinal.  Two host threads that
// look up the same device at once store the same value, so the atomics need no lock.
constexpr int kMaxDevices = 64;
std::atomic<int> g_num_sms[kMaxDevices];
int num_sms() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = -1;
  int n = dev >= 0 ? g_num_sms[dev].load(std::memory_order_relaxed) : 0;
  if (n <= 0) {
    if (dev < 0 || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
    else
      g_num_sms[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

}  // namespace

// ----------------------------------------------------------------- launchers
// Whether activation and binning run as one launch (k_prepare): where the particles are few
// enough that the passes cost less than the launches' boundaries.
// Measured, substep with the launches / a cooperative grid / a cluster: 4 k particles 0.091 / 0.067 /
// 0.062 ms, 140 k 0.109 / 0.096 / 0.102, 490 k 0.171 / 0.165 / 0.194, 3.7 M 0.510 / 0.515 / -, 16 M
// 1.98 / 2.06 / -.  With a learned closure the closure pass runs beside activation and binning, and a
// cooperative grid waits for room beside it (3.7 M: 1.03 / 1.09 ms), so those scenes keep the launches.
constexpr int kPrepMaxParticles = 1 << 20, kPrepClusterParticles = 1 << 15;
bool fused_prepare(const scene_device &s) { return s.prm.cap <= kPrepMaxParticles && !s.aux.learned; }

cudaError_t launch_prepare(scene_device &s, bool activate, bool bin, cudaStream_t st) {
  const int sm = num_sms();
  const bool cluster = s.prm.cap <= kPrepClusterParticles;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster) {
    cfg.gridDim = dim3(kPrepCluster);
    cfg.blockDim = dim3(prep_shape<true>::kThreads);
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kPrepCluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    return cudaLaunchKernelEx(&cfg, k_prepare<true>, s, activate ? 1 : 0, bin ? 1 : 0);
  }
  // about four particles a thread, at most two CTAs per SM (all CTAs are resident at once)
  constexpr int nt = prep_shape<false>::kThreads;
  cfg.gridDim = dim3((unsigned)std::min(2 * sm, std::max(64, s.prm.n / (4 * nt))));
  cfg.blockDim = dim3(nt);
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  return cudaLaunchKernelEx(&cfg, k_prepare<false>, s, activate ? 1 : 0, bin ? 1 : 0);
}

cudaError_t launch_activate(scene_device &s, cudaStream_t st) {
  if (fused_prepare(s)) return launch_prepare(s, true, false, st);
  const int sm = num_sms();
  k_begin<<<sm * 4, kThreads, 0, st>>>(s);
  k_insert_particle_blocks<<<sm * 16, kThreads, 0, st>>>(s);
  k_insert_moved_blocks<<<sm * 2, kThreads, 0, st>>>(s);
  k_enlarge<<<sm * 2, kThreads, 0, st>>>(s);
  k_bitmap_prepare<<<1, 32, 0, st>>>(s);
  k_bitmap_set<<<sm * 2, kThreads, 0, st>>>(s);
  cudaError_t e = device_scan(load_popc{s.bitmap}, &s.ctr[kCtrWords], s.scan_part, s.word_prefix, st);
  if (e != cudaSuccess) return e;
  k_assign_ranks<<<sm * 2, kThreads, 0, st>>>(s);
  k_neighbors<<<sm * 2, kThreads, 0, st>>>(s);
  return cudaGetLastError();
}

// Both binnings are enqueued; each kernel returns at once unless the device counter
// kCtrIncBin (set by the activation) selects its path, so one CUDA graph serves both.
cudaError_t launch_bin(scene_device &s, cudaStream_t st) {
  if (fused_prepare(s)) return launch_prepare(s, false, true, st);
  const int sm = num_sms();
  k_bin_count<<<sm * 16, kThreads, 0, st>>>(s);
  k_inc_map<<<sm, kThreads, 0, st>>>(s);
  k_inc_stayers<<<sm * 8, kThreads, 0, st>>>(s);
  k_inc_movers<<<sm * 4, kThreads, 0, st>>>(s);
  cudaError_t e = device_scan(load_int{s.block_count}, &s.ctr[kCtrBlocks], s.scan_part, s.block_start, st);
  if (e != cudaSuccess) return e;
  k_cell_start<<<sm * 4, 512, 0, st>>>(s);
  k_bin_scatter<<<sm * 16, kThreads, 0, st>>>(s);
  k_inc_place_stayers<<<sm * 8, kThreads, 0, st>>>(s);
  k_inc_place_movers<<<sm * 4, kThreads, 0, st>>>(s);
  k_bin_finalize<<<sm * 3, 512, 0, st>>>(s);
  k_inc_sort<<<sm * 2, kThreads, 0, st>>>(s);
  k_inc_finalize<<<sm * 8, kThreads, 0, st>>>(s);
  return cudaGetLastError();
}

// per-device kernel attributes; called once per scene with its device current, before any
// capture of its launches
cudaError_t prepare_kernels() {
  cudaError_t e = cudaSuccess;
  auto p2g_attrs = [&](const void *fn, int ranks) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p2g_smem_bytes(ranks));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  };
  p2g_attrs((const void *)k_p2g<false, 2>, 8);
  p2g_attrs((const void *)k_p2g<false, 3>, 12);
  p2g_attrs((const void *)k_p2g<false, 4>, 16);
  p2g_attrs((const void *)k_p2g<false, 2, true>, 8);
  p2g_attrs((const void *)k_p2g<true, 2>, 8);
  p2g_attrs((const void *)k_p2g<true, 3>, 12);
  p2g_attrs((const void *)k_p2g<true, 4>, 16);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_prepare<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_force_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g2p_smem_bytes(kThreads));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_g2p<true, true, kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)g2p_smem_bytes(kThreads));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_g2p<true, false, kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)g2p_smem_bytes(kThreads));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_g2p<false, true, kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)g2p_smem_bytes(kThreads));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_g2p<false, false, kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)g2p_smem_bytes(kThreads));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_g2p<false, true, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)g2p_smem_bytes(128));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_g2p<false, false, 128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)g2p_smem_bytes(128));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_g2p<false, false, kThreads, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)g2p_smem_bytes(kThreads));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_g2p<false, false, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)g2p_smem_bytes(128));
}

// the P2G kernel of the scene's staging depth (p2g_ranks: 8, 12 or 16)
template <bool kCell>
static void launch_staged_p2g(scene_device &s, const float4 *rows, int with_mass, cudaStream_t st) {
  const int ranks = s.prm.p2g_ranks > 0 ? s.prm.p2g_ranks : kP2GRanksDefault;
  const int dflt = ranks == 8 ? 4 : ranks == 16 ? 2 : 3;
  const int grid = num_sms() * (s.prm.p2g_ctas_per_sm > 0 ? s.prm.p2g_ctas_per_sm : dflt);
  if (ranks == 8)
    k_p2g<kCell, 2><<<grid, kP2GThreads, p2g_smem_bytes(8), st>>>(s, rows, with_mass, nullptr, 0, nullptr);
  else if (ranks == 16)
    k_p2g<kCell, 4><<<grid, kP2GThreads, p2g_smem_bytes(16), st>>>(s, rows, with_mass, nullptr, 0, nullptr);
  else
    k_p2g<kCell, 3><<<grid, kP2GThreads, p2g_smem_bytes(12), st>>>(s, rows, with_mass, nullptr, 0, nullptr);
}

cudaError_t launch_p2g(scene_device &s, cudaStream_t st) {
  if (s.prm.transfer == kTransferCell) return launch_p2c2g(s, 0, st);
  launch_staged_p2g<false>(s, s.cur.row, 1, st);
  return cudaGetLastError();
}

// part 0: P2C2GTransfer from the stored affine term; 1 (momentum) and 2 (force): the part's
// affine term is formed first, into the next buffer's rows (G2C2P rewrites them)
cudaError_t launch_p2c2g(scene_device &s, int part, cudaStream_t st) {
  const float4 *rows = s.cur.row;
  if (part != 0) {
    k_cell_affine<<<num_sms() * 4, kThreads, 0, st>>>(s, part, s.nxt.row);
    rows = s.nxt.row;
  }
  launch_staged_p2g<true>(s, rows, part == 2 ? 0 : 1, st);
  return cudaGetLastError();
}

cudaError_t launch_grid_update(scene_device &s, cudaStream_t st) {
  k_grid_update<<<num_sms() * 8, kThreads, 0, st>>>(s);
  k_grid_boundaries<<<num_sms() * 4, kThreads, 0, st>>>(s);
  return cudaGetLastError();
}

// The learned closure's pass over the projections the last learned G2P queued: the network on
// the tensor cores, then k_closure_finish.  It writes F, the affine momentum and the plastic
// state of the queued particles only, and reads the queue counter and the substep number the
// G2P recorded, which the next substep's activation and binning leave alone: so it may run
// beside them (a deferred pass), joining before the next P2G.
cudaError_t launch_closure_pass(scene_device &s, cudaStream_t st) {
  cudaError_t e = launch_closure_rows(s.aux.cd, s.aux.q_feat, s.aux.q_out, &s.ctr[kCtrQueue], s.aux.qcap, st);
  if (e != cudaSuccess) return e;
  k_closure_finish<<<num_sms() * 4, kThreads, 0, st>>>(s);
  return cudaGetLastError();
}

cudaError_t launch_g2p(scene_device &s, cudaStream_t st, bool closure_pass) {
  const int per_sm = s.prm.g2p_ctas_per_sm > 0 ? s.prm.g2p_ctas_per_sm : 3;
  const int grid = num_sms() * per_sm;
  const bool small = s.prm.g2p_threads == 128;
  if (s.prm.transfer == kTransferCell) {
    small ? k_g2p<false, false, 128, true><<<grid, 128, g2p_smem_bytes(128), st>>>(s)
          : k_g2p<false, false, kThreads, true><<<grid, kThreads, g2p_smem_bytes(kThreads), st>>>(s);
    return cudaGetLastError();
  }
  if (s.aux.learned) {
    // G2P queues the projections (from an empty queue), the network runs over the queue on the
    // tensor cores, and k_closure_finish completes the queued particles; closure_pass = false
    // leaves the last two to a deferred launch_closure_pass
    cudaError_t e = cudaMemsetAsync(&s.ctr[kCtrQueue], 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    if (s.prm.batch)
      k_g2p<true, true, kThreads><<<grid, kThreads, g2p_smem_bytes(kThreads), st>>>(s);
    else
      k_g2p<true, false, kThreads><<<grid, kThreads, g2p_smem_bytes(kThreads), st>>>(s);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return closure_pass ? launch_closure_pass(s, st) : cudaSuccess;
  }
  if (s.prm.batch)
    small ? k_g2p<false, true, 128><<<grid, 128, g2p_smem_bytes(128), st>>>(s)
          : k_g2p<false, true, kThreads><<<grid, kThreads, g2p_smem_bytes(kThreads), st>>>(s);
  else
    small ? k_g2p<false, false, 128><<<grid, 128, g2p_smem_bytes(128), st>>>(s)
          : k_g2p<false, false, kThreads><<<grid, kThreads, g2p_smem_bytes(kThreads), st>>>(s);
  return cudaGetLastError();
}

// the force operator's two kernels; both work counters are zero on entry
static cudaError_t launch_force(scene_device &s, const float *v, float *f, long long ndofs, float dt, const int *skip,
                                cudaStream_t st) {
  k_force_rows<<<num_sms() * 3, kThreads, g2p_smem_bytes(kThreads), st>>>(s, v, ndofs, dt, skip, s.nxt.row);
  k_p2g<false, 2, true><<<num_sms() * 4, kP2GThreads, p2g_smem_bytes(8), st>>>(s, s.nxt.row, 0, f, ndofs, skip);
  return cudaGetLastError();
}

cudaError_t launch_g2p2g(scene_device &s, const float *v, float *f, long long ndofs, float dt, cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(&s.ctr[kCtrWork + kWorkForceRows], 0, 2 * sizeof(int), st);
  return e != cudaSuccess ? e : launch_force(s, v, f, ndofs, dt, nullptr, st);
}

cudaError_t launch_implicit_mass(scene_device &s, const float *dv, float *out, float dt, long long ndofs,
                                 cudaStream_t st) {
  k_implicit_mass<<<num_sms() * 4, kThreads, 0, st>>>(s, dv, out, dt, ndofs);
  return cudaGetLastError();
}

cudaError_t launch_implicit_project(scene_device &s, float *dof, long long ndofs, cudaStream_t st) {
  k_implicit_project<<<num_sms() * 4, kThreads, 0, st>>>(s, dof, ndofs);
  return cudaGetLastError();
}

cudaError_t launch_implicit_precondition(scene_device &s, const float *in, float *out, long long ndofs,
                                         cudaStream_t st) {
  k_implicit_precondition<<<num_sms() * 4, kThreads, 0, st>>>(s, in, out, ndofs);
  return cudaGetLastError();
}

// CTAs of a pass over the nodes that ndofs admits (at most four per SM)
static int cg_grid(long long ndofs) {
  return (int)std::max(1ll, std::min(4ll * num_sms(), (ndofs / 3 + kThreads - 1) / kThreads));
}

// The solve's start: r = b - A x, project r, p = M r, zTrk = r.p, and the loop's first check.
cudaError_t launch_cg_begin(scene_device &s, const float *x, const float *b, const cg_vectors &v, long long ndofs,
                            float dt, cg_state *cs, float tol, float rel_tol, int max_iters, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(cs, 0, sizeof(cg_state), st);
  if (e != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(v.ap, 0, sizeof(float) * (size_t)ndofs, st)) != cudaSuccess) return e;
  if ((e = launch_g2p2g(s, x, v.ap, ndofs, dt, st)) != cudaSuccess) return e;
  k_cg_start<<<cg_grid(ndofs), kThreads, 0, st>>>(s, x, b, v, ndofs, dt, cs, tol, rel_tol, max_iters);
  return cudaGetLastError();
}

// One loop iteration (ConjugateGradient.hpp:118-171); does nothing once the solve is done.
cudaError_t launch_cg_iteration(scene_device &s, float *x, const cg_vectors &v, long long ndofs, float dt,
                                cg_state *cs, int max_iters, cudaStream_t st) {
  const int grid = cg_grid(ndofs);
  // (its work counters were cleared by the pass before)
  const cudaError_t e = launch_force(s, v.p, v.ap, ndofs, dt, &cs->done, st);
  if (e != cudaSuccess) return e;
  k_cg_apply<<<grid, kThreads, 0, st>>>(s, v, ndofs, dt, cs);
  k_cg_update<<<grid, kThreads, 0, st>>>(s, x, v, ndofs, cs, max_iters);
  k_cg_direction<<<grid, kThreads, 0, st>>>(s, v, ndofs, cs);
  return cudaGetLastError();
}

// k_prepare, or: k_begin, the two particle-block inserts (one returns at once), enlarge, prepare, set,
// 3 scans, ranks, neighbours; the binning's 14 launches (the full and the incremental path, one of
// which returns at once).  Then p2g; grid update and boundaries; g2p
int kernels_per_substep(const scene_device &s) { return (fused_prepare(s) ? 1 : 11 + 14) + 4; }

cudaError_t launch_import(scene_device &s, const float *m, const float *x, const float *v,
                          const float *C, const float *F, const float *plastic, int n,
                          cudaStream_t st) {
  k_import<<<num_sms() * 8, kMoveThreads, 0, st>>>(s, m, x, v, C, F, plastic, n);
  return cudaGetLastError();
}

cudaError_t launch_import_tilevector(scene_device &s, const float *base, int nchn, int off_m,
                                     int off_x, int off_v, int off_C, int off_F, int off_pl,
                                     int n, cudaStream_t st) {
  k_import_tv<<<num_sms() * 4, kThreads, 0, st>>>(s, base, nchn, off_m, off_x, off_v, off_C, off_F,
                                                  off_pl, n);
  return cudaGetLastError();
}

cudaError_t launch_prime(scene_device &s, cudaStream_t st) {
  if (s.prm.transfer == kTransferCell)
    k_cell_affine<<<num_sms() * 4, kThreads, 0, st>>>(s, 0, s.cur.row);
  else
    k_prime<<<num_sms() * 4, kThreads, 0, st>>>(s);
  return cudaGetLastError();
}

cudaError_t launch_export(const scene_device &s, float *m, float *x, float *v, float *C,
                          float *F, float *plastic, cudaStream_t st) {
  k_export<<<num_sms() * 8, kMoveThreads, 0, st>>>(s, m, x, v, C, F, plastic);
  return cudaGetLastError();
}

cudaError_t launch_export_tilevector(const scene_device &s, float *base, int nchn, int off_m,
                                     int off_x, int off_v, int off_C, int off_F, int off_pl,
                                     cudaStream_t st) {
  k_export_tv<<<num_sms() * 4, kThreads, 0, st>>>(s, base, nchn, off_m, off_x, off_v, off_C, off_F,
                                                  off_pl);
  return cudaGetLastError();
}

cudaError_t launch_export_order(const scene_device &s, int *order, cudaStream_t st) {
  k_export_order<<<num_sms() * 4, kThreads, 0, st>>>(s, order);
  return cudaGetLastError();
}

cudaError_t launch_activate_static(scene_device &s, const float *x, int *keys_out, int cap,
                                   int *count_out, cudaStream_t st) {
  const int sm = num_sms();
  k_static_reset<<<sm, kThreads, 0, st>>>(s);
  k_begin<<<sm * 4, kThreads, 0, st>>>(s);
  k_insert_aos<<<sm * 8, kThreads, 0, st>>>(s, x);
  k_enlarge<<<sm * 2, kThreads, 0, st>>>(s);
  k_bitmap_prepare<<<1, 32, 0, st>>>(s);
  k_bitmap_set<<<sm * 2, kThreads, 0, st>>>(s);
  cudaError_t e = device_scan(load_popc{s.bitmap}, &s.ctr[kCtrWords], s.scan_part, s.word_prefix, st);
  if (e != cudaSuccess) return e;
  k_assign_ranks<<<sm * 2, kThreads, 0, st>>>(s);
  k_export_keys<<<sm, kThreads, 0, st>>>(s, keys_out, cap, count_out);
  return cudaGetLastError();
}

cudaError_t launch_exclusive_scan(const int *in, const int *n_ptr, int *part, int *out, cudaStream_t st) {
  return device_scan(load_int{in}, n_ptr, part, out, st);
}

cudaError_t launch_svd_batch(const float *A, float *U, float *S, float *V, long long count,
                             cudaStream_t st) {
  k_svd_batch<<<num_sms() * 4, kThreads, 0, st>>>(A, U, S, V, count);
  return cudaGetLastError();
}

cudaError_t launch_constitutive_batch(const material_dev &mat, float *F, float *plastic,
                                      float *tau, long long count, cudaStream_t st) {
  k_constitutive_batch<<<num_sms() * 4, kThreads, 0, st>>>(mat, F, plastic, tau, count);
  return cudaGetLastError();
}

}  // namespace zsmpm
