// merge.cu -- device-wide merge and merge_by_key (merge path), sm_100a.
//
// Replaces the reference's my_merge (merge.cu:127-162): a thrust::tabulate of
// merge_path at every tile diagonal (locate_merge_path, merge.cu:100-124)
// followed by one staged merge per tile (merge_kernel / staged_merge,
// merge.cu:12-97), which is keys-only; the by-key form follows the bounded
// group merge_by_key (bulk/algorithm/merge.hpp:507-607).
//
// Here: persistent CTAs merge 4096-output tiles (2048 for 8-byte keys) in a
// two-buffer pipeline.  A tile's A/B split comes from a partition kernel where
// a CTA has many tiles, and from the CTA's loader warp otherwise.  The
// loader's first lane brings a tile's A and B key and payload ranges into
// shared memory with untiled bulk (TMA) copies -- each range widened to whole
// 16-byte chunks, the ragged ends by plain loads -- while the compute warps
// merge the previous tile: each thread finds its diagonal with a merge-path
// search in shared memory, merges its outputs serially (branch-free: keys plus
// the shared-memory index of each output's source, which gathers the payload),
// and, once every thread has read its inputs, writes them back in place in the
// 128-byte-swizzled layout; the loader then stores the tile with tiled tensor
// copies, which undo the swizzle.  No thread loads or stores a tile element
// itself on this path.  Inputs that bulk copies cannot bring (an array off the
// 16-byte boundaries) are copied by the compute warps, in a kernel of its own.
#include <algorithm>

#include "bk_common.cuh"
#include "bk_merge.cuh"
#include "bk_tma.cuh"
#include "bk_tune.hpp"

namespace bk {

constexpr int kMergeWarps = 8;                       // compute warps
constexpr int kMergeCompute = 32 * kMergeWarps;      // compute threads
constexpr int kMergeThreads = kMergeCompute + 32;    // + the loader warp
constexpr int kMergeBufs = 2;

template <typename K, typename P>
struct MergeCfg {
  static constexpr int ITEMS = sizeof(K) == 4 ? 16 : 8;         // outputs per thread (64 bytes of keys)
  static constexpr int TILE = kMergeCompute * ITEMS;            // 4096 / 2048 outputs
  static constexpr int PB = payload_bytes<P>();                 // 0, 4 or 8
  static constexpr int KV = 16 / (int)sizeof(K);                // keys per 16-byte chunk
  static constexpr int PV = PB ? 16 / PB : 1;                   // payloads per 16-byte chunk
  static constexpr int L = KV > PV ? KV : PV;                   // the ranges are widened to multiples of L
  // the keys area holds A's range then B's (each widened by < L on either
  // side, B starting at a multiple of L) plus one element read past either
  // end; it takes the tile's outputs afterwards (1024-byte swizzle period).
  // The payloads area is laid out the same way: index i there belongs to the
  // key at index i.
  static constexpr size_t KEY_AREA = align_up(sizeof(K) * (TILE + 4 * L + 1), 1024);
  static constexpr size_t PAY_AREA = PB ? align_up((size_t)PB * (TILE + 4 * L + 1), 1024) : 0;
  static constexpr size_t BUF = KEY_AREA + PAY_AREA;
  static constexpr uint32_t KROWS = sizeof(K) * TILE / 128;     // 128-byte rows of output keys per tile
  static constexpr uint32_t PROWS = PB * TILE / 128;
};

template <typename K, typename P>
constexpr size_t merge_smem_bytes() {
  return (size_t)kMergeBufs * MergeCfg<K, P>::BUF + 1024;  // + room to align the buffers to 1024 bytes
}

// parts[k] = number of A elements among the first min(k*TILE, na+nb) outputs.
template <typename K>
__global__ void merge_partition_kernel(const K *a, uint64_t na, const K *b, uint64_t nb, uint64_t tile,
                                       uint64_t num_parts, uint64_t *parts) {
  grid_dependency_wait();
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= num_parts) return;
  const uint64_t total = na + nb;
  const uint64_t diag = k * tile < total ? k * tile : total;
  parts[k] = merge_path<K, uint64_t>(a, na, b, nb, diag);
}

// The number of A elements among the first `diag` outputs, known to lie in
// [lo, hi]: the first mid there with b[diag - 1 - mid] < a[mid] (ties go to A).
// The whole warp searches: each round its lanes cut the range into 65 parts
// with two probes each, so a tile's 4097 candidates take two rounds of loads
// and 2^26 take five, where a one-thread binary search waits for 12 or 26 one
// after another.
template <typename K>
__device__ __forceinline__ uint64_t merge_split_warp(const K *a, const K *b, uint64_t diag, uint64_t lo, uint64_t hi,
                                                     int lane) {
  while (lo < hi) {
    const uint64_t step = (hi - lo + 64) / 65;
    const uint64_t m0 = lo + (uint64_t)(lane + 1) * step - 1, m1 = m0 + 32 * step;
    const bool in0 = m0 < hi, in1 = m1 < hi;
    K a0 = K(), b0 = K(), a1 = K(), b1 = K();
    if (in0) {
      a0 = a[m0];
      b0 = b[diag - 1 - m0];
    }
    if (in1) {
      a1 = a[m1];
      b1 = b[diag - 1 - m1];
    }
    const unsigned int s0 = __ballot_sync(0xffffffffu, !in0 || b0 < a0), s1 = __ballot_sync(0xffffffffu, !in1 || b1 < a1);
    const unsigned int f = s0 ? (unsigned int)__ffs(s0) - 1u : s1 ? (unsigned int)__ffs(s1) + 31u : 64u;  // first probe past the split
    if (f < 64u && lo + (uint64_t)(f + 1) * step - 1 < hi) hi = lo + (uint64_t)(f + 1) * step - 1;
    lo += (uint64_t)f * step;
  }
  return hi;
}

// What the compute warps need to know of a tile in a buffer (written by the
// loader before it arms the buffer's barrier).
struct MergeDesc {
  uint32_t la, lb;    // A and B elements of the tile
  uint32_t ia, ib;    // index of A's / B's first element in the keys (and payloads) area
  uint32_t count;     // outputs (la + lb)
  uint32_t tile;      // tile index
  uint64_t a0;        // A's first element of the tile
};

// The kernel's parameters.
template <typename K, typename P>
struct MergeArgs {
  CUtensorMap okmap;  // output keys as rows of 128 bytes (boxes of KROWS rows)
  CUtensorMap opmap;  // output payloads (boxes of PROWS rows)
  const K *a;
  const P *av;
  uint64_t na;
  const K *b;
  const P *bv;
  uint64_t nb;
  K *out;
  P *outv;
  const uint64_t *parts;  // PARTS: the split at every tile boundary
  uint64_t tiles;
  uint64_t covered_out;  // leading outputs inside whole rows of both output views (0: none)
  int strided;            // PARTS: CTA c takes tiles c, c + G, c + 2G, ... (G = gridDim.x) instead of a run
};

// Bytes of the bulk copy that merge_load_range issues for [lo, hi).
template <typename T>
__device__ __forceinline__ uint32_t merge_bulk_bytes(uint64_t lo, uint64_t hi) {
  constexpr uint64_t V = 16 / sizeof(T);
  const uint64_t bulk_hi = hi & ~(V - 1);
  return bulk_hi > lo ? (uint32_t)((bulk_hi - lo) * sizeof(T)) : 0u;
}

// Loader: one input range [lo, hi) of `src` (T elements, 16-byte aligned
// array) into shared memory at `dst` (16-byte aligned): the whole 16-byte
// chunks by one bulk copy completing on bar (its bytes already expected),
// the ragged end by plain loads.  lo is a multiple of 16 / sizeof(T).
template <typename T>
__device__ __forceinline__ void merge_load_range(T *dst, const T *src, uint64_t lo, uint64_t hi, uint64_t *bar,
                                                 uint64_t policy) {
  constexpr uint64_t V = 16 / sizeof(T);
  const uint64_t bulk_hi = hi & ~(V - 1);
  if (bulk_hi > lo) tma_load_1d_hint(dst, src + lo, (uint32_t)((bulk_hi - lo) * sizeof(T)), bar, policy);
  for (uint64_t i = bulk_hi > lo ? bulk_hi : lo; i < hi; ++i) dst[i - lo] = src[i];
}

// One element from global to shared memory, with no register in between: the
// compute warps' copy of inputs that bulk copies cannot bring.  Through
// registers it was bound by the loads' latency, or by the instructions of
// loads batched by hand (half as many again, ncu): whether the compiler kept
// several loads in flight turned on the registers left (i32/u32 2 x 2^26 off
// the boundaries on a B200: 654 us, and 1029 after unrelated changes; u32/u64
// 2140).  With all of a tile's copies in flight: 598, 817.
template <typename T>
__device__ __forceinline__ void copy_async(T *dst, const T *src) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "4 or 8 bytes");
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"((int)sizeof(T)) : "memory");
}
// Until this thread's copies have arrived.
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Persistent merge.  Warps 0-7 merge; warp 8's lane 0 loads and stores.
// Where a tile's inputs begin (its split) comes from a partition kernel
// (PARTS) or, with few tiles a CTA, from the loader warp itself, two tiles
// ahead: CTA c then takes the c-th of gridDim.x equal runs of consecutive
// tiles, a tile's split lies within a tile of the one before, so its search
// reads what is loaded next anyway and runs while the compute warps merge.
// (The partition kernel, one thread a split, waits for 21 to 26 reads one after
// another: 14 us before a merge of 3.7 million i32 keys that takes 12.)  A warp
// of its own for the searches made the kernel's registers spill: 447 us for
// 2 x 2^26 f32/u32 pairs against 408.  Kernels of their own for either source
// of splits (PARTS needs one loader lane alone) and for unaligned inputs
// (!TMA_IN) leave each the registers the others would take: in one kernel f64
// 2 x 2^26 took 481 us against 461 here, f64/u32 7 + 9 million 91 against 82.
// Tile i of the CTA uses buffer i mod 2 and goes through:
//   loader: (once the compute warps have written tile i-2's outputs to the
//           buffer and that tile's stores have read them) write the tile's
//           descriptor, bulk-copy its ranges in; full[b] completes;
//   compute: merge-path search and serial merge into registers; a barrier
//           among the compute warps (every input read); outputs written in
//           place, swizzled; each warp arrives on out[b];
//   loader: tensor stores of the keys and payloads (rows past the output
//           view are clipped; a last tile's ragged end is stored by the
//           compute threads directly).
// All waits are bounded; after a timeout the kernel records
// BK_ERR_SPIN_TIMEOUT in the header and every role stops.
template <typename K, typename P, bool TMA_IN, bool PARTS>
__global__ void __launch_bounds__(kMergeThreads, (sizeof(K) == 4 && payload_bytes<P>() == 8) ? 2 : 3)
merge_kernel(const __grid_constant__ MergeArgs<K, P> args,
                                                                 WsHeader *hdr, unsigned long long spin_limit_ns) {
  using C = MergeCfg<K, P>;
  constexpr int ITEMS = C::ITEMS, TILE = C::TILE, NB = kMergeBufs;
  constexpr bool HP = has_payload<P>();
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  unsigned char *const smem_raw = smem_dyn + ((1024u - (smem_addr(smem_dyn) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t s_full[NB];
  __shared__ __align__(8) uint64_t s_out[NB];
  __shared__ MergeDesc s_desc[NB];
  __shared__ int s_abort;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto buf = [&](int b) { return smem_raw + (size_t)b * C::BUF; };
  auto aborted = [&]() -> bool { return *reinterpret_cast<volatile int *>(&s_abort) != 0; };
  const uint64_t total = args.na + args.nb;
  const uint64_t G = gridDim.x;

  if (tid == kMergeCompute) {
    for (int b = 0; b < NB; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&s_out[b], kMergeWarps);
    }
    fence_proxy_async_smem();
    s_abort = 0;
  }
  __syncthreads();
  grid_dependency_wait();

  // tiles of this CTA: first + i * step for i < mine (the grid is no larger than the tile count)
  const bool strided = PARTS && args.strided;
  const uint64_t first = strided ? blockIdx.x : args.tiles * blockIdx.x / G, step = strided ? G : 1;
  const uint64_t mine = strided ? (args.tiles - blockIdx.x + G - 1) / G : args.tiles * (blockIdx.x + 1) / G - first;

  if (warp == kMergeWarps) {
    // ================= the loader (lane 0; the splits: all lanes) =================
    if (PARTS && lane != 0) return;
    // A elements before tile k, given that `from` lie before a tile no more than `tiles` before it
    auto split = [&](uint64_t k, uint64_t from, uint64_t tiles) -> uint64_t {
      const uint64_t diag = k * TILE < total ? k * TILE : total;
      uint64_t lo = diag > args.nb ? diag - args.nb : 0, hi = diag < args.na ? diag : args.na;
      if (lo < from) lo = from;
      if (hi > from + tiles * TILE) hi = from + tiles * TILE;
      return merge_split_warp(args.a, args.b, diag, lo, hi, lane);
    };
    // Into L2: tile k's payloads (its A range [f, t)) and the keys that the
    // search for the tile after it can reach.
    uint64_t pa = 0, pb = 0;  // keys up to here have been asked for
    auto prefetch = [&](uint64_t k, uint64_t f, uint64_t t) {
      const uint64_t d0 = k * TILE, d1 = d0 + TILE < total ? d0 + TILE : total;
      if constexpr (HP) {
        prefetch_l2_range(args.av + f, (t - f) * sizeof(P));
        prefetch_l2_range(args.bv + (d0 - f), (d1 - d0 - (t - f)) * sizeof(P));
      }
      const uint64_t ea = t + TILE < args.na ? t + TILE : args.na;
      const uint64_t eb = d1 - t + TILE < args.nb ? d1 - t + TILE : args.nb;
      if (pa < f) pa = f;
      if (pb < d0 - f) pb = d0 - f;
      if (pa < ea) prefetch_l2_range(args.a + pa, (ea - pa) * sizeof(K));
      if (pb < eb) prefetch_l2_range(args.b + pb, (eb - pb) * sizeof(K));
      pa = ea;
      pb = eb;
    };
    const uint64_t *const parts = args.parts;
    uint64_t a0, a1;  // the A range of the tile to load next
    if constexpr (PARTS) {
      a0 = parts[first];
      a1 = parts[first + 1];
    } else {
      a0 = split(first, 0, first);
      a1 = split(first + 1, a0, 1);
      if (lane == 0 && mine > 1) prefetch(first, a0, a1);
    }
    const uint64_t policy = l2_policy_evict_first();  // inputs and outputs are read / written once
    uint32_t outpar = 0u, armpar = 0u, armany = 0u;
    bool stored = false, failed = false;
    uint64_t fail_tile = 0;
    for (uint64_t i = 0; i < mine + 2; ++i) {
      const int b = (int)(i & 1);
      if (i >= 2) {
        // tile i-2's outputs are in buffer b: store them
        if (lane == 0 && !mbar_wait_or_abort(&s_out[b], (outpar >> b) & 1u, spin_limit_ns, &s_abort)) {
          failed = true;
          fail_tile = first + (i - 2) * step;
        }
        if (PARTS ? failed : __shfl_sync(0xffffffffu, (int)failed, 0) != 0) break;
        outpar ^= 1u << b;
        const uint32_t tile = s_desc[b].tile;
        if (lane == 0 && args.covered_out > (uint64_t)tile * TILE) {
          tma_store_rows(&args.okmap, tile * C::KROWS, buf(b), policy);
          if constexpr (HP) tma_store_rows(&args.opmap, tile * C::PROWS, buf(b) + C::KEY_AREA, policy);
          tma_store_commit();
          stored = true;
        }
      }
      if (i >= mine) continue;
      // ---- tile k: its A range [a0, a1) and B range [b0, b1)
      const uint64_t k = first + i * step;
      if (lane == 0) {
        if (stored) tma_store_wait_read();  // the stores have read the buffer
        const uint64_t d0 = k * TILE, d1 = d0 + TILE < total ? d0 + TILE : total;
        const uint64_t b0 = d0 - a0, b1 = d1 - a1;
        MergeDesc d;
        d.la = (uint32_t)(a1 - a0);
        d.lb = (uint32_t)(b1 - b0);
        d.count = (uint32_t)(d1 - d0);
        d.tile = (uint32_t)k;
        d.a0 = a0;
        if constexpr (TMA_IN) {
          const uint64_t alo = a0 & ~(uint64_t)(C::L - 1), blo = b0 & ~(uint64_t)(C::L - 1);
          const uint32_t bstart = (uint32_t)align_up(a1 - alo, (size_t)C::L);  // B's copy: a multiple of L
          d.ia = (uint32_t)(a0 - alo);
          d.ib = bstart + (uint32_t)(b0 - blo);
          uint32_t bytes =
              (a1 > a0 ? merge_bulk_bytes<K>(alo, a1) : 0u) + (b1 > b0 ? merge_bulk_bytes<K>(blo, b1) : 0u);
          if constexpr (HP)
            bytes += (a1 > a0 ? merge_bulk_bytes<P>(alo, a1) : 0u) + (b1 > b0 ? merge_bulk_bytes<P>(blo, b1) : 0u);
          if (bytes) mbar_expect_tx(&s_full[b], bytes);
          K *sk = reinterpret_cast<K *>(buf(b));
          P *sp = reinterpret_cast<P *>(buf(b) + C::KEY_AREA);
          if (a1 > a0) merge_load_range<K>(sk, args.a, alo, a1, &s_full[b], policy);
          if (b1 > b0) merge_load_range<K>(sk + bstart, args.b, blo, b1, &s_full[b], policy);
          if constexpr (HP) {
            if (a1 > a0) merge_load_range<P>(sp, args.av, alo, a1, &s_full[b], policy);
            if (b1 > b0) merge_load_range<P>(sp + bstart, args.bv, blo, b1, &s_full[b], policy);
          }
        } else {  // the compute warps copy the ranges themselves
          d.ia = 0;
          d.ib = d.la;
        }
        s_desc[b] = d;
        // the loader's one arrival, after its plain stores (descriptor, ragged
        // ends): the phase completes once the bulk copies' bytes have landed
        mbar_arrive(&s_full[b]);
      }
      if constexpr (!PARTS) __syncwarp();
      armpar ^= 1u << b;
      armany |= 1u << b;
      if (i + 1 < mine) {  // the next tile's end, while this one is merged
        if constexpr (PARTS) {
          a0 = parts[k + step];
          a1 = parts[k + step + 1];
        } else {
          a0 = a1;
          a1 = split(k + 2, a0, 1);
          if (lane == 0) prefetch(k + 1, a0, a1);
        }
      }
    }
    if (lane != 0) return;
    if (failed) {
      record_error(hdr, BK_ERR_SPIN_TIMEOUT, (unsigned int)fail_tile);
      *reinterpret_cast<volatile int *>(&s_abort) = 1;
    }
    if (stored) tma_store_wait_all();
    // every load must land before the CTA's shared memory goes away
    for (int b = 0; b < NB; ++b)
      if ((armany >> b) & 1u) (void)mbar_wait(&s_full[b], ((armpar >> b) & 1u) ^ 1u, spin_limit_ns);
    return;
  }

  // ================= the compute warps =================
  uint32_t fullpar = 0u;
  bool bad = false;
  for (uint64_t i = 0; i < mine; ++i) {
    const int b = (int)(i & 1);
    const uint64_t k = first + i * step;
    if (!mbar_wait_or_abort(&s_full[b], (fullpar >> b) & 1u, spin_limit_ns, &s_abort)) bad = true;
    fullpar ^= 1u << b;
    if (named_barrier_or(1, kMergeCompute, bad || aborted())) {
      if (tid == 0) record_error(hdr, BK_ERR_SPIN_TIMEOUT, (unsigned int)k);
      *reinterpret_cast<volatile int *>(&s_abort) = 1;
      break;
    }
    const MergeDesc d = s_desc[b];
    K *const sk = reinterpret_cast<K *>(buf(b));
    P *const sp = reinterpret_cast<P *>(buf(b) + C::KEY_AREA);
    if constexpr (!TMA_IN) {
      const uint64_t a0 = d.a0, b0 = k * TILE - a0;
      for (uint32_t j = tid; j < d.la; j += kMergeCompute) {
        copy_async(sk + j, args.a + a0 + j);
        if constexpr (HP) copy_async(sp + j, args.av + a0 + j);
      }
      for (uint32_t j = tid; j < d.lb; j += kMergeCompute) {
        copy_async(sk + d.la + j, args.b + b0 + j);
        if constexpr (HP) copy_async(sp + d.la + j, args.bv + b0 + j);
      }
      copy_async_wait();
      named_barrier_sync(2, kMergeCompute);
    }
    // ---- merge-path search for this thread's first output, then its outputs
    const uint32_t diag = (uint32_t)tid * ITEMS;
    K okey[ITEMS];
    uint32_t osrc[ITEMS / 2];  // indexes of the outputs' sources, two to a register
    const int valid = (int)min((int)d.count - (int)diag, ITEMS);
    if (valid > 0) {
      uint32_t lo = diag > d.lb ? diag - d.lb : 0u;
      uint32_t hi = diag < d.la ? diag : d.la;
      while (lo < hi) {  // ties go to A: move left while b[diag-1-mid] < a[mid]
        const uint32_t mid = (lo + hi) >> 1;
        if (sk[d.ib + diag - 1 - mid] < sk[d.ia + mid]) hi = mid;
        else lo = mid + 1;
      }
      uint32_t ia = d.ia + lo, ib = d.ib + (diag - lo);
      const uint32_t ea = d.ia + d.la, eb = d.ib + d.lb;
      // reads reach at most one element past either range (a neighbour
      // inside the buffer, never used): the loop stops at `valid`
      K ka = sk[ia], kb = sk[ib];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        if (valid == ITEMS || j < valid) {
          // take A while B is exhausted or !(b < a): equal keys keep A first
          const bool take_a = ia < ea && (ib >= eb || !(kb < ka));
          okey[j] = take_a ? ka : kb;
          const uint32_t at = take_a ? ia : ib;
          if (j & 1) osrc[j >> 1] |= at << 16;
          else osrc[j >> 1] = at;
          ia += take_a ? 1u : 0u;
          ib += take_a ? 0u : 1u;
          if (j + 1 < ITEMS) {
            const K nk = sk[take_a ? ia : ib];
            ka = take_a ? nk : ka;
            kb = take_a ? kb : nk;
          }
        }
      }
    }
    P opay[ITEMS];
    if constexpr (HP) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (j < valid) opay[j] = sp[(j & 1) ? osrc[j >> 1] >> 16 : osrc[j >> 1] & 0xffffu];
    }
    named_barrier_sync(2, kMergeCompute);  // every thread has read its inputs
    // ---- outputs: in place, swizzled for the tensor stores (which write
    // the rows inside the output views); outputs past covered_out (a last
    // tile's ragged end, or every output when the views could not be made)
    // are also stored directly
    const uint64_t o0 = k * TILE + diag;
    if (valid == ITEMS) {
      constexpr int KCH = ITEMS * (int)sizeof(K) / 16;
#pragma unroll
      for (int c = 0; c < KCH; ++c) {
        uint4 q;
        memcpy(&q, &okey[c * (16 / sizeof(K))], 16);
        *reinterpret_cast<uint4 *>(buf(b) + swz128(diag * (uint32_t)sizeof(K) + 16u * c)) = q;
      }
      if constexpr (HP) {
        constexpr int PCH = ITEMS * C::PB / 16;
#pragma unroll
        for (int c = 0; c < PCH; ++c) {
          uint4 q;
          memcpy(&q, &opay[c * (16 / C::PB)], 16);
          *reinterpret_cast<uint4 *>(buf(b) + C::KEY_AREA + swz128(diag * (uint32_t)C::PB + 16u * c)) = q;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        if (j < valid) {
          *reinterpret_cast<K *>(buf(b) + swz128((diag + j) * (uint32_t)sizeof(K))) = okey[j];
          if constexpr (HP)
            *reinterpret_cast<P *>(buf(b) + C::KEY_AREA + swz128((diag + j) * (uint32_t)C::PB)) = opay[j];
        }
      }
    }
    if (valid > 0 && o0 + (uint64_t)valid > args.covered_out) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        if (j < valid && o0 + j >= args.covered_out) {
          args.out[o0 + j] = okey[j];
          if constexpr (HP) args.outv[o0 + j] = opay[j];
        }
      }
    }
    fence_proxy_async_smem();  // the tensor stores read what this thread wrote
    __syncwarp();
    if (lane == 0) mbar_arrive(&s_out[b]);
  }
}

constexpr int kOther = 1 << 30;  // no status

template <typename K>
size_t merge_ws_bytes(uint64_t n) {
  const uint64_t tiles = (n + MergeCfg<K, NoPayload>::TILE - 1) / MergeCfg<K, NoPayload>::TILE;
  return kHeaderBytes + align_up((tiles + 1) * sizeof(uint64_t), 256);
}

template <typename K, typename P>
int merge_launch(const K *a, const P *av, uint64_t na, const K *b, const P *bv, uint64_t nb, K *out, P *outv,
                 void *d_ws, size_t ws_bytes, cudaStream_t stream) {
  using C = MergeCfg<K, P>;
  host::DeviceInfo di;
  int st = host::device_info(&di);
  if (st != BK_OK) return st;
  const uint64_t n = na + nb;
  if (n == 0) return BK_OK;
  if ((na && a == nullptr) || (nb && b == nullptr) || out == nullptr) return BK_ERR_INVALID_ARGUMENT;
  if (has_payload<P>() && ((na && av == nullptr) || (nb && bv == nullptr) || outv == nullptr))
    return BK_ERR_INVALID_ARGUMENT;
  if (!host::aligned_to<K>(a) || !host::aligned_to<K>(b) || !host::aligned_to<K>(out)) return BK_ERR_MISALIGNED;
  if constexpr (has_payload<P>()) {
    if (!host::aligned_to<P>(av) || !host::aligned_to<P>(bv) || !host::aligned_to<P>(outv)) return BK_ERR_MISALIGNED;
  }
  const uint64_t tiles = (n + C::TILE - 1) / C::TILE;
  if (tiles >= 0x7fffffffull) return BK_ERR_TOO_LARGE;
  st = host::check_ws(d_ws, ws_bytes, merge_ws_bytes<K>(n));
  if (st != BK_OK) return st;
  WsHeader *hdr = reinterpret_cast<WsHeader *>(d_ws);

  MergeArgs<K, P> args;
  memset(&args, 0, sizeof(args));
  args.a = a;
  args.av = av;
  args.na = na;
  args.b = b;
  args.bv = bv;
  args.nb = nb;
  args.out = out;
  args.outv = outv;
  args.tiles = tiles;
  auto a16 = [](const void *p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const bool tma_in = a16(a) && a16(b) && a16(av) && a16(bv);  // inputs arrive by bulk copies
  // output row views: the outputs inside whole 128-byte rows of both leave by
  // tensor stores, the rest by plain stores
  const uint64_t krows = n * sizeof(K) / 128, prows = n * (uint64_t)C::PB / 128;
  if (a16(out) && a16(outv) && krows > 0 && host::encode_rows_128b(&args.okmap, out, krows, C::KROWS) == BK_OK) {
    args.covered_out = krows * (128 / sizeof(K));
    if constexpr (has_payload<P>()) {
      if (prows > 0 && host::encode_rows_128b(&args.opmap, outv, prows, C::PROWS) == BK_OK)
        args.covered_out = std::min<uint64_t>(args.covered_out, prows * (128 / C::PB));
      else
        args.covered_out = 0;
    }
  }
  const size_t smem = merge_smem_bytes<K, P>();
  const tune::Knobs kn = tune::knobs_for(tune::kMerge, (int)(sizeof(K) + C::PB), n);
  const host::DebugFault dbg = host::debug_fault();
  const unsigned long long limit = dbg.spin_limit_ns ? dbg.spin_limit_ns : host::kDefaultSpinLimitNs;
  // Many tiles a CTA: a partition kernel first, whose splits cost the loader
  // nothing; few: the loader finds them (see merge_kernel).  Measured on a
  // B200, partition / loader: i32/u32 2 x 2^18 13.3 / 9.7 us, 2 x 2^22 38.9 /
  // 35.3, 2 x 2^23 (9 tiles a CTA) random 60.4 / 65.9 and of few values 89.1 /
  // 84.5, 2 x 2^24 (18) 105 / 111; f64/u32 2 x 2^21 33.8 / 31.2, 2 x 2^22 (9)
  // 51.2 / 57.9, 2 x 2^24 163 / 178; f64 2 x 2^22 (9) 44.0 / 43.5, 2 x 2^23
  // 70.6 / 72.2; i32 2 x 2^18 11.2 / 8.7, 2 x 2^26 257 / 256 (keys of 4 bytes
  // alone never need it).
  constexpr uint64_t kPerCta = C::PB == 0 ? (sizeof(K) == 4 ? ~0ull : 16) : (sizeof(K) == 4 ? 16 : 8);
  // With a partition kernel the CTAs' tiles are interleaved, so that all of
  // them read and write close to one another; 4-byte keys from 32 tiles a CTA
  // on do better with a run each.  Interleaved / runs: i32/u32 2 x 2^24 (18 a
  // CTA) 107.5 / 111.6 us, 2 x 2^25 (37) 208.8 / 202.7, 2 x 2^26 403 / 397;
  // i32/u64 2 x 2^24 (28) 151.6 / 158.7, 2 x 2^25 (55) 293.7 / 286.6; f64/u32
  // 7 + 9 million 83.9 / 91.1, 2 x 2^25 of few values 280 / 290; f64/u64 60
  // million + 1000 309 / 328.
  constexpr uint64_t kRunsFrom = sizeof(K) == 4 ? 32 : ~0ull;
  auto launch = [&](auto tma, auto parted) -> int {  // kOther when the other source of splits is the better one
    constexpr bool PARTS = decltype(parted)::value;
    auto kern = merge_kernel<K, P, decltype(tma)::value, PARTS>;
    struct Site {};
    host::KernelSetup ks;
    int e = host::kernel_setup<Site>(kern, kMergeThreads, smem, &ks);
    if (e != BK_OK) return e;
    const uint64_t per_sm = ks.resident_ctas / (uint64_t)di.sm_count;  // what fits (shared memory, registers)
    const uint64_t want = (uint64_t)di.sm_count * (uint64_t)std::max(kn.ctas_per_sm, 1);
    const unsigned grid =
        (unsigned)std::min<uint64_t>(tiles, std::min<uint64_t>(want, std::max<uint64_t>(per_sm, 1) * di.sm_count));
    if (!PARTS && tiles / kPerCta >= grid) return kOther;
    if constexpr (PARTS) {
      uint64_t *parts = reinterpret_cast<uint64_t *>(reinterpret_cast<char *>(d_ws) + kHeaderBytes);
      const uint64_t np = tiles + 1;
      e = host::launch_overlapped(merge_partition_kernel<K>, (unsigned)((np + 255) / 256), 256, 0, stream, 1, a, na, b, nb,
                                  (uint64_t)C::TILE, np, parts);
      if (e != BK_OK) return e;
      args.parts = parts;
      args.strided = tiles / kRunsFrom < grid;
    }
    return host::launch_overlapped(kern, grid, kMergeThreads, smem, stream, 1, args, hdr, limit);
  };
  auto merge = [&](auto tma) -> int {
    const int e = launch(tma, std::false_type());
    if constexpr (kPerCta != ~0ull) {
      if (e == kOther) return launch(tma, std::true_type());
    }
    return e;
  };
  return tma_in ? merge(std::true_type()) : merge(std::false_type());
}

size_t merge_workspace_bytes(int key_dtype, int value_dtype, uint64_t n) {
  if (value_dtype != BK_DTYPE_NONE && value_dtype != BK_DTYPE_U32 && value_dtype != BK_DTYPE_U64 &&
      value_dtype != BK_DTYPE_I32 && value_dtype != BK_DTYPE_I64 && value_dtype != BK_DTYPE_F32 &&
      value_dtype != BK_DTYPE_F64)
    return 0;
  switch (key_dtype) {
    case BK_DTYPE_I32: case BK_DTYPE_U32: case BK_DTYPE_F32: return merge_ws_bytes<float>(n);
    case BK_DTYPE_I64: case BK_DTYPE_U64: case BK_DTYPE_F64: return merge_ws_bytes<double>(n);
    default: return 0;
  }
}

}  // namespace bk

#define BK_DEFINE_MERGE(KN, K)                                                                               \
  extern "C" int bk_merge_##KN(const K *a, uint64_t na, const K *b, uint64_t nb, K *out, void *d_ws,         \
                               size_t ws_bytes, bk_stream_t stream) {                                       \
    return bk::merge_launch<K, bk::NoPayload>(a, nullptr, na, b, nullptr, nb, out, nullptr, d_ws, ws_bytes,  \
                                              (cudaStream_t)stream);                                        \
  }                                                                                                          \
  extern "C" int bk_merge_by_key_##KN##_u32(const K *a_keys, const uint32_t *a_vals, uint64_t na,            \
                                            const K *b_keys, const uint32_t *b_vals, uint64_t nb,            \
                                            K *out_keys, uint32_t *out_vals, void *d_ws, size_t ws_bytes,    \
                                            bk_stream_t stream) {                                           \
    return bk::merge_launch<K, uint32_t>(a_keys, a_vals, na, b_keys, b_vals, nb, out_keys, out_vals, d_ws,   \
                                         ws_bytes, (cudaStream_t)stream);                                   \
  }                                                                                                          \
  extern "C" int bk_merge_by_key_##KN##_u64(const K *a_keys, const uint64_t *a_vals, uint64_t na,            \
                                            const K *b_keys, const uint64_t *b_vals, uint64_t nb,            \
                                            K *out_keys, uint64_t *out_vals, void *d_ws, size_t ws_bytes,    \
                                            bk_stream_t stream) {                                           \
    return bk::merge_launch<K, unsigned long long>(                                                          \
        a_keys, reinterpret_cast<const unsigned long long *>(a_vals), na, b_keys,                            \
        reinterpret_cast<const unsigned long long *>(b_vals), nb, out_keys,                                  \
        reinterpret_cast<unsigned long long *>(out_vals), d_ws, ws_bytes, (cudaStream_t)stream);             \
  }

BK_DEFINE_MERGE(i32, int32_t)
BK_DEFINE_MERGE(u32, uint32_t)
BK_DEFINE_MERGE(i64, int64_t)
BK_DEFINE_MERGE(u64, uint64_t)
BK_DEFINE_MERGE(f32, float)
BK_DEFINE_MERGE(f64, double)
