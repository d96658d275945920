// radix_sort.cu -- stable LSD radix sort by key (the sort_by_key entry
// points below 2^30 elements), sm_100a.
//
// The reference sorts by merging (stable_merge_sort_by_key,
// merge_sort_by_key.cu:150-209): ceil(log2(n / 896)) global passes, 17 at
// 2^26.  A stable sort's output is unique -- equal keys keep their input
// order -- so a stable least-significant-digit radix sort gives exactly the
// same keys and payloads, in sizeof(K) passes of 8 bits instead: 4 for 32-bit
// keys, 8 for 64-bit ones.  Keys are mapped to unsigned integers with the same
// order (signed: flip the sign bit; floating point: flip all bits of
// negatives and the sign bit of the rest, with -0.0 read as +0.0 so that the
// two zeros tie as they do under operator<).  Keys must not be NaN.
//
// One kernel counts every pass's digits in one read of the keys; then each
// pass is one kernel (rs_pass_kernel) that reads the keys once and writes them
// once: a tile is ranked by digit and staged in shared memory in digit order,
// where its keys of a digit go follows from the counts and a look-back over
// the groups of tiles before it, and each digit's run is written contiguously
// to its position.  Large arrays of 8-byte keys are sorted by their upper four
// digits alone where those tell the keys apart well enough (RsPlanWs below).
//
// A single array of up to 131,072 keys is sorted instead by one launch of one
// thread-block cluster whose CTAs exchange their digit counts through
// distributed shared memory (rs_cluster_kernel below), of up to 4096 keys by
// one CTA (rs_block_kernel).
#include <type_traits>

#include "bk_common.cuh"
#include "bk_tune.hpp"
#include "bk_merge.cuh"  // NoPayload, has_payload, payload_bytes
#include "bk_tma.cuh"    // smem_addr, mbarriers
#include "bulk_b200.h"

namespace bk {

constexpr int kRsBins = 256;                    // 8-bit digits
constexpr uint64_t kRsMaxN = 1ull << 30;
constexpr int kRsBatchMax = 256;
constexpr int kRsWindow = 32;                   // words a lane of the scout reads in one look-back round

// Order-preserving map of a key to an unsigned integer.
template <typename K>
struct RadixKey;
template <>
struct RadixKey<uint32_t> {
  using U = uint32_t;
  static __device__ __forceinline__ U to(uint32_t k) { return k; }
};
template <>
struct RadixKey<int32_t> {
  using U = uint32_t;
  static __device__ __forceinline__ U to(int32_t k) { return (uint32_t)k ^ 0x80000000u; }
};
template <>
struct RadixKey<float> {
  using U = uint32_t;
  static __device__ __forceinline__ U to(float k) {
    uint32_t b = __float_as_uint(k);
    if (b == 0x80000000u) b = 0u;  // -0.0 ties with +0.0
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  }
};
template <>
struct RadixKey<uint64_t> {
  using U = uint64_t;
  static __device__ __forceinline__ U to(uint64_t k) { return k; }
};
template <>
struct RadixKey<int64_t> {
  using U = uint64_t;
  static __device__ __forceinline__ U to(int64_t k) { return (uint64_t)k ^ 0x8000000000000000ull; }
};
template <>
struct RadixKey<double> {
  using U = uint64_t;
  static __device__ __forceinline__ U to(double k) {
    uint64_t b = (uint64_t)__double_as_longlong(k);
    if (b == 0x8000000000000000ull) b = 0ull;
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
  }
};

template <typename K>
constexpr int rs_passes() {
  return (int)sizeof(K);  // 8-bit digits
}

template <typename K>
__device__ __forceinline__ int rs_digit(K k, int shift) {
  return (int)((RadixKey<K>::to(k) >> shift) & (kRsBins - 1));
}

// The eight bits [8 * (pass & 3), +8) of the 32-bit half of `u` that holds
// byte `pass`: the word a digit is taken from.
__device__ __forceinline__ uint32_t rs_word(uint32_t u, int) { return u; }
__device__ __forceinline__ uint32_t rs_word(uint64_t u, int pass) {
  return pass < 4 ? (uint32_t)u : (uint32_t)(u >> 32);
}
// The digits of four keys packed into one word (key i's in byte i): two byte
// permutes pick the digit byte of two keys each, a third joins them.
template <typename K>
__device__ __forceinline__ uint32_t rs_digits4(const K *k, int pass) {
  const uint32_t b = (uint32_t)pass & 3u;
  const uint32_t sel = b | (b + 4u) << 4;
  const uint32_t lo = __byte_perm(rs_word(RadixKey<K>::to(k[0]), pass), rs_word(RadixKey<K>::to(k[1]), pass), sel);
  const uint32_t hi = __byte_perm(rs_word(RadixKey<K>::to(k[2]), pass), rs_word(RadixKey<K>::to(k[3]), pass), sel);
  return __byte_perm(lo, hi, 0x5410);
}

// The digit of one key.
template <typename K>
__device__ __forceinline__ uint32_t rs_digit1(K k, int pass) {
  return __byte_perm(rs_word(RadixKey<K>::to(k), pass), 0u, 0x4440u | ((uint32_t)pass & 3u));
}

// ---------------------------------------------------------------------------
// Ranking the keys of a warp by digit, in input order (the keys' index is
// item * 32 + lane).
//
// For every item a lane needs the set of lanes that hold the same digit.
// Eight ballots with their selects cost about 32 instructions an item on the
// ALU pipe, which issues one warp instruction every two cycles: that pipe
// bounded the scatter (357 us of a 445 us pass at 2^26 u32/u32 keys on a
// B200).  Here four items are matched at a time:
//   transpose  the 32 lanes' words of four packed digits are transposed as a
//              32 x 32 bit matrix (five shuffles): lane 8 * i + b then holds
//              bit b of item i's digit over all lanes, what a ballot gives;
//   tables     from those words lane h * 16 + x of the warp works out, for
//              each item, the set of lanes whose nibble h equals x (four
//              three-input logic operations) and stores it;
//   look-up    a lane's peers are the low nibble's set AND the high nibble's:
//              two shared-memory reads of a 16-word table each, free of bank
//              conflicts whatever the digits are.
// The keys' ranks then come from a counter a digit (256 words a warp): each
// lane reads its digit's counter, adds the peers below it, and the highest
// peer writes the counter back.  No atomics, and no cost that depends on how
// the digits are distributed.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t rs_lds_u16(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
// Stores the low 16 bits of v where `none` is zero (predicated, no branch).
__device__ __forceinline__ void rs_sts_u16_if_zero(uint32_t a, uint32_t v, uint32_t none) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, 0;\n\t@p st.shared.u16 [%0], %1;\n\t}" ::"r"(a), "r"(v),
               "r"(none)
               : "memory");
}
template <int OFF>
__device__ __forceinline__ uint32_t rs_lds_at(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(OFF) : "memory");
  return v;
}
__device__ __forceinline__ void rs_sts(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

class RsRanker {
 public:
  // a warp's tables (512 bytes, on a 256-byte boundary) and transposed bits (128 bytes, on 16)
  __device__ __forceinline__ RsRanker(const void *table, const void *bits)
      : table_(smem_addr(table)), bits_(smem_addr(bits)) {
    const uint32_t lane = threadIdx.x & 31;
    sel16_ = (lane & 16) ? 0x3276u : 0x5410u;
    sel8_ = (lane & 8) ? 0x3715u : 0x6240u;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint32_t lo = i == 0 ? 0x0f0f0f0fu : i == 1 ? 0x33333333u : 0x55555555u;
      keep_[i] = (lane & (4u >> i)) ? ~lo : lo;
      rot_[i] = (lane & (4u >> i)) ? 32 - (4 >> i) : (4 >> i);
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) not_[b] = (lane >> b) & 1u ? 0u : ~0u;
    lt_ = (1u << lane) - 1u;
    gt_ = ~(lt_ | (1u << lane));
  }

  // rank2[j / 2] receives four times item j's rank among the warp's keys of
  // its digit, in 16 bits; digits of items 4i .. 4i + 3 are packed in
  // dig4[i].  The counters (256 16-bit words; one digit's counter counts by four)
  // start zeroed and end as four times the warp's count of each digit.
  template <int ITEMS>
  __device__ __forceinline__ void rank(const uint16_t *counters, const uint32_t (&dig4)[ITEMS / 4],
                                       uint32_t (&rank2)[ITEMS / 2]) const {
    const uint32_t cbase = smem_addr(counters);
#pragma unroll
    for (int g = 0; g < ITEMS / 4; ++g) {
      uint32_t peers[4];
      match4(dig4[g], peers);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t c = cbase + 2u * __byte_perm(dig4[g], 0u, 0x4440u | (uint32_t)i);
        const uint32_t r = rs_lds_u16(c) + 4u * (uint32_t)__popc(peers[i] & lt_);
        __syncwarp();
        rs_sts_u16_if_zero(c, r + 4u, peers[i] & gt_);
        __syncwarp();
        const int j = 4 * g + i;
        if (j & 1) rank2[j >> 1] |= r << 16;
        else rank2[j >> 1] = r;
      }
    }
  }

 private:
  // peers[i]: the lanes whose byte i of `d` equals this lane's.
  __device__ __forceinline__ void match4(uint32_t d, uint32_t (&peers)[4]) const {
    const uint32_t lane = threadIdx.x & 31;
    // bit (lane, column) -> (column, lane): swap off-diagonal blocks of 16, 8, 4, 2, 1
    uint32_t x = d;
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), sel16_);
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), sel8_);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4 >> i);
      x = (x & keep_[i]) | (__funnelshift_l(y, y, rot_[i]) & ~keep_[i]);
    }
    rs_sts(bits_ + 4u * lane, x);
    __syncwarp();
    const uint32_t src = bits_ + (lane & 16u);  // lanes 16-31 read the high nibble's four words
    const uint32_t dst = table_ + 4u * lane;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 v;
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                   : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                   : "r"(src + 32u * i)
                   : "memory");
      // lanes whose nibble equals this lane's number mod 16, bit by bit
      rs_sts(dst + 128u * i, (v.x ^ not_[0]) & (v.y ^ not_[1]) & (v.z ^ not_[2]) & (v.w ^ not_[3]));
    }
    __syncwarp();
    // byte i of lo / hi: the byte offset of the item's entry in the low / high nibble's table
    const uint32_t lo = (d << 2) & 0x3c3c3c3cu, hi = (d >> 2) & 0x3c3c3c3cu;
    peers[0] = rs_lds_at<0>(__byte_perm(lo, table_, 0x7650)) & rs_lds_at<64>(__byte_perm(hi, table_, 0x7650));
    peers[1] = rs_lds_at<128>(__byte_perm(lo, table_, 0x7651)) & rs_lds_at<192>(__byte_perm(hi, table_, 0x7651));
    peers[2] = rs_lds_at<256>(__byte_perm(lo, table_, 0x7652)) & rs_lds_at<320>(__byte_perm(hi, table_, 0x7652));
    peers[3] = rs_lds_at<384>(__byte_perm(lo, table_, 0x7653)) & rs_lds_at<448>(__byte_perm(hi, table_, 0x7653));
  }

  uint32_t table_, bits_;
  uint32_t sel16_, sel8_, keep_[3], rot_[3], not_[4], lt_, gt_;
};

// ---------------------------------------------------------------------------
// Cluster helpers (also for a cluster of one CTA).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t rs_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t rs_cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Barrier over every thread of the cluster; earlier shared-memory writes
// (local and remote) are visible to every thread after it.
__device__ __forceinline__ void rs_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of `local` (this CTA's shared memory) in CTA `rank`'s window.
__device__ __forceinline__ uint32_t rs_peer_addr(const void *local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr(local)), "r"(rank));
  return r;
}
// Load from another CTA's shared memory.  The cluster barriers around its
// uses order it, so it has no memory clobber and one thread's loads may all
// be in flight at once.
__device__ __forceinline__ uint32_t rs_peer_ld_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
// mbarriers initialised before this are ready for the cluster after its next barrier.
__device__ __forceinline__ void rs_fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Bounded wait for phase `parity` of a barrier that other CTAs of the cluster
// complete; what they stored with it is visible after it.
__device__ __forceinline__ bool rs_wait_cluster(uint64_t *bar, uint32_t parity, unsigned long long limit_ns) {
  const uint32_t a = smem_addr(bar);
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 15u) == 15u) {
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > limit_ns) return false;
    }
  }
}
// Stores v in CTA `rank`'s copy of *local and completes four bytes on its copy
// of `bar`: a thread that saw the barrier's phase complete reads the value,
// with no fence on either side.
__device__ __forceinline__ void rs_push_u32(const void *local, uint32_t v, const uint64_t *bar, uint32_t rank) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(
                   rs_peer_addr(local, rank)),
               "r"(v), "r"(rs_peer_addr(bar, rank))
               : "memory");
}
// Exclusive sum scan of v over threads 0-255 of the CTA (the digit threads;
// the other warps do not take part), with the total; s_w holds 8 words.
__device__ __forceinline__ unsigned int rs_scan_digits(unsigned int v, unsigned int *s_w, unsigned int &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned int incl = warp_inclusive_scan(v, OpSum<unsigned int>(), lane);
  if (lane == 31) s_w[warp] = incl;
  named_barrier_sync(1, kRsBins);
  unsigned int pre = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kRsBins / 32; ++w) {
    const unsigned int x = s_w[w];
    tot += x;
    if (w < warp) pre += x;
  }
  total = tot;
  return pre + incl - v;
}

// ---------------------------------------------------------------------------
// Global-memory passes.
// ---------------------------------------------------------------------------
// A CTA's tile: THREADS threads of ITEMS keys (and one more warp, the scout),
// two CTAs an SM.  The thread count is the largest whose registers hold the
// keys and payloads without spilling: on a B200, 2^26 pairs, 416 threads sort
// u32/u32 in 1.40 ms (480 spill: 1.44; 256, three CTAs an SM: 1.68), 288 sort
// u64/u32 in 3.50 ms (256: 4.02, 320 and 352 spill: 3.84, 3.71; 352 of 12
// keys: 3.58).
template <typename K, typename P>
struct RsCfg {
  static constexpr int BYTES = (int)sizeof(K) + payload_bytes<P>();
  static constexpr int ITEMS = BYTES <= 12 ? 16 : 12;
  static constexpr int THREADS = BYTES <= 8 && sizeof(K) == 4 ? 416 : 288;
  static constexpr int TILE = THREADS * ITEMS;
  static constexpr int WARPS = THREADS / 32;
  static constexpr int CTA_THREADS = THREADS + 32;
  static constexpr int MIN_BLOCKS = 2;
  static_assert(THREADS >= kRsBins, "threads 0-255 are the digit threads");
};

// A group of C tiles of one array, which one cluster of C CTAs sorts by one
// digit: its array (keys and temporaries: even passes read the keys, odd
// passes the temporaries), length, the group's index in the array and the
// array's index in the batch.
template <typename K, typename P>
struct RsGroup {
  K *keys;
  P *vals;
  K *tk;
  P *tv;
  const K *src_k;       // what the first pass reads (keys, or a separate source)
  const P *src_v;
  uint64_t n;
  uint32_t local;
  uint32_t array;
};

template <typename K, typename P>
struct RsOne {
  K *keys;
  P *vals;
  K *tk;
  P *tv;
  uint64_t n;
  static constexpr bool kMany = false;
  __device__ __forceinline__ unsigned int find(unsigned int) const { return 0u; }
  __device__ __forceinline__ RsGroup<K, P> group(unsigned int g, unsigned int = 0u) const {
    return RsGroup<K, P>{keys, vals, tk, tv, keys, vals, n, g, 0u};
  }
};

// A batch: array i owns groups [start[i], start[i + 1]).
template <typename K, typename P>
struct RsBatch {
  K *keys[kRsBatchMax];
  P *vals[kRsBatchMax];
  const K *src_k[kRsBatchMax];  // what the first pass reads
  const P *src_v[kRsBatchMax];
  K *tk[kRsBatchMax];
  P *tv[kRsBatchMax];
  uint64_t n[kRsBatchMax];
  uint32_t start[kRsBatchMax + 1];
  uint32_t count;
  static constexpr bool kMany = true;
  // the array that owns group g
  __device__ __forceinline__ unsigned int find(unsigned int g) const {
    int lo = 0, hi = (int)count - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (start[mid] <= g) lo = mid;
      else hi = mid - 1;
    }
    return (unsigned int)lo;
  }
  __device__ __forceinline__ RsGroup<K, P> group(unsigned int g, unsigned int a) const {
    return RsGroup<K, P>{keys[a], vals[a], tk[a], tv[a], src_k[a], src_v[a], n[a], g - start[a], a};
  }
  __device__ __forceinline__ RsGroup<K, P> group(unsigned int g) const { return group(g, find(g)); }
};

// Elements of tile `rank` of group `g` (0 past the array's end) and where it starts.
template <typename K, typename P>
__device__ __forceinline__ int rs_tile_count(const RsGroup<K, P> &g, uint64_t base) {
  constexpr int T = RsCfg<K, P>::TILE;
  return base >= g.n ? 0 : (g.n - base) < (uint64_t)T ? (int)(g.n - base) : T;
}

// ---- 8-byte keys: the upper half of the digits first.
//
// A large array's 8-byte keys seldom agree in their upper 32 bits unless they
// are drawn from few values.  Where they do not, four passes over the upper
// digits leave only short runs of keys that agree there, in input order, and
// one read of the keys finds and sorts those runs in place: half the passes.
// A sample decides which of the two an array gets (rs_sample_kernel); every
// kernel launched after it works the decision out (a kernel with nothing to
// do leaves at once):
//   full    the passes of digits 0-3 and 4-7
//   upper   the passes of digits 4-7, then rs_fix_kernel; where that met runs
//           longer than it sorts and out of order (the sample missed them),
//           rs_late_kernel sorts those
//   rescue  more or longer runs than rs_late_kernel takes: the passes of
//           digits 0-3 and 4-7 follow.  The array then holds its keys in
//           another order, but equal keys still in input order, so the result
//           is the same.
struct RsPlanWs {
  unsigned int repeats;    // sampled keys whose upper half another one has
  unsigned int zeros;      // sampled keys whose upper half is zero
  unsigned int unordered;  // a run that rs_fix_kernel left alone is out of order
  unsigned int too_many;   // such runs do not fit their list, or one is longer than rs_late_kernel takes
  unsigned int runs[2];    // listed runs: of up to kRsRunWarp keys, longer
  unsigned int pad[2];
};
enum RsPlan { kPlanFull, kPlanUpper, kPlanRescue };

constexpr int kRsSampleThreads = 512, kRsSampleCtas = 32, kRsSamples = kRsSampleThreads * kRsSampleCtas;
constexpr int kRsSampleSlots = 65536;
constexpr uint32_t kRsSampleWindow = 65536;   // keys a CTA samples from
// From here on arrays are planned.  u64/u32 on a B200, planned / all eight
// passes: random keys 2^20 95 / 111 us, 2^22 183 / 269, 2^25 1018 / 1767, 2^26
// 1967 / 3457; keys of 1000 values (the plan is all passes, and the idle
// launches are lost) 2^20 123 / 96, 2^22 252 / 224, 2^25 1533 / 1499, 2^26
// 2956 / 2921.  f64 uniform in [-1, 1): 2^22 217 / 284, 2^25 1570 / 1912, but
// 2^26 3821 / 3782, where the plan is all passes.
constexpr uint64_t kRsPlanMinN = 1ull << 22;
// What rs_late_kernel takes: runs of up to kRsRunWarp keys a warp each, of up to
// kRsRunMax a CTA each.  They are listed in the status rows that the passes
// between use next (one word in 54 to 72 keys): the longer ones from the end.
// Without it one such run sent the array to the rescue, whose twelve passes
// take longer than eight by separate counting and scattering did.  u64/u32 on a
// B200, random keys and some such runs: those eight 430 us at 2^22 and 4610 at
// 2^26, rescue 471 and 5408, now, by the runs: one of 400 231 and 2015, one of
// 60,000 299 (all passes) and 2280, one of 66 keys for each 1000 300 and 2850.
// (Runs of 1000 by a warp each took 409 us at 2^22, by a CTA 232.)
constexpr unsigned int kRsRunWarp = 256, kRsRunMax = 131072;
struct RsRunList {
  unsigned int *start;  // where each run begins
  unsigned int room;
  __device__ __forceinline__ unsigned int room_for(bool longer, uint32_t n) const {
    return longer ? n / kRsRunWarp : room - n / kRsRunWarp;
  }
  __device__ __forceinline__ unsigned int *slot(bool longer, unsigned int i) const {
    return start + (longer ? room - 1u - i : i);
  }
};

// A key's run has on average 1 + n * sum(p^2) keys (p the shares of the upper
// halves' values), of which the sample's repeats estimate 2 * repeats /
// samples^2: the upper digits alone are sorted by up to an average of about 8.
__device__ __forceinline__ RsPlan rs_plan(const RsPlanWs *plan, uint64_t n) {
  if (plan == nullptr) return kPlanFull;
  const uint4 w = ld_cg_v4(plan);
  if (w.z != 0u && w.w != 0u) return kPlanRescue;
  return (uint64_t)w.x * n <= 4ull * kRsSamples * kRsSamples ? kPlanUpper : kPlanFull;
}

// The digit that launch `launch` of an array's passes (three blocks of four)
// sorts by, -1 for none; without a plan launch i sorts by digit i.
__device__ __forceinline__ int rs_launch_digit(int launch, const RsPlanWs *plan, uint64_t n) {
  if (plan == nullptr) return launch;
  const RsPlan p = rs_plan(plan, n);
  const int block = launch >> 2, i = launch & 3;
  if (p == kPlanFull) return block < 2 ? launch : -1;
  if (p == kPlanUpper) return block == 0 ? 4 + i : -1;
  return block == 1 ? i : 4 + i;
}

// Clears the counts, tickets and sample (a kernel, not a memset, so that its
// launch and its successor's overlap as all others here do).
__global__ void rs_zero_kernel(uint4 *p, uint32_t vecs) {
  grid_dependency_wait();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < vecs; i += gridDim.x * blockDim.x)
    p[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Every CTA takes one key from each 128th of a random window of 65,536 keys
// and enters its upper half in a table of values seen (zeroed before; a zero
// half is counted apart).  Windows, because reading 16,384 keys all over 2^26
// costs their address translation; 128 keys apart, so that a sorted array's
// runs that are short enough to be sorted in place rarely count.  The positions
// come from MurmurHash3's 32-bit finaliser, the table's slots from Fibonacci
// hashing (both published).
template <typename K>
__global__ void __launch_bounds__(kRsSampleThreads) rs_sample_kernel(const K *keys, uint32_t n, unsigned int *table,
                                                                     RsPlanWs *plan) {
  constexpr uint32_t STRIDE = kRsSampleWindow / kRsSampleThreads;
  auto mixed = [](unsigned int x) {
    unsigned int h = (x + 1u) * 0x9e3779b1u;
    h = (h ^ (h >> 15)) * 0x85ebca6bu;
    h = (h ^ (h >> 13)) * 0xc2b2ae35u;
    return h ^ (h >> 16);
  };
  grid_dependency_wait();
  const unsigned int me = blockIdx.x * kRsSampleThreads + threadIdx.x;
  const uint64_t window = (uint64_t)mixed(blockIdx.x) * (n - kRsSampleWindow) >> 32;
  const uint32_t at_key = threadIdx.x * STRIDE + mixed(me + kRsSampleCtas) % STRIDE;
  const unsigned int up = (unsigned int)(RadixKey<K>::to(keys[window + at_key]) >> 32);
  bool repeat = false;
  if (up == 0u) {
    repeat = atomicAdd(&plan->zeros, 1u) != 0u;
  } else {
    unsigned int at = (up * 0x9e3779b1u) / (unsigned int)(0x100000000ull / kRsSampleSlots);
    for (int probe = 0; probe < kRsSamples; ++probe) {  // ends before: a quarter of the slots are taken at most
      const unsigned int was = atomicCAS(table + at, 0u, up);
      repeat = was == up;
      if (was == 0u || repeat) break;
      at = (at + 1) & (kRsSampleSlots - 1);
    }
  }
  const int repeats = __syncthreads_count(repeat);
  if (threadIdx.x == 0 && repeats != 0) atomicAdd(&plan->repeats, (unsigned int)repeats);
}

// Sorts every run of keys with equal upper halves (all of them in input order
// within a run) by the lower halves, in place.  A warp sorts the runs that
// start in its chunk of keys, which may reach into the kRsFixHalo keys after
// it; the warp there sees that its first keys belong to an earlier run (their
// upper halves do not change) and leaves those in the halo alone.  A key's
// place in its run is the number of keys before it with a lower half not above
// its own plus the number after it with one below: runs are a few keys long,
// and a key without equal neighbours costs two comparisons.  A run longer than
// kRsFixHalo is left as it is and entered in a list by the warp that sees its
// first key.  The list matters only when one of those runs is out of order
// (not one value many times): each of their keys is compared with the one
// before, by the warp before for a chunk's first kRsFixHalo keys and by the
// chunk's own warp from the next on.  One read of
// the keys, bound by memory where runs are rare; warps work on their own, so
// that one warp's loads run behind another's comparisons (a CTA-wide tile of
// 4096 keys between barriers took 271 us for 2^26 random keys on a B200).
constexpr int kRsFixThreads = 128, kRsFixPer = 8, kRsFixChunk = 32 * kRsFixPer, kRsFixHalo = 64;

template <typename K, typename P>
__global__ void __launch_bounds__(kRsFixThreads, 10) rs_fix_kernel(K *keys, P *vals, uint32_t n, RsPlanWs *plan,
                                                                     RsRunList list) {
  constexpr int WARPS = kRsFixThreads / 32, LEN = kRsFixChunk + kRsFixHalo, PER = LEN / 32;
  using V = typename std::conditional<has_payload<P>(), P, char>::type;
  grid_dependency_wait();
  if (rs_plan(plan, n) == kPlanFull) return;
  // the keys' halves (up[-1]: of the key before the chunk); later, in the same
  // place, the keys that move, at their new places
  __shared__ uint64_t s_halves[WARPS][LEN + 1];
  __shared__ uint16_t s_to[WARPS][LEN];  // where a key that moves goes
  __shared__ V s_val[WARPS][has_payload<P>() ? LEN : 1];  // the payloads of the keys that move
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned int *low = reinterpret_cast<unsigned int *>(s_halves[warp]), *up = low + LEN + 1;
  K *moved = reinterpret_cast<K *>(s_halves[warp]);
  const uint64_t step = (uint64_t)gridDim.x * WARPS * kRsFixChunk;
  for (uint64_t base = ((uint64_t)blockIdx.x * WARPS + warp) * kRsFixChunk; base < n; base += step) {
    const int len = (int)((n - base) < (uint64_t)LEN ? (n - base) : (uint64_t)LEN);
    K *const kp = keys + base;
    {
      K k[PER];
#pragma unroll
      for (int j = 0; j < PER; ++j)
        if (j * 32 + lane < len) k[j] = kp[j * 32 + lane];
      if (lane == 0) {
        const unsigned int u = (unsigned int)(RadixKey<K>::to(base > 0 ? kp[-1] : k[0]) >> 32);
        up[-1] = base > 0 ? u : ~u;
      }
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        if (j * 32 + lane < len) {
          const uint64_t u = RadixKey<K>::to(k[j]);
          low[j * 32 + lane] = (unsigned int)u;
          up[j * 32 + lane] = (unsigned int)(u >> 32);
        }
      }
    }
    __syncwarp();
    unsigned int todo = 0;  // bit j: key j * 32 + lane has an equal neighbour
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int i = j * 32 + lane;
      if (i < len && (up[i - 1] == up[i] || (i + 1 < len && up[i + 1] == up[i]))) todo |= 1u << j;
    }
    unsigned int moves = 0;
    while (todo != 0) {
      const int j = __ffs(todo) - 1, i = j * 32 + lane;
      todo &= todo - 1;
      const unsigned int u = up[i], l = low[i];
      int first = i, last = i, rank = 0;  // the run is [first, last]
      while (first > 0 && last - first < kRsFixHalo && up[first - 1] == u) {
        --first;
        rank += low[first] <= l;
      }
      // another warp's: the run begins before the chunk and the key lies in the
      // halo of the warp before, or it begins in the halo
      if ((first == 0 && up[-1] == u && i < kRsFixHalo) || first >= kRsFixChunk) continue;
      while (last - first < kRsFixHalo && last + 1 < len && up[last + 1] == u) {
        ++last;
        rank += low[last] < l;
      }
      if (last - first >= kRsFixHalo) {  // (true of a run that reaches the halo's end)
        if (i > first) {
          if (low[i - 1] > l) plan->unordered = 1u;
        } else {  // its first key
          auto reaches = [&](unsigned int q) {  // key q of the run, counted from 0
            return n - base - i > q && (unsigned int)(RadixKey<K>::to(kp[i + q]) >> 32) == u;
          };
          const bool longer = reaches(kRsRunWarp);
          const unsigned int at = atomicAdd(&plan->runs[longer], 1u);
          if (at >= list.room_for(longer, n) || (longer && reaches(kRsRunMax))) plan->too_many = 1u;
          else *list.slot(longer, at) = (unsigned int)base + (unsigned int)i;
        }
      } else if (first + rank != i) {
        s_to[warp][i] = (uint16_t)(first + rank);
        moves |= 1u << j;
      }
    }
    if (__any_sync(0xffffffffu, moves != 0)) {
      // the places that keys leave are the places that keys take
      __syncwarp();
      for (unsigned int m = moves; m != 0; m &= m - 1) {
        const int i = (__ffs(m) - 1) * 32 + lane, to = s_to[warp][i];
        moved[to] = kp[i];
        if constexpr (has_payload<P>()) s_val[warp][to] = vals[base + i];
      }
      __syncwarp();  // everything is read before anything is written
      for (unsigned int m = moves; m != 0; m &= m - 1) {
        const int i = (__ffs(m) - 1) * 32 + lane;
        kp[i] = moved[i];
        if constexpr (has_payload<P>()) vals[base + i] = s_val[warp][i];
      }
    }
    __syncwarp();
  }
}

// ---- digit counts of every pass in one read of the keys.
// Counters are spread over columns by lane, so that no two lanes of a warp
// (two, where eight digits are counted) ever meet in a bank, however the
// digits are distributed; a CTA adds its sums to the array's counts when its
// run of tiles leaves the array.  128 KB of counters, one CTA of 1024 threads
// an SM.  With a plan it counts the digits that the passes after it need
// (rs_late_kernel counts the rest for the rescue).  It also clears the status
// rows that the first pass will publish in.
constexpr int kRsHistThreads = 1024;
constexpr size_t kRsHistSmemBytes = 128 * 1024;

// Counts digits [FIRST, FIRST + DIGITS); the counters in shared memory start zeroed.
template <typename K, typename P, typename Src, int C, int FIRST, int DIGITS>
__device__ __forceinline__ void rs_count_digits(const Src &src, unsigned int groups, unsigned int *hist) {
  constexpr int BINS = DIGITS * kRsBins, COPIES = (int)(kRsHistSmemBytes / 4) / BINS;
  constexpr int TILE = RsCfg<K, P>::TILE;
  constexpr int VEC = 16 / (int)sizeof(K), UNROLL = 4;
  extern __shared__ __align__(16) unsigned int rs_hist_smem[];
  const int tid = threadIdx.x, lane = tid & 31;
  unsigned int *col = rs_hist_smem + (lane & (COPIES - 1));
  auto add = [&](K key) {
    const auto u = RadixKey<K>::to(key);
#pragma unroll
    for (int p = 0; p < DIGITS; ++p)
      atomicAdd(col + (p * kRsBins + (int)((u >> (8 * (FIRST + p))) & 0xffu)) * COPIES, 1u);
  };
  const uint64_t tiles = (uint64_t)groups * C;
  uint64_t t = tiles * blockIdx.x / gridDim.x;
  const uint64_t t_end = tiles * (blockIdx.x + 1) / gridDim.x;
  __syncthreads();
  while (t < t_end) {
    // the part of this CTA's tiles that lies in one array
    const RsGroup<K, P> gr = src.group((unsigned int)(t / C));
    const uint64_t first = (uint64_t)gr.local * C + t % C;  // tile within the array
    const uint64_t arr_tiles = (gr.n + (uint64_t)(C * TILE) - 1) / (uint64_t)(C * TILE) * C;
    const uint64_t take = (arr_tiles - first) < (t_end - t) ? (arr_tiles - first) : (t_end - t);
    const uint64_t lo = first * TILE;
    const uint64_t hi = (first + take) * TILE < gr.n ? (first + take) * TILE : gr.n;
    if (lo < hi) {
      const K *p = gr.src_k + lo;
      const uint64_t cnt = hi - lo;
      const uint64_t mis = (reinterpret_cast<uintptr_t>(p) & 15u) / sizeof(K);
      const uint64_t head = mis == 0 ? 0 : (VEC - mis < cnt ? VEC - mis : cnt);
      if ((uint64_t)tid < head) add(p[tid]);
      const uint64_t nv = (cnt - head) / VEC;
      const uint4 *pv = reinterpret_cast<const uint4 *>(p + head);
      for (uint64_t i = tid; i < nv; i += (uint64_t)UNROLL * kRsHistThreads) {
        uint4 v[UNROLL];
#pragma unroll
        for (int q = 0; q < UNROLL; ++q)
          if (i + (uint64_t)q * kRsHistThreads < nv) v[q] = pv[i + (uint64_t)q * kRsHistThreads];
#pragma unroll
        for (int q = 0; q < UNROLL; ++q) {
          if (i + (uint64_t)q * kRsHistThreads < nv) {
            K k[VEC];
            memcpy(k, &v[q], 16);
#pragma unroll
            for (int e = 0; e < VEC; ++e) add(k[e]);
          }
        }
      }
      for (uint64_t i = head + nv * VEC + tid; i < cnt; i += kRsHistThreads) add(p[i]);
    }
    __syncthreads();
    unsigned int *out = hist + ((uint64_t)gr.array * rs_passes<K>() + FIRST) * kRsBins;
    for (int b = tid; b < BINS; b += kRsHistThreads) {
      unsigned int sum = 0;
#pragma unroll 8
      for (int c = 0; c < COPIES; ++c) {
        unsigned int *w = rs_hist_smem + b * COPIES + ((c + lane) & (COPIES - 1));
        sum += *w;
        *w = 0u;
      }
      if (sum != 0) atomicAdd(out + b, sum);
    }
    __syncthreads();
    t += take;
  }
}

template <typename K, typename P, typename Src, int C>
__global__ void __launch_bounds__(kRsHistThreads, 1) rs_hist_kernel(const __grid_constant__ Src src,
                                                                    unsigned int groups, unsigned int *hist,
                                                                    uint4 *status, const RsPlanWs *plan) {
  extern __shared__ __align__(16) unsigned int rs_hist_smem[];
  for (int i = threadIdx.x; i < (int)(kRsHistSmemBytes / 16); i += kRsHistThreads)
    reinterpret_cast<uint4 *>(rs_hist_smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  grid_dependency_wait();
  const RsPlan p = rs_plan(plan, plan != nullptr ? src.group(0).n : 0);
  for (uint64_t i = (uint64_t)blockIdx.x * kRsHistThreads + threadIdx.x; i < (uint64_t)groups * (kRsBins / 4);
       i += (uint64_t)gridDim.x * kRsHistThreads)
    status[i] = make_uint4(0u, 0u, 0u, 0u);
  if constexpr (sizeof(K) == 4) rs_count_digits<K, P, Src, C, 0, 4>(src, groups, hist);
  else if (p == kPlanFull) rs_count_digits<K, P, Src, C, 0, 8>(src, groups, hist);
  else rs_count_digits<K, P, Src, C, 4, 4>(src, groups, hist);
}

// ---- what the fix kernel left: the long runs it listed, or the rescue's counts.
//
// A warp sorts a run of up to kRsRunWarp keys by counting: a key's place is the
// number of keys below it, and of equal ones before it.  The keys go to the
// temporaries (the run's own stretch of them; the passes are done with them)
// and back.  Bound by instructions, about 3.5 a comparison.  A run that is in
// order is passed over.
template <typename K, typename P>
__device__ __forceinline__ void rs_sort_run_warp(K *keys, P *vals, K *tk, P *tv, uint32_t len, uint32_t *low) {
  constexpr int ITEMS = 4;
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t i = lane; i < len; i += 32) low[i] = (uint32_t)RadixKey<K>::to(ld_cg(keys + i));
  if (lane < ((0u - len) & 3u)) low[len + lane] = ~0u;  // not below any key, after all
  __syncwarp();
  bool down = false;
  for (uint32_t i = lane; i + 1 < len; i += 32) down |= low[i] > low[i + 1];
  if (!__any_sync(0xffffffffu, down)) return;
  for (uint32_t first = lane; first - lane < len; first += 32 * ITEMS) {  // this lane's keys: first + 32 j
    uint32_t l[ITEMS], rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      l[j] = first + 32 * j < len ? low[first + 32 * j] : 0u;
      rank[j] = 0u;
    }
    for (uint32_t q = 0; q < len; q += 4) {
      const uint4 x = *reinterpret_cast<const uint4 *>(low + q);
      const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
          rank[j] += (unsigned int)(xs[t] < l[j]) | ((unsigned int)(xs[t] == l[j]) & (unsigned int)(q + t < first + 32 * j));
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (first + 32 * j < len) {
        tk[rank[j]] = ld_cg(keys + first + 32 * j);
        if constexpr (has_payload<P>()) tv[rank[j]] = ld_cg(vals + first + 32 * j);
      }
    }
  }
  __syncwarp();
  for (uint32_t i = lane; i < len; i += 32) {
    keys[i] = ld_cg(tk + i);
    if constexpr (has_payload<P>()) vals[i] = ld_cg(tv + i);
  }
}

// A CTA sorts a longer run by the four lower digits, a tile at a time: ranked
// and staged as in the passes, each digit's run written to where the run's own
// counts and its tiles before put it, to and fro between the array and the
// temporaries.  Bound by latency: a tile's load, ranking and barriers, 4 to 5
// us each.
constexpr int kRsRunItems = 8, kRsRunTile = kRsHistThreads * kRsRunItems;
template <typename K, typename P>
__device__ __forceinline__ void rs_sort_run(K *keys, P *vals, K *tk, P *tv, uint32_t len) {
  constexpr int TH = kRsHistThreads, ITEMS = kRsRunItems, WARPS = TH / 32, WARP_KEYS = 32 * ITEMS;
  constexpr size_t VOFF = sizeof(K) * kRsRunTile;
  static_assert(VOFF + (size_t)payload_bytes<P>() * kRsRunTile <= kRsHistSmemBytes, "the tile fits");
  extern __shared__ __align__(16) unsigned int rs_hist_smem[];
  unsigned char *const smem = reinterpret_cast<unsigned char *>(rs_hist_smem);
  K *const sk = reinterpret_cast<K *>(smem);  // the tile in digit order
  P *const sv = reinterpret_cast<P *>(smem + VOFF);
  __shared__ __align__(16) uint16_t s_whist[WARPS][kRsBins];  // per-warp digit counters, then staging starts (both x4)
  __shared__ unsigned int s_at[4][kRsBins];  // counts of the four digits, then where a digit's next key goes
  __shared__ unsigned int s_dst[kRsBins];    // output position of staged position 0 for digit d
  __shared__ unsigned int s_scan[kRsBins / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the ranking tables lie in the staging area, which is written after every warp has ranked its keys
  unsigned char *const tables = smem + (256u - (smem_addr(smem) & 255u));
  const RsRanker ranker(tables + warp * 512, tables + WARPS * 512 + warp * 128);
  uint4 *const mine = reinterpret_cast<uint4 *>(&s_whist[warp][0]) + lane;  // a warp clears its own counters
  *mine = make_uint4(0u, 0u, 0u, 0u);
  (&s_at[0][0])[tid] = 0u;
  __syncthreads();
  bool down = false;
  for (uint32_t i = tid; i < len; i += TH) {
    const uint32_t l = (uint32_t)RadixKey<K>::to(ld_cg(keys + i));
#pragma unroll
    for (int d = 0; d < 4; ++d) atomicAdd(&s_at[d][(l >> (8 * d)) & 0xffu], 1u);
    if (i > 0) down |= (uint32_t)RadixKey<K>::to(ld_cg(keys + i - 1)) > l;
  }
  if (!__syncthreads_or(down)) return;
  for (int pass = 0; pass < 4; ++pass) {
    const K *const in_k = (pass & 1) ? tk : keys;
    const P *const in_v = (pass & 1) ? tv : vals;
    K *const out_k = (pass & 1) ? keys : tk;
    P *const out_v = (pass & 1) ? vals : tv;
    if (tid < kRsBins) {
      unsigned int all;
      s_at[pass][tid] = rs_scan_digits(s_at[pass][tid], s_scan, all);
    }
    __syncthreads();
    for (uint32_t base = 0; base < len; base += kRsRunTile) {
      const int count = (int)(len - base < (uint32_t)kRsRunTile ? len - base : (uint32_t)kRsRunTile);
      const int warps = (count + WARP_KEYS - 1) / WARP_KEYS;  // that have keys
      auto elem = [&](int j) { return warp * WARP_KEYS + j * 32 + lane; };
      K k[ITEMS];
      P v[ITEMS];
      uint32_t dig4[ITEMS / 4], rank2[ITEMS / 2];
      if (warp < warps) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
          const bool ok = elem(j) < count;
          k[j] = ok ? ld_cg(in_k + base + elem(j)) : K();
          if constexpr (has_payload<P>()) v[j] = ok ? ld_cg(in_v + base + elem(j)) : P();
        }
        // past the run's end the digit is 255: those items stay last
#pragma unroll
        for (int i = 0; i < ITEMS / 4; ++i) dig4[i] = rs_digits4(k + 4 * i, pass);
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
          if (elem(j) >= count) dig4[j >> 2] |= 0xffu << (8 * (j & 3));
        ranker.rank<ITEMS>(s_whist[warp], dig4, rank2);
      }
      __syncthreads();
      if (tid < kRsBins) {
        unsigned int cnt = 0, all;
        for (int w = 0; w < warps; ++w) cnt += s_whist[w][tid];
        const unsigned int excl = rs_scan_digits(cnt, s_scan, all);
        unsigned int run = excl;
        for (int w = 0; w < warps; ++w) {
          const unsigned int c = s_whist[w][tid];
          s_whist[w][tid] = (uint16_t)run;
          run += c;
        }
        cnt >>= 2;
        if (tid == kRsBins - 1) cnt -= (unsigned int)(warps * WARP_KEYS - count);
        const unsigned int at = s_at[pass][tid];
        s_dst[tid] = at - (excl >> 2);
        s_at[pass][tid] = at + cnt;
      }
      __syncthreads();
      if (warp < warps) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
          const uint32_t d = (dig4[j >> 2] >> (8 * (j & 3))) & 0xffu;
          const uint32_t pos = (s_whist[warp][d] + ((rank2[j >> 1] >> (16 * (j & 1))) & 0xffffu)) >> 2;
          sk[pos] = k[j];
          if constexpr (has_payload<P>()) sv[pos] = v[j];
        }
        __syncwarp();
        *mine = make_uint4(0u, 0u, 0u, 0u);
      }
      __syncthreads();
      for (int p = tid; p < count; p += TH) {
        const K key = sk[p];
        const uint32_t to = s_dst[rs_digit1(key, pass)] + (uint32_t)p;
        if (to < len) {
          out_k[to] = key;
          if constexpr (has_payload<P>()) out_v[to] = sv[p];
        }
      }
      __syncthreads();
    }
  }
}

template <typename K, typename P, typename Src, int C>
__global__ void __launch_bounds__(kRsHistThreads, 1) rs_late_kernel(const __grid_constant__ Src src,
                                                                    unsigned int groups, unsigned int *hist,
                                                                    const RsPlanWs *plan, RsRunList list) {
  extern __shared__ __align__(16) unsigned int rs_hist_smem[];
  static_assert((size_t)kRsHistThreads / 32 * kRsRunWarp * 4 <= kRsHistSmemBytes, "a warp's run each");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < (int)(kRsHistSmemBytes / 16); i += kRsHistThreads)
    reinterpret_cast<uint4 *>(rs_hist_smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  grid_dependency_wait();
  const RsGroup<K, P> gr = src.group(0);
  const RsPlan p = rs_plan(plan, gr.n);
  if (p == kPlanRescue) rs_count_digits<K, P, Src, C, 0, 4>(src, groups, hist);
  if (p != kPlanUpper || ld_cg(&plan->unordered) == 0u) return;
  auto upper = [&](uint64_t i) { return (unsigned int)(RadixKey<K>::to(ld_cg(gr.keys + i)) >> 32); };
  const unsigned int longer = ld_cg(&plan->runs[1]), shorter = ld_cg(&plan->runs[0]);
  for (unsigned int r = blockIdx.x; r < longer; r += gridDim.x) {
    const uint64_t start = ld_cg(list.slot(true, r));
    const unsigned int u = upper(start);
    auto in_run = [&](uint32_t q) { return start + q < gr.n && upper(start + q) == u; };
    // its length: whole steps, then the keys of the step that is not
    constexpr uint32_t STEP = kRsRunMax / kRsHistThreads;
    uint32_t len = STEP * (uint32_t)__syncthreads_count(in_run(threadIdx.x * STEP + STEP - 1));
    len += (uint32_t)__syncthreads_count(threadIdx.x < STEP && in_run(len + threadIdx.x));
    rs_sort_run<K, P>(gr.keys + start, has_payload<P>() ? gr.vals + start : nullptr, gr.tk + start,
                      has_payload<P>() ? gr.tv + start : nullptr, len);
    __syncthreads();
  }
  // one warp of each CTA first
  for (unsigned int r = warp * gridDim.x + blockIdx.x; r < shorter; r += gridDim.x * (kRsHistThreads / 32)) {
    const uint64_t start = ld_cg(list.slot(false, r));
    const unsigned int u = upper(start);
    auto in_run = [&](uint32_t q) { return start + q < gr.n && upper(start + q) == u; };
    constexpr uint32_t STEP = kRsRunWarp / 32;
    uint32_t len = STEP * (uint32_t)__popc(__ballot_sync(0xffffffffu, in_run(lane * STEP + STEP - 1)));
    if (len < kRsRunWarp) len += (uint32_t)__popc(__ballot_sync(0xffffffffu, in_run(len + lane)));
    rs_sort_run_warp<K, P>(gr.keys + start, has_payload<P>() ? gr.vals + start : nullptr, gr.tk + start,
                           has_payload<P>() ? gr.tv + start : nullptr, len, rs_hist_smem + warp * kRsRunWarp);
    __syncwarp();
  }
}

// ---- one pass: stable scatter by digit (keys -> temporaries on even passes,
// back on odd ones).
//
// Persistent clusters of C CTAs take groups of C tiles from a ticket.  Every
// CTA ranks its tile's keys by digit and sends its digit counts to the others
// through distributed shared memory, to CTA r those of the digits
// [r * 256 / C, (r + 1) * 256 / C).  Where a group's keys of a digit go
// follows from the groups before it: a group publishes its count of the digit
// (its AGGREGATE) and, once known, the end position (its PREFIX), one 32-bit
// word each: a flag in the two top bits and the value below (n < 2^30).
//
// The look-back reads 16 earlier groups in one round (eight where a group has
// two tiles): kRsWindow words a lane of the scout warp, for its two digits
// (four).  A look-back by single tiles that walks one predecessor a round trip
// does not keep up: a pass runs through 30 tiles of 6656 pairs a microsecond
// (2^26 u32/u32 on a B200), and a round trip takes most of one.  Groups of four
// tiles and rounds of 16 groups do, and a round reads 16 KB for the 208 KB of
// pairs of a group.
//
// A CTA's loop is pipelined by one tile: tile i + 1 is ranked and its counts
// are sent before tile i, staged in shared memory in digit order, is written
// out, so the exchange and the look-back of a tile run while its CTA writes
// the tile before and ranks the one after.  The exchange uses st.async stores
// that complete on the receiver's mbarrier: a cluster barrier's release would
// wait for the tile's scattered global stores.
//
// Waits are bounded.  A look-back that gives up records the error and goes on
// with what it has (all writes are held below the array's length); a CTA
// whose peers do not answer records the error and leaves the loop.
constexpr unsigned int kRsAggregate = 1u << 30, kRsPrefix = 2u << 30, kRsValue = (1u << 30) - 1u;

template <typename K, typename P>
constexpr size_t rs_smem_bytes() {
  return align_up(sizeof(K) * RsCfg<K, P>::TILE, 16) + (size_t)payload_bytes<P>() * RsCfg<K, P>::TILE;
}

// The scout, the CTA's last warp: for every group of its cluster, as soon as
// the cluster's counts of this CTA's digits are in, publishes their sums,
// looks back for where they go and sends every CTA the output positions of
// its tile's keys of those digits.  A lane has DPC / 32 digits.
template <typename Src, int C, typename K, typename P>
__device__ __forceinline__ void rs_scout(const Src &src, int pass, unsigned int groups, unsigned int g,
                                         unsigned int array, const unsigned int *hist, unsigned int *status, unsigned int *status_next,
                                         WsHeader *hdr, unsigned long long limit_ns, const unsigned int *s_x,
                                         unsigned int *s_base, const uint2 *s_next, uint64_t *cnt_bar,
                                         uint64_t *base_bar) {
  constexpr int DPC = kRsBins / C, DPL = DPC / 32;
  constexpr int WINDOW = kRsWindow / DPL;
  const int lane = threadIdx.x & 31;
  const unsigned int me = rs_cluster_rank();
  for (unsigned int it = 0; g < groups; ++it) {
    const uint32_t par = it & 1u, phase = (it >> 1) & 1u;
    if (!rs_wait_cluster(&cnt_bar[par], phase, limit_ns)) {
      if (lane == 0) record_error(hdr, BK_ERR_SPIN_TIMEOUT, g);
      return;
    }
    // Read before any position is sent: the positions let the cluster's first
    // CTA run on to the iteration after next, whose group it hands out in the
    // same place.
    const uint2 next = s_next[par];
    const RsGroup<K, P> gr = src.group(g, array);
    const unsigned int *xs = s_x + par * kRsBins + lane;
    unsigned int *row = status + (uint64_t)g * kRsBins + me * DPC + lane;
    unsigned int x[C][DPL], total[DPL], excl[DPL];
#pragma unroll
    for (int e = 0; e < DPL; ++e) {
      total[e] = 0;
      excl[e] = 0;
#pragma unroll
      for (int q = 0; q < C; ++q) {
        x[q][e] = xs[q * DPC + 32 * e];
        total[e] += x[q][e];
      }
    }
    if (gr.local == 0) {  // the array's first group: positions from the counts of the whole array
      const unsigned int *h = hist + ((uint64_t)gr.array * rs_passes<K>() + pass) * kRsBins;
      unsigned int before = 0;
      for (int d = lane; d < (int)me * DPC; d += 32) before += h[d];
      before = warp_reduce(before, OpSum<unsigned int>());
#pragma unroll
      for (int e = 0; e < DPL; ++e) {
        const unsigned int c = h[me * DPC + 32 * e + lane];
        const unsigned int incl = warp_inclusive_scan(c, OpSum<unsigned int>(), lane);
        excl[e] = before + incl - c;
        before += __shfl_sync(0xffffffffu, incl, 31);
      }
    } else {
#pragma unroll
      for (int e = 0; e < DPL; ++e) st_relaxed_u32(row + 32 * e, kRsAggregate | total[e]);
      bool found[DPL];
#pragma unroll
      for (int e = 0; e < DPL; ++e) found[e] = false;
      unsigned long long t0 = 0;
      unsigned int spins = 0;
      for (int nearest = 1;;) {
        unsigned int w[WINDOW][DPL];
#pragma unroll
        for (int i = 0; i < WINDOW; ++i)
#pragma unroll
          for (int e = 0; e < DPL; ++e)
            w[i][e] = nearest + i <= (int)gr.local ? ld_relaxed_u32(row - (int64_t)(nearest + i) * kRsBins + 32 * e)
                                                   : kRsPrefix;
        // all digits move through the window together: one that meets a
        // missing word makes the warp read the window again from there
        int ready = WINDOW;
#pragma unroll
        for (int i = WINDOW - 1; i >= 0; --i)
#pragma unroll
          for (int e = 0; e < DPL; ++e)
            if (w[i][e] < kRsAggregate) ready = i;
        ready = __reduce_min_sync(0xffffffffu, ready);
        bool open = false;
#pragma unroll
        for (int e = 0; e < DPL; ++e) {
#pragma unroll
          for (int i = 0; i < WINDOW; ++i) {
            if (i < ready && !found[e]) {
              excl[e] += w[i][e] & kRsValue;
              found[e] = w[i][e] >= kRsPrefix;
            }
          }
          open |= !found[e];
        }
        if (!__any_sync(0xffffffffu, open)) break;
        nearest += ready;
        if (ready == 0 && (++spins & 15u) == 0u) {
          const unsigned long long now = globaltimer_ns();
          bool give_up = false;
          if (t0 == 0) t0 = now;
          else give_up = now - t0 > limit_ns || ld_relaxed_s32(&hdr->status) != 0;
          if (__any_sync(0xffffffffu, give_up)) {
            if (lane == 0) record_error(hdr, BK_ERR_SPIN_TIMEOUT, g);
            break;
          }
        }
      }
    }
#pragma unroll
    for (int e = 0; e < DPL; ++e) {
      st_relaxed_u32(row + 32 * e, kRsPrefix | ((excl[e] + total[e]) & kRsValue));
      unsigned int at = excl[e];
#pragma unroll
      for (int q = 0; q < C; ++q) {
        rs_push_u32(s_base + par * kRsBins + me * DPC + 32 * e + lane, at, &base_bar[par], (uint32_t)q);
        at += x[q][e];
      }
      status_next[(uint64_t)g * kRsBins + me * DPC + 32 * e + lane] = 0u;
    }
    g = next.x;
    array = next.y;
  }
}

template <typename K, typename P, typename Src, int C>
__global__ void __launch_bounds__((RsCfg<K, P>::CTA_THREADS), (RsCfg<K, P>::MIN_BLOCKS)) rs_pass_kernel(
    const __grid_constant__ Src src, int launch, const RsPlanWs *plan, unsigned int groups, const unsigned int *hist, unsigned int *tickets,
    unsigned int *status, unsigned int *status_next, WsHeader *hdr, unsigned int ahead, unsigned long long limit_ns) {
  using Cfg = RsCfg<K, P>;
  constexpr int ITEMS = Cfg::ITEMS, WARPS = Cfg::WARPS, THREADS = Cfg::THREADS, TILE = Cfg::TILE;
  constexpr int DPC = kRsBins / C;  // digits whose positions this CTA works out
  constexpr uint32_t GROUP_TX = Src::kMany ? 8 : 4, COUNT_TX = kRsBins * 4 + GROUP_TX, BASE_TX = kRsBins * 4;
  extern __shared__ __align__(16) unsigned char smem[];
  K *sk = reinterpret_cast<K *>(smem);  // the tile in digit order
  P *sv = reinterpret_cast<P *>(smem + align_up(sizeof(K) * TILE, 16));
  __shared__ __align__(16) uint16_t s_whist[2][WARPS][kRsBins];  // per-warp digit counters, then staging starts (x4)
  __shared__ __align__(512) uint32_t s_table[WARPS][4 * 32];
  __shared__ __align__(16) uint32_t s_bits[WARPS][32];
  // what the peers send, by the iteration's parity (a peer may be one iteration ahead):
  __shared__ unsigned int s_x[2][C][DPC];      // the cluster's counts of this CTA's digits
  __shared__ unsigned int s_base[2][kRsBins];  // output position of the tile's first key of a digit
  __shared__ uint2 s_next[2];                  // the next iteration's group and its array
  __shared__ __align__(8) uint64_t s_cnt_bar[2], s_base_bar[2];  // counts and a group, positions are in
  __shared__ unsigned int s_dst[kRsBins];   // output position of staged position 0 for digit d
  __shared__ unsigned int s_scan[kRsBins / 32];
  __shared__ uint2 s_group;                  // the first group
  __shared__ __align__(8) uint64_t s_group_bar;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned int me = rs_cluster_rank();
  const bool odd = launch & 1;
  const RsRanker ranker(s_table[warp], s_bits[warp]);

  // ---- shared memory made ready while the kernel before this one ends
  auto clear_counters = [&](int b) {
    uint4 *z = reinterpret_cast<uint4 *>(&s_whist[b][0][0]);
#pragma unroll
    for (int i = tid; i < WARPS * kRsBins / 8; i += THREADS) z[i] = make_uint4(0u, 0u, 0u, 0u);
  };
  if (tid < THREADS) clear_counters(0);
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&s_cnt_bar[b], 1);
      mbar_init(&s_base_bar[b], 1);
    }
    mbar_init(&s_group_bar, 1);
    rs_fence_mbar_init();
    mbar_arrive_expect_tx(&s_group_bar, GROUP_TX);
    s_group.y = s_next[0].y = s_next[1].y = 0u;
  }
  rs_cluster_sync();  // every CTA of the cluster runs, its barriers ready, before anything is sent to it
  grid_dependency_wait();
  const int pass = rs_launch_digit(launch, plan, plan != nullptr ? src.group(0).n : 0);  // the digit
  if (pass < 0) return;

  auto elem = [&](int j) { return warp * 32 * ITEMS + j * 32 + lane; };
  K k[ITEMS];
  auto load_keys = [&](const RsGroup<K, P> &gr) {
    const uint64_t base = ((uint64_t)gr.local * C + me) * TILE;
    const int count = rs_tile_count(gr, base);
    const K *in = (odd ? gr.tk : (launch == 0 ? gr.src_k : gr.keys)) + base + elem(0);
    if (count == TILE) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) k[j] = in[j * 32];
    } else {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) k[j] = elem(j) < count ? in[j * 32] : K();
    }
  };

  // ---- the first group.  With no more groups than clusters each takes one,
  // whoever starts first.
  const unsigned int clusters = gridDim.x / C;
  const bool more = groups > clusters;
  // the cluster's first warp gives every CTA group t and the array that owns
  // it (found here once, not by every thread that needs it)
  auto hand_out = [&](unsigned int t, uint2 *to, const uint64_t *bar) {
    if (lane < C) {
      rs_push_u32(&to->x, t, bar, (uint32_t)lane);
      if constexpr (Src::kMany) rs_push_u32(&to->y, src.find(t), bar, (uint32_t)lane);
    }
  };
  if (me == 0 && warp == 0) {
    unsigned int t = 0;
    if (lane == 0) t = atomicAdd(&tickets[launch], 1u);
    hand_out(__shfl_sync(0xffffffffu, t, 0), &s_group, &s_group_bar);
  }
  bool failed = !rs_wait_cluster(&s_group_bar, 0, limit_ns);
  failed = __syncthreads_or(failed);
  unsigned int g = failed ? groups : s_group.x, array = s_group.y;
  if (warp == WARPS) {
    rs_scout<Src, C, K, P>(src, pass, groups, g, array, hist, status, status_next, hdr, limit_ns, &s_x[0][0][0], &s_base[0][0],
                           s_next, s_cnt_bar, s_base_bar);
    rs_cluster_sync();
    return;
  }
  if (g < groups) load_keys(src.group(g, array));

  // the tile before this iteration's, staged and waiting for its positions
  unsigned int prev_g = groups, prev_array = 0, prev_excl = 0;
  for (unsigned int it = 0;; ++it) {
    const bool cur = g < groups, prev = prev_g < groups;  // the same in every CTA of the cluster
    if (!cur && !prev) break;
    const uint32_t par = it & 1u, phase = (it >> 1) & 1u;
    uint16_t(*whist)[kRsBins] = s_whist[par];
    const RsGroup<K, P> gr = cur ? src.group(g, array) : src.group(prev_g, prev_array);
    const uint64_t tbase = ((uint64_t)gr.local * C + me) * TILE;
    const int count = rs_tile_count(gr, tbase);
    uint32_t dig4[ITEMS / 4];
    uint32_t rank2[ITEMS / 2];
    unsigned int tile_excl = 0;
    P v[ITEMS];
    if (cur) {
      if (tid == 0) {
        mbar_arrive_expect_tx(&s_cnt_bar[par], COUNT_TX);
        mbar_arrive_expect_tx(&s_base_bar[par], BASE_TX);
      }
      unsigned int ticket = groups;
      if (more && me == 0 && tid == 0) ticket = atomicAdd(&tickets[launch], 1u);
      if (tid == THREADS - 1 && ahead != 0 && g + ahead < groups) {
        // into L2: the tile of a group that a cluster will take about an iteration from now
        const RsGroup<K, P> f = src.group(g + ahead);
        const uint64_t base = ((uint64_t)f.local * C + me) * TILE;
        const uint64_t fc = (uint64_t)rs_tile_count(f, base);
        if (fc > 0) {
          prefetch_l2_range((odd ? f.tk : (launch == 0 ? f.src_k : f.keys)) + base, fc * sizeof(K));
          if constexpr (has_payload<P>())
            prefetch_l2_range((odd ? f.tv : (launch == 0 ? f.src_v : f.vals)) + base, fc * sizeof(P));
        }
      }
      // ---- digits and ranks.  Past the tile's end the digit is 255: those
      // items come after every real one in (warp, item, lane) order, so they
      // rank last in the tile and are never written out.
#pragma unroll
      for (int i = 0; i < ITEMS / 4; ++i) dig4[i] = rs_digits4(k + 4 * i, pass);
      if (count != TILE) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
          if (elem(j) >= count) dig4[j >> 2] |= 0xffu << (8 * (j & 3));
      }
      ranker.rank<ITEMS>(whist[warp], dig4, rank2);
      named_barrier_sync(2, THREADS);

      // ---- thread d: the digit's tile count, and its start in the staged tile for each warp
      if (tid < kRsBins) {
        unsigned int c[WARPS], cnt = 0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
          c[w] = whist[w][tid];
          cnt += c[w];
        }
        unsigned int tile_total;
        tile_excl = rs_scan_digits(cnt, s_scan, tile_total);
        unsigned int run = tile_excl;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
          whist[w][tid] = (uint16_t)run;
          run += c[w];
        }
        cnt >>= 2;
        tile_excl >>= 2;
        if (tid == kRsBins - 1) cnt -= (unsigned int)(TILE - count);
        rs_push_u32(&s_x[par][me][tid % DPC], cnt, &s_cnt_bar[par], (uint32_t)(tid / DPC));
      }
      if (me == 0 && warp == 0) {
        hand_out(__shfl_sync(0xffffffffu, ticket, 0), &s_next[par], &s_cnt_bar[par]);
      }
      // payloads on their way
      if constexpr (has_payload<P>()) {
        const P *in = (odd ? gr.tv : (launch == 0 ? gr.src_v : gr.vals)) + tbase + elem(0);
        if (count == TILE) {
#pragma unroll
          for (int j = 0; j < ITEMS; ++j) v[j] = in[j * 32];
        } else {
#pragma unroll
          for (int j = 0; j < ITEMS; ++j) v[j] = elem(j) < count ? in[j * 32] : P();
        }
      }
    }
    if (prev) {
      if (tid < kRsBins) {
        failed = !rs_wait_cluster(&s_base_bar[par ^ 1u], ((it - 1u) >> 1) & 1u, limit_ns);
        s_dst[tid] = s_base[par ^ 1u][tid] - prev_excl;
      }
    }
    failed = named_barrier_or(2, THREADS, failed);
    if (failed) break;
    if (prev) {
      // ---- the tile before is written out: staged position p goes to s_dst[digit] + p
      const RsGroup<K, P> pg = src.group(prev_g, prev_array);
      const int pcount = rs_tile_count(pg, ((uint64_t)pg.local * C + me) * TILE);
      K *out_k = odd ? pg.keys : pg.tk;
      P *out_v = odd ? pg.vals : pg.tv;
      const uint32_t n = (uint32_t)pg.n;
      auto put = [&](int p) {
        const K key = sk[p];
        // always below n when the counts are consistent
        const uint32_t to = min(s_dst[rs_digit1(key, pass)] + (uint32_t)p, n - 1u);
        out_k[to] = key;
        if constexpr (has_payload<P>()) out_v[to] = sv[p];
      };
      if (pcount == TILE) {
#pragma unroll 4
        for (int i = 0; i < ITEMS; ++i) put(tid + i * THREADS);
      } else {
        for (int p = tid; p < pcount; p += THREADS) put(p);
      }
    }
    if (!cur) break;
    // ---- the other counters ready for the next tile; this one's counts in
    clear_counters((int)(par ^ 1u));
    failed = !rs_wait_cluster(&s_cnt_bar[par], phase, limit_ns);
    failed = named_barrier_or(2, THREADS, failed);
    if (failed) break;

    // ---- stage in digit order
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const uint32_t d = __byte_perm(dig4[j >> 2], 0u, 0x4440u | (uint32_t)(j & 3));
      const uint32_t pos4 = whist[warp][d] + ((j & 1) ? rank2[j >> 1] >> 16 : rank2[j >> 1] & 0xffffu);
      *reinterpret_cast<K *>(reinterpret_cast<unsigned char *>(sk) + pos4 * (sizeof(K) / 4)) = k[j];
      if constexpr (has_payload<P>())
        *reinterpret_cast<P *>(reinterpret_cast<unsigned char *>(sv) + pos4 * (sizeof(P) / 4)) = v[j];
    }
    prev_g = g;
    prev_excl = tile_excl;
    prev_array = array;
    g = s_next[par].x;
    array = s_next[par].y;
    if (g < groups) load_keys(src.group(g, array));
  }
  if (failed && tid == 0) record_error(hdr, BK_ERR_SPIN_TIMEOUT, g);
  rs_cluster_sync();  // nothing is sent to a CTA that has left
}

// ---------------------------------------------------------------------------
// Small arrays (up to 16 tiles): every pass in one launch of one thread-block
// cluster, one CTA per tile.  A pass ranks a tile's keys at the rate of the
// SM's shared-memory pipe (about 31 accesses of a warp for 32 keys), so the
// tile is the smallest that 16 CTAs cover: 1024, 2048 or 4096 keys of 256, 512
// or 1024 threads, then 8192.  The CTAs exchange their digit counts through
// distributed shared memory (each reads every other CTA's 256 counts across
// the cluster) instead of a count scan in global memory, and a cluster barrier
// takes the place of each kernel boundary: two barriers a pass replace the
// launches of the global-memory path.  The keys move
// between passes through the workspace temporaries, which stay in L2 at these
// sizes (storing each key straight into the owning CTA's shared memory was
// measured slower: 42.9 against 32.8 us for 2^16 u32/u32 keys on a B200).
constexpr int kRsClusterMax = 16;  // CTAs (non-portable above 8)

// Shared memory of a cluster-sort CTA of ITEMS items a thread: one tile
// (TH * ITEMS keys and payloads), or the ranking tables that lie in the same place.
template <typename K, typename P, int TH, int ITEMS>
constexpr size_t rs_cluster_smem_bytes() {
  constexpr size_t tile = align_up(sizeof(K) * TH * ITEMS, 16) + (size_t)payload_bytes<P>() * TH * ITEMS;
  constexpr size_t tables = 256 + (size_t)(TH / 32) * (512 + 128);
  return tile > tables ? tile : tables;
}

// The cluster sort: CTA r of the cluster owns tile r.  Each pass reads the
// tile from the pass's input (the array on even passes, the workspace
// temporaries on odd ones; all L2-resident at these sizes), ranks its keys as
// the scatter above does (ITEMS items a thread), exchanges its 256 digit
// counts with the other CTAs through distributed shared memory, stages the
// tile in digit order and writes each digit's run to the pass's output.  The
// cluster barrier after the writes (release / acquire at cluster scope) makes
// them visible to the CTA that reads that tile next.  Even passes end in the
// array, so the last one leaves the result in place.
template <typename K, typename P, int TH, int ITEMS>
__global__ void __launch_bounds__(TH, 1) rs_cluster_kernel(K *keys, P *vals, K *tk, P *tv, uint32_t n) {
  constexpr int WARPS = TH / 32, TILE = TH * ITEMS;
  constexpr size_t VOFF = align_up(sizeof(K) * TILE, 16);
  extern __shared__ __align__(16) unsigned char rs_cl_smem[];
  K *sk = reinterpret_cast<K *>(rs_cl_smem);  // the tile in digit order
  P *sv = reinterpret_cast<P *>(rs_cl_smem + VOFF);
  __shared__ __align__(16) uint16_t s_whist[WARPS][kRsBins];  // per-warp digit counters, then staging starts (both x4)
  __shared__ unsigned int s_cnt[kRsBins];           // this tile's count of each digit (read by the peers)
  __shared__ unsigned int s_dst[kRsBins];           // output position of staged position 0 for digit d
  __shared__ unsigned int s_scan[2 * (kRsBins / 32)];  // the two digit scans' warp totals
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  grid_dependency_wait();
  const uint32_t me = rs_cluster_rank(), csize = rs_cluster_size();
  const uint32_t base = me * (uint32_t)TILE;
  const int count = (int)((n - base) < (uint32_t)TILE ? (n - base) : (uint32_t)TILE);
  for (int i = tid; i < WARPS * kRsBins / 8; i += TH)
    reinterpret_cast<uint4 *>(&s_whist[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  // the ranking tables lie in the staging area, which is written after every warp has ranked its keys
  unsigned char *tables = rs_cl_smem + (256u - (smem_addr(rs_cl_smem) & 255u));
  const RsRanker ranker(tables + warp * 512, tables + WARPS * 512 + warp * 128);
  for (int pass = 0; pass < rs_passes<K>(); ++pass) {
    const int shift = 8 * pass;
    const K *in_k = (pass & 1) ? tk : keys;
    const P *in_v = (pass & 1) ? tv : vals;
    K *out_k = (pass & 1) ? keys : tk;
    P *out_v = (pass & 1) ? vals : tv;
    K k[ITEMS];
    P v[ITEMS];
    auto elem = [&](int j) { return warp * 32 * ITEMS + j * 32 + lane; };
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const bool ok = elem(j) < count;
      k[j] = ok ? ld_cg(in_k + base + elem(j)) : K();
      if constexpr (has_payload<P>()) v[j] = ok ? ld_cg(in_v + base + elem(j)) : P();
    }
    uint32_t dig4[ITEMS / 4];
#pragma unroll
    for (int i = 0; i < ITEMS / 4; ++i) dig4[i] = rs_digits4(k + 4 * i, pass);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
      if (elem(j) >= count) dig4[j >> 2] |= 0xffu << (8 * (j & 3));
    auto digit_of = [&](int j) { return (int)((dig4[j >> 2] >> (8 * (j & 3))) & 0xffu); };
    uint32_t rank2[ITEMS / 2];
    ranker.rank<ITEMS>(s_whist[warp], dig4, rank2);
    __syncthreads();
    const int d = tid;
    unsigned int tile_excl = 0;
    if (d < kRsBins) {
      unsigned int cnt = 0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) cnt += s_whist[w][d];
      unsigned int tile_total;
      tile_excl = rs_scan_digits(cnt, s_scan, tile_total);
      unsigned int run = tile_excl;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const unsigned int c = s_whist[w][d];
        s_whist[w][d] = (uint16_t)run;
        run += c;
      }
      tile_excl >>= 2;
      cnt >>= 2;
      s_cnt[d] = d == kRsBins - 1 ? cnt - (unsigned int)(TILE - count) : cnt;
    }
    rs_cluster_sync();
    if (d < kRsBins) {
      unsigned int c[kRsClusterMax];
#pragma unroll
      for (int q = 0; q < kRsClusterMax; ++q)
        c[q] = (uint32_t)q < csize ? rs_peer_ld_u32(rs_peer_addr(&s_cnt[d], (uint32_t)q)) : 0u;
      unsigned int before = 0, total = 0;
#pragma unroll
      for (int q = 0; q < kRsClusterMax; ++q) {
        total += c[q];
        if ((uint32_t)q < me) before += c[q];
      }
      unsigned int all;
      const unsigned int start = rs_scan_digits(total, s_scan + kRsBins / 32, all);
      s_dst[d] = start + before - tile_excl;
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int dj = digit_of(j);
      const unsigned int pos = (s_whist[warp][dj] + ((rank2[j >> 1] >> (16 * (j & 1))) & 0xffffu)) >> 2;
      sk[pos] = k[j];
      if constexpr (has_payload<P>()) sv[pos] = v[j];
    }
    __syncthreads();
    for (int i = tid; i < WARPS * kRsBins / 8; i += TH)
    reinterpret_cast<uint4 *>(&s_whist[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int p = tid; p < count; p += TH) {
      const K key = sk[p];
      const uint32_t g = s_dst[rs_digit(key, shift)] + (uint32_t)p;
      if (g < n) {
        out_k[g] = key;
        if constexpr (has_payload<P>()) out_v[g] = sv[p];
      }
    }
    rs_cluster_sync();
  }
}

// Once per device: the largest cluster (16 or 8 CTAs, 0 for none) that the
// cluster sort can be launched with, for tiles of TH * ITEMS keys.
template <typename K, typename P, int TH, int ITEMS>
int rs_cluster_setup(int *max_ctas) {
  struct Site {};
  return host::once_per_device<Site>(max_ctas, [](int *mx) -> int {
    auto kern = rs_cluster_kernel<K, P, TH, ITEMS>;
    constexpr size_t smem = rs_cluster_smem_bytes<K, P, TH, ITEMS>();
    int st;
    if ((st = host::set_smem_attrs(kern, smem)) != BK_OK) return st;
    *mx = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
      (void)cudaGetLastError();
    for (int c : {kRsClusterMax, 8}) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)c);
      cfg.blockDim = dim3(TH);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)c;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        continue;
      }
      if (clusters > 0) {
        *mx = c;
        break;
      }
    }
    return BK_OK;
  });
}

// The cluster sort of n elements (n <= TH * ITEMS * max_ctas), one launch;
// tk / tv are the workspace temporaries of n elements.
template <typename K, typename P, int TH, int ITEMS>
int rs_cluster_launch(K *keys, P *vals, K *tk, P *tv, uint64_t n, cudaStream_t stream) {
  constexpr uint64_t TILE = (uint64_t)TH * ITEMS;
  const unsigned c = (unsigned)((n + TILE - 1) / TILE);
  return host::launch_overlapped(rs_cluster_kernel<K, P, TH, ITEMS>, c, TH, rs_cluster_smem_bytes<K, P, TH, ITEMS>(),
                                 stream, c, keys, vals, tk, tv, (uint32_t)n);
}

// CTAs a group: four (eight leave up to an eighth of the SMs' room for CTAs
// unused, since a cluster lies within one GPC: 4 % slower at 2^26 keys), or
// two for a batch whose arrays would leave more than a quarter of the larger
// groups' tiles empty.
constexpr int kRsCtas = 4, kRsCtasSmall = 2;
template <typename K, typename P>
inline int rs_group_ctas(const uint64_t *sizes, uint32_t count) {
  constexpr uint64_t T = RsCfg<K, P>::TILE;
  uint64_t tiles = 0, padded = 0;
  for (uint32_t i = 0; i < count; ++i) {
    const uint64_t t = (sizes[i] + T - 1) / T;
    tiles += t;
    padded += align_up(t, kRsCtas);
  }
  return count == 1 || padded <= tiles + tiles / 4 ? kRsCtas : kRsCtasSmall;
}

// Workspace (after the 256-byte header): every array's key and payload
// temporaries; zeroed before each sort: the arrays' digit counts, the passes'
// tickets and a planned sort's decision and sample; two buffers of status rows
// (one word a digit and group), of which each pass publishes in one and clears
// the other.
template <typename K, typename P>
struct RsLayout {
  size_t tmp, hist, tickets, plan, samples, zero_bytes, status[2], total;
  uint64_t groups;
  int ctas;
  RsLayout(const uint64_t *sizes, uint32_t count) {
    size_t o = kHeaderBytes;
    tmp = o;
    groups = 0;
    ctas = rs_group_ctas<K, P>(sizes, count);
    const uint64_t span = (uint64_t)ctas * RsCfg<K, P>::TILE;
    for (uint32_t i = 0; i < count; ++i) {
      o += align_up(sizes[i] * sizeof(K), 256) + align_up(sizes[i] * (size_t)payload_bytes<P>(), 256);
      groups += (sizes[i] + span - 1) / span;
    }
    hist = o;
    o += (size_t)count * rs_passes<K>() * kRsBins * 4;
    tickets = o;
    plan = o + 128;
    o += 256;
    samples = o;
    if (sizeof(K) == 8 && count == 1 && sizes[0] >= kRsPlanMinN) o += (size_t)kRsSampleSlots * 4;
    zero_bytes = o - hist;
    for (size_t &s : status) {
      s = o;
      o += (size_t)groups * kRsBins * 4;
    }
    total = o;
  }
};

template <typename K, typename P>
size_t radix_sort_ws_bytes(uint64_t n) {
  return RsLayout<K, P>(&n, 1).total;
}

template <typename K, typename P>
size_t radix_sort_batch_ws_bytes(const uint64_t *sizes, uint32_t count) {
  uint64_t sz[kRsBatchMax];
  uint32_t m = 0;
  for (uint32_t i = 0; i < count && m < (uint32_t)kRsBatchMax; ++i)
    if (sizes[i] > 1) sz[m++] = sizes[i];  // arrays of 0 or 1 element need nothing
  return RsLayout<K, P>(sz, m).total;
}

// The passes over `src` (one array or a batch).
template <typename K, typename P, typename Src, int C>
int radix_sort_run(const Src &src, const RsLayout<K, P> &L, char *ws, cudaStream_t stream) {
  // one array of 8-byte keys: see RsPlanWs
  constexpr bool kPlanned = sizeof(K) == 8 && std::is_same<Src, RsOne<K, P>>::value;
  int st;
  auto hist_kern = rs_hist_kernel<K, P, Src, C>;
  auto pass_kern = rs_pass_kernel<K, P, Src, C>;
  struct HistSite {};
  struct PassSite {};
  host::KernelSetup hs;
  if ((st = host::kernel_setup<HistSite>(hist_kern, kRsHistThreads, kRsHistSmemBytes, &hs)) != BK_OK) return st;
  int clusters = 0;  // resident at once
  st = host::once_per_device<PassSite>(&clusters, [&](int *out) -> int {
    int e = host::set_smem_attrs(pass_kern, rs_smem_bytes<K, P>());
    if (e != BK_OK) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(RsCfg<K, P>::CTA_THREADS);
    cfg.dynamicSmemBytes = rs_smem_bytes<K, P>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if ((e = host::from_cuda(cudaOccupancyMaxActiveClusters(out, pass_kern, &cfg))) != BK_OK) {
      (void)cudaGetLastError();
      return e;
    }
    return *out > 0 ? BK_OK : BK_ERR_UNSUPPORTED;
  });
  if (st != BK_OK) return st;
  auto *hist = reinterpret_cast<unsigned int *>(ws + L.hist);
  auto *tickets = reinterpret_cast<unsigned int *>(ws + L.tickets);
  auto *hdr = reinterpret_cast<WsHeader *>(ws);
  const unsigned groups = (unsigned)L.groups;
  const host::DebugFault df = host::debug_fault();
  const unsigned long long limit = df.spin_limit_ns ? df.spin_limit_ns : host::kDefaultSpinLimitNs;
  const uint32_t zero_vecs = (uint32_t)(L.zero_bytes / 16);
  const unsigned zero_ctas = (zero_vecs + 1023) / 1024;
  if ((st = host::launch_overlapped(rs_zero_kernel, zero_ctas, 256, 0, stream, 1, reinterpret_cast<uint4 *>(hist),
                                    zero_vecs)) != BK_OK)
    return st;
  RsPlanWs *plan = nullptr;
  unsigned fix_ctas = 0, late_ctas = 0;
  if constexpr (kPlanned) {
    if (src.n >= kRsPlanMinN) {
      plan = reinterpret_cast<RsPlanWs *>(ws + L.plan);
      struct FixSite {};
      host::KernelSetup fs;
      if ((st = host::kernel_setup<FixSite>(rs_fix_kernel<K, P>, kRsFixThreads, 0, &fs)) != BK_OK) return st;
      fix_ctas = (unsigned)fs.resident_ctas;
      struct LateSite {};
      if ((st = host::kernel_setup<LateSite>(rs_late_kernel<K, P, Src, C>, kRsHistThreads, kRsHistSmemBytes, &fs)) != BK_OK)
        return st;
      late_ctas = (unsigned)fs.resident_ctas;
      st = host::launch_overlapped(rs_sample_kernel<K>, kRsSampleCtas, kRsSampleThreads, 0, stream, 1,
                                   (const K *)src.keys, (uint32_t)src.n,
                                   reinterpret_cast<unsigned int *>(ws + L.samples), plan);
      if (st != BK_OK) return st;
    }
  }
  const uint64_t tiles = L.groups * C;
  const unsigned hist_ctas = (unsigned)(tiles < hs.resident_ctas ? tiles : hs.resident_ctas);
  st = host::launch_overlapped(hist_kern, hist_ctas, kRsHistThreads, kRsHistSmemBytes, stream, 1, src, groups, hist,
                               reinterpret_cast<uint4 *>(ws + L.status[0]), (const RsPlanWs *)plan);
  if (st != BK_OK) return st;
  const unsigned used = groups < (unsigned)clusters ? groups : (unsigned)clusters;
  // L2 prefetch distance: the table's number of rounds of all clusters ahead (0: none)
  const tune::Knobs kn = tune::knobs_for(tune::kSort, RsCfg<K, P>::BYTES, L.groups * C * RsCfg<K, P>::TILE);
  const unsigned ahead = used * (unsigned)kn.prefetch;
  const int launches = plan != nullptr ? 12 : rs_passes<K>();
  for (int p = 0; p < launches; ++p) {
    st = host::launch_overlapped(pass_kern, used * C, RsCfg<K, P>::CTA_THREADS, rs_smem_bytes<K, P>(), stream, C, src, p,
                                 (const RsPlanWs *)plan, groups, (const unsigned int *)hist, tickets,
                                 reinterpret_cast<unsigned int *>(ws + L.status[p & 1]),
                                 reinterpret_cast<unsigned int *>(ws + L.status[(p & 1) ^ 1]), hdr, ahead, limit);
    if (st != BK_OK) return st;
    if constexpr (kPlanned) {
      if (plan != nullptr && p == 3) {
        // the rows that launch 3 published in and launch 4 clears
        const RsRunList list{reinterpret_cast<unsigned int *>(ws + L.status[1]), groups * (unsigned)kRsBins};
        st = host::launch_overlapped(rs_fix_kernel<K, P>, fix_ctas, kRsFixThreads, 0, stream, 1, src.keys, src.vals,
                                     (uint32_t)src.n, plan, list);
        if (st != BK_OK) return st;
        st = host::launch_overlapped(rs_late_kernel<K, P, Src, C>, late_ctas, kRsHistThreads, kRsHistSmemBytes, stream, 1,
                                     src, groups, hist, (const RsPlanWs *)plan, list);
        if (st != BK_OK) return st;
      }
    }
  }
  return BK_OK;
}

constexpr int kNoCluster = 1 << 30;  // no status

template <typename K, typename P>
int radix_sort_launch(K *keys, P *vals, uint64_t n, void *d_ws, size_t ws_bytes, cudaStream_t stream) {
  host::DeviceInfo di;
  int st = host::device_info(&di);
  if (st != BK_OK) return st;
  if (n <= 1) return BK_OK;
  if (keys == nullptr || (has_payload<P>() && vals == nullptr)) return BK_ERR_INVALID_ARGUMENT;
  if (!host::aligned_to<K>(keys)) return BK_ERR_MISALIGNED;
  if constexpr (has_payload<P>()) {
    if (!host::aligned_to<P>(vals)) return BK_ERR_MISALIGNED;
  }
  if (n >= kRsMaxN) return BK_ERR_TOO_LARGE;  // the caller sorts these by merging
  const RsLayout<K, P> L(&n, 1);
  if ((st = host::check_ws(d_ws, ws_bytes, L.hist)) != BK_OK) return st;  // the temporaries: all a cluster needs
  char *ws = reinterpret_cast<char *>(d_ws);
  K *tk = reinterpret_cast<K *>(ws + L.tmp);
  P *tv = reinterpret_cast<P *>(ws + L.tmp + align_up(n * sizeof(K), 256));
  auto cluster = [&](auto th, auto items) -> int {  // the sort's status, or kNoCluster when n needs more CTAs
    constexpr int TH = decltype(th)::value, ITEMS = decltype(items)::value;
    int ctas = 0;
    const int e = rs_cluster_setup<K, P, TH, ITEMS>(&ctas);
    if (e != BK_OK) return e;
    if (n > (uint64_t)TH * ITEMS * (uint64_t)ctas) return kNoCluster;
    return rs_cluster_launch<K, P, TH, ITEMS>(keys, vals, tk, tv, n, stream);
  };
  using std::integral_constant;
  if ((st = cluster(integral_constant<int, 256>(), integral_constant<int, 4>())) != kNoCluster) return st;
  if ((st = cluster(integral_constant<int, 512>(), integral_constant<int, 4>())) != kNoCluster) return st;
  if ((st = cluster(integral_constant<int, 1024>(), integral_constant<int, 4>())) != kNoCluster) return st;
  if ((st = cluster(integral_constant<int, 1024>(), integral_constant<int, 8>())) != kNoCluster) return st;
  if ((st = host::check_ws(d_ws, ws_bytes, L.total)) != BK_OK) return st;
  return radix_sort_run<K, P, RsOne<K, P>, kRsCtas>(RsOne<K, P>{keys, vals, tk, tv, n}, L, ws, stream);
}

// A batch item: sort in_keys / in_vals (left unchanged) into keys / vals;
// in place when they are the same arrays.
template <typename K, typename P>
struct RsItem {
  const K *in_keys;
  const P *in_vals;
  K *keys;
  P *vals;
  uint64_t n;
};

// ---------------------------------------------------------------------------
// Arrays of up to kRsBlockMax keys: one CTA each, every pass in shared memory.
// The keys and payloads go round through the staging area (ranked as above,
// stored in digit order, read back); three barriers a pass.  Bound by the
// SM's shared-memory pipe, as the cluster sort is, but with nothing exchanged,
// and a CTA sees all keys: passes whose digit is the same in every key are
// left out, and 8-byte keys whose upper halves mostly differ are sorted by
// their upper digits, then their short runs of equal upper halves are put in
// order in place (by counting, as rs_fix_kernel does).  The keys are counted
// by a hash of their upper half first, which bounds the runs: a slot holds at
// least the run's keys, and the sum of the slots' squares at least the
// comparisons.  (A guess from a sample of the keys met runs of hundreds: 4096
// u64/u32 keys of which 70 agree took 52 us.)  Runs of up to 64 keys, six on
// average, cost less than the four lower passes (4096 u64/u32 of 1000 upper
// halves 20.2 us, by all digits 21.5; of 70 equal ones 28 against 22).
// 512 threads of eight keys where 1024 of four left each 64 registers and 32
// warps' counters to sum (u64/u32 4096 random 15.7 us, now 14.1; all digits
// 24.0, now 21.0).  On a B200, with the block sort by merging before: u32/u32
// 1024 keys 5.0 us (22.7), 4096 11.0 (24.7); u64/u32 1024 6.3 (18.6), 4096
// 14.1 (20.9; 22.1 where more than 64 keys share an upper half and all digits
// occur).
// ---------------------------------------------------------------------------
constexpr int kRsBlockMax = 4096;
constexpr unsigned int kRsBlockRun = 64, kRsBlockRunMean = 6;

template <typename K, typename P, int N>
struct RsBlockItems {
  const K *in_k[N];
  const P *in_v[N];
  K *out_k[N];
  P *out_v[N];
  uint32_t n[N];
};

template <typename K, typename P, int TH, int ITEMS>
constexpr size_t rs_block_smem_bytes() {
  constexpr size_t tile = (size_t)TH * ITEMS;
  return 256 + (size_t)(TH / 32) * (512 + 128) + align_up(sizeof(K) * tile, 16) + (size_t)payload_bytes<P>() * tile;
}

template <typename K, typename P, int TH, int ITEMS, int N>
__global__ void __launch_bounds__(TH, 1) rs_block_kernel(const __grid_constant__ RsBlockItems<K, P, N> items) {
  constexpr int WARPS = TH / 32, TILE = TH * ITEMS;
  extern __shared__ __align__(16) unsigned char rs_bl_smem[];
  __shared__ __align__(16) uint16_t s_whist[WARPS][kRsBins];  // per-warp digit counters, then staging starts (both x4)
  __shared__ unsigned int s_scan[kRsBins / 32];
  __shared__ unsigned int s_vary[2];  // bits that differ between keys: lower and upper halves
  __shared__ unsigned int s_run[2];   // the most keys in a slot, and the sum of the slots' squares
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char *tables = rs_bl_smem + (256u - (smem_addr(rs_bl_smem) & 255u));
  unsigned char *bits = tables + WARPS * 512;
  K *sk = reinterpret_cast<K *>(bits + WARPS * 128);
  P *sv = reinterpret_cast<P *>(reinterpret_cast<unsigned char *>(sk) + align_up(sizeof(K) * TILE, 16));
  const RsRanker ranker(tables + warp * 512, bits + warp * 128);
  uint4 *const mine = reinterpret_cast<uint4 *>(&s_whist[warp][0]) + lane;  // a warp clears its own counters
  *mine = make_uint4(0u, 0u, 0u, 0u);
  // 8-byte keys are counted by a hash of their upper half, in the staging area
  unsigned int *const slots = reinterpret_cast<unsigned int *>(sk);
  if constexpr (sizeof(K) == 8) {
#pragma unroll
    for (int j = 0; j < ITEMS / 2; ++j) reinterpret_cast<uint4 *>(slots)[j * TH + tid] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (tid < 2) s_vary[tid] = s_run[tid] = 0u;
  __syncthreads();
  grid_dependency_wait();
  const K *in_k = items.in_k[blockIdx.x];
  const P *in_v = items.in_v[blockIdx.x];
  const int count = (int)items.n[blockIdx.x];
  auto elem = [&](int j) { return warp * 32 * ITEMS + j * 32 + lane; };
  auto slot_of = [&](K key) {
    return slots + ((unsigned int)rs_word(RadixKey<K>::to(key), 4) * 0x9e3779b1u) / (0x80000000u / (unsigned int)TILE);
  };
  K k[ITEMS];
  P v[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    k[j] = elem(j) < count ? in_k[elem(j)] : K();
    if constexpr (has_payload<P>()) v[j] = elem(j) < count ? in_v[elem(j)] : P();
  }
  // the digits that differ between keys
  unsigned int todo;
  {
    const auto first = RadixKey<K>::to(in_k[0]);
    typename RadixKey<K>::U x = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (elem(j) < count) {
        x |= RadixKey<K>::to(k[j]) ^ first;
        if constexpr (sizeof(K) == 8) atomicAdd(slot_of(k[j]), 1u);
      }
    }
#pragma unroll
    for (int h = 0; h < (int)sizeof(K) / 4; ++h) {
      const unsigned int o = __reduce_or_sync(0xffffffffu, rs_word(x, 4 * h));
      if (lane == 0 && o != 0u) atomicOr(&s_vary[h], o);
    }
    __syncthreads();
    auto digits = [](unsigned int w) {
      return (w & 0xffu ? 1u : 0u) | (w & 0xff00u ? 2u : 0u) | (w & 0xff0000u ? 4u : 0u) | (w & 0xff000000u ? 8u : 0u);
    };
    todo = digits(s_vary[0]);
    if constexpr (sizeof(K) == 8) todo |= digits(s_vary[1]) << 4;
  }
  bool upper = false;  // the upper digits alone, then the runs that agree there
  if constexpr (sizeof(K) == 8) {
    unsigned int most = 0, sum = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (elem(j) < count) {
        const unsigned int c = *slot_of(k[j]);
        most = c > most ? c : most;
        sum += c;
      }
    }
    most = __reduce_max_sync(0xffffffffu, most);
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) {
      atomicMax(&s_run[0], most);
      atomicAdd(&s_run[1], sum);
    }
    __syncthreads();
    upper = (todo >> 4) != 0u && (todo & 15u) != 0u && s_run[0] <= kRsBlockRun &&
            s_run[1] <= kRsBlockRunMean * (unsigned int)count;
  }
  if (upper) todo &= 0xf0u;
  while (todo != 0u) {
    const int pass = __ffs(todo) - 1;
    todo &= todo - 1u;
    // past the array's end the digit is 255: those items stay last
    uint32_t dig4[ITEMS / 4];
#pragma unroll
    for (int i = 0; i < ITEMS / 4; ++i) dig4[i] = rs_digits4(k + 4 * i, pass);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
      if (elem(j) >= count) dig4[j >> 2] |= 0xffu << (8 * (j & 3));
    uint32_t rank2[ITEMS / 2];
    ranker.rank<ITEMS>(s_whist[warp], dig4, rank2);
    __syncthreads();
    if (tid < kRsBins) {
      unsigned int c[WARPS], cnt = 0, total;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        c[w] = s_whist[w][tid];
        cnt += c[w];
      }
      unsigned int run = rs_scan_digits(cnt, s_scan, total);
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        s_whist[w][tid] = (uint16_t)run;
        run += c[w];
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const uint32_t d = (dig4[j >> 2] >> (8 * (j & 3))) & 0xffu;
      const uint32_t pos = (s_whist[warp][d] + ((rank2[j >> 1] >> (16 * (j & 1))) & 0xffffu)) >> 2;
      sk[pos] = k[j];
      if constexpr (has_payload<P>()) sv[pos] = v[j];
    }
    __syncwarp();
    *mine = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      k[j] = sk[elem(j)];
      if constexpr (has_payload<P>()) v[j] = sv[elem(j)];
    }
    if constexpr (sizeof(K) == 8) {
      if (upper && todo == 0u) {
        int to[ITEMS];
        bool move = false;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
          const int i = elem(j);
          to[j] = -1;
          if (i >= count) continue;
          const uint64_t u = RadixKey<K>::to(k[j]);
          auto same = [&](int q) { return (unsigned int)((RadixKey<K>::to(sk[q]) ^ u) >> 32) == 0u; };
          int first = i, rank = 0;
          for (; first > 0 && same(first - 1); --first) rank += RadixKey<K>::to(sk[first - 1]) <= u;
          for (int q = i + 1; q < count && same(q); ++q) rank += RadixKey<K>::to(sk[q]) < u;
          if (first + rank != i) {
            to[j] = first + rank;
            move = true;
          }
        }
        if (__syncthreads_or(move)) {
#pragma unroll
          for (int j = 0; j < ITEMS; ++j) {
            if (to[j] >= 0) {
              sk[to[j]] = k[j];
              if constexpr (has_payload<P>()) sv[to[j]] = v[j];
            }
          }
          __syncthreads();
#pragma unroll
          for (int j = 0; j < ITEMS; ++j) {
            k[j] = sk[elem(j)];
            if constexpr (has_payload<P>()) v[j] = sv[elem(j)];
          }
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    if (elem(j) < count) {
      items.out_k[blockIdx.x][elem(j)] = k[j];
      if constexpr (has_payload<P>()) items.out_v[blockIdx.x][elem(j)] = v[j];
    }
  }
}

template <typename K, typename P, int TH, int ITEMS, int N>
int rs_block_run(const RsBlockItems<K, P, N> &items, uint32_t count, cudaStream_t stream) {
  struct Site {};
  host::KernelSetup ks;
  constexpr size_t smem = rs_block_smem_bytes<K, P, TH, ITEMS>();
  const int st = host::kernel_setup<Site>(rs_block_kernel<K, P, TH, ITEMS, N>, TH, smem, &ks);
  if (st != BK_OK) return st;
  return host::launch_overlapped(rs_block_kernel<K, P, TH, ITEMS, N>, count, TH, smem, stream, 1, items);
}

// `count` arrays of 1 to kRsBlockMax keys each, checked by the caller.
template <typename K, typename P>
int radix_sort_blocks(const RsItem<K, P> *items, uint32_t count, cudaStream_t stream) {
  auto run = [&](auto cap) {
    RsBlockItems<K, P, decltype(cap)::value> b;
    uint64_t longest = 0;
    uint32_t m = 0;
    for (uint32_t i = 0; i < count; ++i) {
      if (items[i].n == 0) continue;
      b.in_k[m] = items[i].in_keys;
      b.in_v[m] = items[i].in_vals;
      b.out_k[m] = items[i].keys;
      b.out_v[m] = items[i].vals;
      b.n[m++] = (uint32_t)items[i].n;
      longest = items[i].n > longest ? items[i].n : longest;
    }
    if (m == 0) return (int)BK_OK;
    return longest <= 1024   ? rs_block_run<K, P, 256, 4, decltype(cap)::value>(b, m, stream)
           : longest <= 2048 ? rs_block_run<K, P, 512, 4, decltype(cap)::value>(b, m, stream)
                             : rs_block_run<K, P, 512, 8, decltype(cap)::value>(b, m, stream);
  };
  return count == 1 ? run(std::integral_constant<int, 1>()) : run(std::integral_constant<int, kRsBatchMax>());
}

template <typename K, typename P>
int radix_sort_batch_launch(const RsItem<K, P> *items, uint32_t count, void *d_ws, size_t ws_bytes,
                            cudaStream_t stream) {
  if (count > 0 && items == nullptr) return BK_ERR_INVALID_ARGUMENT;
  if (count > (uint32_t)kRsBatchMax) return BK_ERR_TOO_LARGE;
  host::DeviceInfo di;
  int st = host::device_info(&di);
  if (st != BK_OK) return st;
  uint64_t sz[kRsBatchMax];
  uint32_t m = 0;
  for (uint32_t i = 0; i < count; ++i) {
    const RsItem<K, P> &it = items[i];
    if (it.n > 0 && (it.keys == nullptr || it.in_keys == nullptr ||
                     (has_payload<P>() && (it.vals == nullptr || it.in_vals == nullptr))))
      return BK_ERR_INVALID_ARGUMENT;
    if (!host::aligned_to<K>(it.keys) || !host::aligned_to<K>(it.in_keys)) return BK_ERR_MISALIGNED;
    if constexpr (has_payload<P>()) {
      if (!host::aligned_to<P>(it.vals) || !host::aligned_to<P>(it.in_vals)) return BK_ERR_MISALIGNED;
    }
    if (it.n == 1 && it.in_keys != it.keys) {  // a single element out of place: copied, not sorted
      if ((st = host::from_cuda(cudaMemcpyAsync(it.keys, it.in_keys, sizeof(K), cudaMemcpyDeviceToDevice,
                                                stream))) != BK_OK)
        return st;
      if constexpr (has_payload<P>()) {
        if ((st = host::from_cuda(cudaMemcpyAsync(it.vals, it.in_vals, sizeof(P), cudaMemcpyDeviceToDevice,
                                                  stream))) != BK_OK)
          return st;
      }
    }
    if (it.n >= kRsMaxN) return BK_ERR_TOO_LARGE;
    if (it.n > 1) sz[m++] = it.n;
  }
  if (m == 0) return BK_OK;
  const RsLayout<K, P> L(sz, m);
  if (L.groups >= 0x1fffffffull) return BK_ERR_TOO_LARGE;
  if ((st = host::check_ws(d_ws, ws_bytes, L.total)) != BK_OK) return st;
  char *ws = reinterpret_cast<char *>(d_ws);
  RsBatch<K, P> b;
  b.count = 0;
  size_t off = L.tmp;
  const uint64_t span = (uint64_t)L.ctas * RsCfg<K, P>::TILE;
  uint64_t groups = 0;
  for (uint32_t i = 0; i < count; ++i) {
    const RsItem<K, P> &it = items[i];
    if (it.n <= 1) continue;
    const uint32_t k = b.count++;
    b.keys[k] = it.keys;
    b.vals[k] = it.vals;
    b.src_k[k] = it.in_keys;
    b.src_v[k] = it.in_vals;
    b.tk[k] = reinterpret_cast<K *>(ws + off);
    off += align_up(it.n * sizeof(K), 256);
    b.tv[k] = reinterpret_cast<P *>(ws + off);
    off += align_up(it.n * (size_t)payload_bytes<P>(), 256);
    b.n[k] = it.n;
    b.start[k] = (uint32_t)groups;
    groups += (it.n + span - 1) / span;
  }
  b.start[b.count] = (uint32_t)groups;
  return L.ctas == kRsCtas ? radix_sort_run<K, P, RsBatch<K, P>, kRsCtas>(b, L, ws, stream)
                           : radix_sort_run<K, P, RsBatch<K, P>, kRsCtasSmall>(b, L, ws, stream);
}

// explicit instantiations used by sort.cu
#define BK_RS_INST_P(K, P)                                                                                  \
  template int radix_sort_launch<K, P>(K *, P *, uint64_t, void *, size_t, cudaStream_t);                  \
  template size_t radix_sort_ws_bytes<K, P>(uint64_t);                                                      \
  template int radix_sort_blocks<K, P>(const RsItem<K, P> *, uint32_t, cudaStream_t);                       \
  template int radix_sort_batch_launch<K, P>(const RsItem<K, P> *, uint32_t, void *, size_t, cudaStream_t); \
  template size_t radix_sort_batch_ws_bytes<K, P>(const uint64_t *, uint32_t);
#define BK_RS_INST(K)        \
  BK_RS_INST_P(K, NoPayload) \
  BK_RS_INST_P(K, uint32_t)  \
  BK_RS_INST_P(K, unsigned long long)
BK_RS_INST(int32_t)
BK_RS_INST(uint32_t)
BK_RS_INST(int64_t)
BK_RS_INST(uint64_t)
BK_RS_INST(float)
BK_RS_INST(double)

}  // namespace bk
