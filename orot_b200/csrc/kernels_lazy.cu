// kernels_lazy.cu -- LZ77 with hash chains and lazy evaluation (levels 4-12)
// and dynamic Huffman blocks, on sm_100a.
//
// Search semantics follow the reference's standard path
// (src/deflate/lz77.cpp:66-156, 435-495): chains of earlier positions with the
// same 16-bit hash, newest first; up to max_chain members examined, a 4-byte
// mismatch counts as a miss and miss_limit consecutive misses end the walk,
// the longest match wins (ties keep the nearest), nice_len ends the walk;
// the lazy step moves to pos+1 when the match there is two bytes longer.
// GPU-native differences, all keeping the stream valid:
//   * a chain ends at the 32 KiB window edge (the reference keeps walking
//     with distances taken mod 32768);
//   * every position is searched once with the full chain, and the lazy
//     step uses that match (the reference searches pos+1 again with half the
//     chain, skipping the candidate at distance 1);
//   * the input is cut into independent 4 KiB tiles (16 x 258 bytes): each
//     tile parses from its own first byte and matches do not run past its
//     end, while still referencing up to 32 KiB before the tile;
//   * levels 10-12 use the same chains with 1024/2048/4096 steps instead of
//     the reference's binary tree, and an optimal parse: costs from the
//     histogram of a lazy parse, then a backward pass over the tile picks the
//     cheapest literal / match (the found match shortened by up to 31 bytes)
//     at every position;
//   * code lengths come from an optimal two-queue Huffman construction with
//     the ITU-T T.81 Annex K.3 length limiter, and the block type is chosen
//     on exact sizes (the reference uses a flat header estimate).
//
//   k_link   one CTA per run of tiles: the link of every position to the
//            previous one with the same hash, into scratch.
//   k_search one CTA per group of tiles: their input, window and links
//            staged by bulk copies, the match searched at every position
//            (lanes take new positions as their chains end).
//   k_lparse one CTA per tile: the lazy parse split across lanes with a
//            convergence fix-up (levels 10-12: then the optimal parse), token
//            words and the histogram.
//   k_huff   one CTA per segment: code lengths, canonical codes, block type,
//            RLE code-length header (deflate_block.cpp:196-290 rules).
//   k_enc    one CTA per tile: packs the tokens' codes into the tile's bit
//            buffer.
#include <cuda_runtime.h>
#include <cstdint>
#include "engine.cuh"
#include "deflate_device.cuh"
#include "kernels.cuh"

namespace orotb {

namespace {

constexpr uint32_t kAll = 0xFFFFFFFFu;
constexpr uint32_t T = kLazyTile, W = kLazyWindow;
constexpr uint32_t kMaxDist = 32767;     // farthest candidate a search takes
constexpr uint32_t kLinkDiff = 0x8000u;  // link flag: the linked position starts with other 4 bytes (alone: no link)

// chain, nice, lazy depth, miss limit, optimal parse (levels 10-12)
struct LazyCfg { int chain, nice, lazy, miss, opt; };
__constant__ LazyCfg c_lazy[13] = {
    {0, 0, 0, 5, 0},       {0, 0, 0, 5, 0},       {0, 0, 0, 5, 0},       {0, 0, 0, 5, 0},
    {64, 128, 1, 5, 0},    {128, 128, 1, 5, 0},   {128, 258, 1, 5, 0},   {256, 258, 2, 6, 0},
    {512, 258, 2, 6, 0},   {768, 258, 3, 6, 0},   {1024, 258, 3, 8, 1},  {2048, 258, 3, 8, 1},
    {4096, 258, 3, 8, 1}};

struct SmemBytes {
  const uint32_t* w;  // 16-byte aligned shared words
  uint32_t boff;      // byte offset of region position 0
  __device__ __forceinline__ uint32_t load4(uint32_t r) const {
    const uint32_t i = r + boff;
    return __funnelshift_r(w[i >> 2], w[(i >> 2) + 1], (i & 3) * 8);
  }
};

__device__ __forceinline__ uint32_t hash16(uint32_t v) { return (v * 0x9E3779B1u) >> 16; }
__device__ __forceinline__ uint32_t hash15(uint32_t v) { return (v * 0x9E3779B1u) >> 17; }

// -- staging by the bulk-copy engine (TMA, untiled; the source is this GPU's
// own memory, no multicast): one thread starts the copies and the CTA waits on
// an mbarrier for their bytes.
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Orders this thread's earlier generic-proxy accesses to shared memory before
// later bulk-copy writes (every thread that touched the staged bytes runs it
// before the barrier that precedes the next copy).
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for the mbarrier's phase; gives up (false) after `limit_ns`.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, uint64_t limit_ns) {
  if (mbar_try_wait(bar, phase)) return true;
  const uint64_t t0 = global_ns();
  while (!mbar_try_wait(bar, phase))
    if (global_ns() - t0 > limit_ns) return false;
  return true;
}
constexpr uint64_t kStageWaitNs = 1000000000ull;  // a copy of at most 111 KB that takes a second has failed

// Lanes of the warp whose low NB bits of `h` equal this lane's, among the
// lanes of `among`: one ballot per bit, so the cost does not depend on how
// many values differ (match.any serialises over them).
template <int NB>
__device__ __forceinline__ uint32_t same_bits(uint32_t h, uint32_t among) {
  uint32_t m = among;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const bool on = (h >> b) & 1u;
    const uint32_t bal = __ballot_sync(kAll, on);
    m &= on ? bal : ~bal;
  }
  return m;
}

}  // namespace

// ---------------------------------------------------------------- k_link
// link[x] for every position x of a segment: distance to the latest earlier
// position with the same 15-bit hash (0: none within 32767 bytes), with bit 15
// set when the 4 bytes there are the same too.  One CTA per run of
// consecutive tiles: it first fills its last-position table from the 32 KiB
// before the run (atomicMax, any order), then goes through the run 4,096
// positions a round.  In a round every warp takes four chunks of 32
// positions; links inside a chunk come from ballots over the hash bits, and
// each hash's first and last position in the chunk become one entry.  The
// entries are partitioned, in order, by the top five hash bits into 32 lists,
// and warp b owns list b and its 1,024 table slots: so the ordered part
// (table read, table write) is one warp's walk over 1/32 of the entries, and
// all warps do it at once.
//
// This replaces the ordered pass of one warp over all chunks of a tile inside
// the search kernel: 30% of that kernel on mixed data, with 31 warps idle.
// Bound by instruction issue (the ballots) and four barriers per round.  64 MiB
// of mixed data in 128 KiB blocks 1249 us with ten ballots per 32 entries of a
// list, 1124 with a lane number read back from the table.
namespace {
constexpr uint32_t kLkRound = 4096;             // positions per round: 128 chunks
constexpr uint32_t kLkChunks = kLkRound / 32;
constexpr uint32_t kLkRing = 65536;             // staged input, by arena address mod 64 KiB
struct LinkSmem {
  uint32_t ring[kLkRing / 4];
  uint32_t tbl[32768];                          // last position + 1 of every hash (0: none)
  uint32_t list[kLkRound];                      // first | last << 12, positions in the round
  uint16_t cnt[32][kLkChunks];                  // entries per list and chunk, then their offsets
  uint16_t out[kLkRound];
  uint32_t tot[32];
  uint64_t bar;
};
static_assert(sizeof(LinkSmem) <= 227 * 1024, "one CTA per SM");

struct RingBytes {
  const uint32_t* w;
  uint32_t base;  // ring byte of position 0
  __device__ __forceinline__ uint32_t load4(uint32_t x) const {
    const uint32_t i = x + base;
    return __funnelshift_r(w[(i >> 2) & (kLkRing / 4 - 1)], w[((i >> 2) + 1) & (kLkRing / 4 - 1)], (i & 3) * 8);
  }
};

// Starts the copy of arena bytes [a, b) (multiples of 16, at most 64 KiB) to
// their ring places.
__device__ __forceinline__ void ring_stage(LinkSmem& S, const uint8_t* in, uint64_t a, uint64_t b) {
  mbar_expect(&S.bar, uint32_t(b - a));
  uint8_t* ring = reinterpret_cast<uint8_t*>(S.ring);
  while (a < b) {
    const uint32_t o = uint32_t(a) & (kLkRing - 1);
    const uint32_t n = min(uint32_t(b - a), kLkRing - o);
    bulk_copy(ring + o, in + a, n, &S.bar);
    a += n;
  }
}
}  // namespace

__global__ void __launch_bounds__(1024, 1) k_link(Work wk, const uint32_t* __restrict__ runs, uint32_t nruns) {
  begin_kernel();
  extern __shared__ __align__(128) uint8_t link_sm[];
  LinkSmem& S = *reinterpret_cast<LinkSmem*>(link_sm);
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (blockIdx.x >= nruns) return;
  const uint32_t first = runs[2 * blockIdx.x], count = runs[2 * blockIdx.x + 1];
  const uint32_t seg = wk.tiles[first].seg;
  const Segment sg = wk.segs[seg];
  const uint32_t p0 = wk.tiles[first].start;
  const uint32_t p1 = wk.tiles[first + count - 1].start + wk.tiles[first + count - 1].len;
  const uint32_t hashed = sg.len >= 4 ? sg.len - 3 : 0;  // positions with 4 bytes
  uint16_t* link = reinterpret_cast<uint16_t*>(wk.scratch + sg.links);
  if (p0 == 0 && tid < 320) reinterpret_cast<uint32_t*>(wk.scratch + sg.hist)[tid] = 0;  // k_lparse adds to it
  if (p0 >= p1) return;  // an empty segment's tile
  if (tid == 0) mbar_init(&S.bar, 1);
  for (uint32_t i = tid; i < 32768 / 4; i += 1024) reinterpret_cast<uint4*>(S.tbl)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();

  // staged so far: arena bytes up to `have`; the first copy brings the bytes
  // before the run and the first round's, each later one a round's
  const uint32_t warm0 = p0 > kMaxDist ? p0 - kMaxDist : 0;
  uint64_t have = (sg.in_off + warm0) & ~uint64_t(15);
  auto stage_to = [&](uint32_t x) {  // bytes of positions below x, and the 8 after them
    const uint64_t to = (sg.in_off + min(uint64_t(sg.len), uint64_t(x) + 8) + 15) & ~uint64_t(15);
    if (tid == 0) ring_stage(S, wk.in, have, to);
    have = to;
  };
  stage_to(min(p1, p0 + kLkRound));
  uint32_t phase = 0;
  const RingBytes rb{S.ring, uint32_t(sg.in_off) & (kLkRing - 1)};

  for (uint32_t q0 = p0; q0 < p1; q0 += kLkRound) {
    const bool staged = mbar_wait(&S.bar, phase, kStageWaitNs);
    if (!__syncthreads_and(staged)) {
      // the copy did not complete: mark the stream failed, give the copy
      // another bounded wait so that none is left in flight, and stop
      if (tid == 0) atomicOr(&wk.segs[seg].flags, kSegFault);
      mbar_wait(&S.bar, phase, kStageWaitNs);
      return;
    }
    phase ^= 1u;
    const uint32_t q1 = min(p1, q0 + kLkRound);
    if (q0 == p0 && warm0 < p0) {
      // the table at the start of the run; a position followed by one with
      // the same hash needs no atomic (the later position wins anyway)
      for (uint32_t x = warm0 + 4 * tid; x < min(p0, hashed); x += 4096) {
        const uint32_t i = x + rb.base;
        uint32_t wd[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) wd[j] = S.ring[((i >> 2) + j) & (kLkRing / 4 - 1)];
        const uint32_t lo = __funnelshift_r(wd[0], wd[1], (i & 3) * 8), hi = __funnelshift_r(wd[1], wd[2], (i & 3) * 8);
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = hash15(__funnelshift_r(lo, hi, j * 8));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool in = x + j < min(p0, hashed), next_in = j < 3 && x + j + 1 < min(p0, hashed);
          if (in && !(next_in && h[j] == h[j + 1])) atomicMax(&S.tbl[h[j]], x + j + 1);
        }
      }
      __syncthreads();
    }
    // the next round's bytes; their ring places hold bytes more than 32 KiB
    // behind this round, last read before the barrier above
    if (q1 < p1) stage_to(min(p1, q1 + kLkRound));
    reinterpret_cast<uint2*>(S.cnt)[tid] = make_uint2(0, 0);
    __syncthreads();

    // -- links inside the chunks; one entry per distinct hash of a chunk
    const uint32_t lt = (1u << lane) - 1;
    uint32_t entry[4], where[4];  // entry: first | last << 12; where: list | rank << 8, or kAll
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t c = wid * 4 + j, o = c * 32 + lane, x = q0 + o;
      const bool valid = x < q1 && x < hashed;
      const uint32_t v = valid ? rb.load4(x) : 0u;
      const uint32_t h = hash15(v);
      const uint32_t in_list = same_bits<5>(h >> 10, __ballot_sync(kAll, valid));
      const uint32_t peers = same_bits<10>(h, in_list);
      const uint32_t before = valid ? peers & lt : 0u;
      const uint32_t src = before ? 31 - __clz(before) : lane;
      const uint32_t vs = __shfl_sync(kAll, v, src);
      S.out[o] = before ? uint16_t((lane - src) | (vs == v ? 0u : kLinkDiff)) : uint16_t(kLinkDiff);
      const bool is_first = valid && !before;
      const uint32_t firsts = __ballot_sync(kAll, is_first) & in_list;
      const uint32_t rank = __popc(firsts & lt);
      if (is_first && rank == 0) S.cnt[h >> 10][c] = uint16_t(__popc(firsts));
      entry[j] = o | ((c * 32 + 31 - __clz(peers | 1u)) << 12);
      where[j] = is_first ? (h >> 10) | (rank << 8) : kAll;
    }
    __syncthreads();
    // -- offsets: warp b scans list b's counts over the chunks
    {
      uint2* row = reinterpret_cast<uint2*>(S.cnt[wid]) + lane;  // four chunks per lane
      const uint2 r = *row;
      const uint32_t a = r.x & 0xFFFFu, b = r.x >> 16, c = r.y & 0xFFFFu, d = r.y >> 16;
      uint32_t incl = a + b + c + d;
      const uint32_t sum = incl;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const uint32_t t = __shfl_up_sync(kAll, incl, s);
        if (lane >= uint32_t(s)) incl += t;
      }
      const uint32_t e = incl - sum;
      *row = make_uint2(e | ((e + a) << 16), (e + a + b) | ((e + a + b + c) << 16));
      if (lane == 31) S.tot[wid] = incl;
    }
    __syncthreads();
    // -- scatter the entries to their lists
    const uint32_t mytot = S.tot[lane];
    uint32_t start = mytot;  // exclusive scan over the lists
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t t = __shfl_up_sync(kAll, start, s);
      if (lane >= uint32_t(s)) start += t;
    }
    start -= mytot;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t b = where[j] & 31u;
      const uint32_t sb = __shfl_sync(kAll, start, b);
      if (where[j] != kAll) S.list[sb + S.cnt[b][wid * 4 + j] + (where[j] >> 8)] = entry[j];
    }
    __syncthreads();
    // -- warp b walks list b in order
    {
      const uint32_t l0 = __shfl_sync(kAll, start, wid), n = __shfl_sync(kAll, mytot, wid);
      uint32_t* tb = S.tbl + (wid << 10);
      for (uint32_t k = 0; k < n; k += 32) {
        const bool valid = k + lane < n;
        const uint32_t e = valid ? S.list[l0 + k + lane] : 0u;
        const uint32_t x = q0 + (e & 0xFFFu), xl = q0 + (e >> 12);
        const uint32_t v = rb.load4(x);
        const uint32_t h = hash15(v) & 1023u;
        // What the table holds, then a lane number in its place: entries of one
        // hash read back the same one, whose bits tell them apart.
        uint32_t p = valid ? tb[h] : 0u;  // previous position + 1
        __syncwarp();
        if (valid) tb[h] = lane;
        __syncwarp();
        const uint32_t who = valid ? tb[h] : lane;
        bool last = valid;
        if (__any_sync(kAll, who != lane)) {
          const uint32_t peers = same_bits<5>(who, __ballot_sync(kAll, valid));
          const uint32_t before = valid ? peers & lt : 0u;
          const uint32_t pl = __shfl_sync(kAll, xl, before ? 31 - __clz(before) : lane);
          if (before) p = pl + 1;
          last = valid && (peers >> lane) == 1u;
        }
        if (last) tb[h] = xl + 1;
        __syncwarp();
        if (valid && p && x + 1 - p <= kMaxDist)
          S.out[e & 0xFFFu] = uint16_t((x + 1 - p) | (rb.load4(p - 1) == v ? 0u : kLinkDiff));
      }
    }
    fence_proxy_async_smem();  // this round's reads of the ring, before a later copy into it
    __syncthreads();
    // -- write out; a warp writes the positions whose places it fills next round
    {
      const uint32_t o = wid * 128 + lane * 4;
      const uint2 v = *reinterpret_cast<const uint2*>(S.out + o);
      if (q0 + o + 4 <= q1) {
        *reinterpret_cast<uint2*>(link + q0 + o) = v;
      } else {
        for (uint32_t i = 0; i < 4; ++i)
          if (q0 + o + i < q1) link[q0 + o + i] = S.out[o + i];
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------- k_search
// The longest match at every position, walking the chain newest first
// with the reference's rules (src/deflate/lz77.cpp:66-156): candidates of the
// same 15-bit bucket but another 16-bit hash are skipped, `chain` candidates
// with the same 16-bit hash are examined, miss_limit consecutive 4-byte
// mismatches end the walk, ties keep the nearest, nice length ends the walk.
// Result: length << 16 | distance per position, 0 for no match.
//
// One CTA of 1024 threads searches up to 9 consecutive tiles: their bytes
// and links and the 32 KiB before them (210 KB) come in two bulk copies.
// A warp takes 32 positions at a time and, one per lane, compares each with
// its first candidate; the positions that must go on are queued.  Chains differ
// in length by a factor of hundreds, so a lane takes a position from the queue
// as soon as its chain ends, and only at the end of the whole group do lanes
// run out of positions.
//
// The walk is bound by instruction issue, so a step is one link and one byte:
//   * while the links carry the same-bytes flag the candidate's 4 bytes are
//     known equal and are not loaded;
//   * a longer match must also agree at byte `best`, so one byte rejects most
//     candidates; lanes whose byte agrees stop and are compared together.
// When a match gets longer, the chain of the 4 bytes that end one past it is
// followed a few links: any longer match has these bytes at its own distance,
// so when that chain holds nothing farther than the current candidate the
// search is over.  Neither changes a result: both only skip candidates that
// cannot be longer than the best one.
// Measured with k_link and k_lparse against one CTA per run that did all three
// (B200, ms): 64 MiB mixed at level 6 in 128 KiB chunks 9.1 -> 3.7, 32 MiB text
// at level 9 in 256 KiB chunks 18.7 -> 5.3, the same of 8-byte periods with 1%
// flips 76 -> 12.0, 8 MiB mixed at level 12 9.7 -> 1.8.  Ten candidates per
// round of the warp: 4 cost 25% more on text, 14 the same.
namespace {
constexpr uint32_t kMaxRegion = W + kSearchTiles * T;  // positions with links
constexpr uint32_t kDataBytes = (kMaxRegion + 48 + 127) / 128 * 128;  // + alignment + over-read tail
constexpr uint32_t kLinkBytes = (kMaxRegion * 2 + 127) / 128 * 128;
constexpr uint32_t kSearchSmem = kDataBytes + kLinkBytes;
constexpr int kSearchThreads = 1024;
static_assert(kSearchSmem + kSearchThreads / 32 * 64 * 8 + 64 <= 227 * 1024, "one CTA per SM");
constexpr int kStopped = 0x7FFFFFFF;
constexpr int kWalkSteps = 10;    // candidates a lane takes before the warp compares and re-balances
constexpr int kSlowSteps = 16;    // at most, of the candidates whose 4 bytes are compared
constexpr int kTailHops = 2;     // links followed on the chain one past a new best match

// Common-prefix length (at most maxm) of the bytes at r and at its candidate
// c, whose first 4 bytes agree: aligned words on both sides, each loaded once,
// 16 bytes a step (4 bytes a step cost 15% more on data of long matches).
__device__ __forceinline__ uint32_t match_length(const SmemBytes& sd, uint32_t r, uint32_t c, uint32_t maxm) {
  uint32_t len = 4;
  const uint32_t pi = r + 4 + sd.boff, qi = c + 4 + sd.boff;
  const uint32_t ps = (pi & 3) * 8, qs = (qi & 3) * 8;
  const uint32_t* pw = sd.w + (pi >> 2);
  const uint32_t* qw = sd.w + (qi >> 2);
  uint32_t plo = pw[0], qlo = qw[0];
#pragma unroll 1
  while (len < maxm) {
    uint32_t x[4];
    uint32_t any = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t ph = pw[k + 1], qh = qw[k + 1];
      x[k] = __funnelshift_r(plo, ph, ps) ^ __funnelshift_r(qlo, qh, qs);
      any |= x[k];
      plo = ph;
      qlo = qh;
    }
    if (any) {
      const uint32_t k = x[0] ? 0u : x[1] ? 1u : x[2] ? 2u : 3u;
      const uint32_t v = x[0] ? x[0] : x[1] ? x[1] : x[2] ? x[2] : x[3];
      len += 4 * k + ((__ffs(v) - 1) >> 3);
      break;
    }
    len += 16;
    pw += 4;
    qw += 4;
  }
  return min(len, maxm);
}

// Whether r cannot have a match longer than `len` farther than distance bd:
// such a match has the 4 bytes ending one past `len` at its own distance too,
// so their chain (followed a few links) would hold a position there.
__device__ __forceinline__ bool none_longer(const uint16_t* link, uint32_t r, uint32_t len, uint32_t bd) {
  const int s = int(r + len - 3);
  int u = s;
#pragma unroll 1
  for (int k = 0; k < kTailHops; ++k) {
    const int d = int(link[u] & 0x7FFFu);
    u -= d;
    if (d == 0 || s - u > int(kMaxDist)) return true;
    if (s - u > int(bd)) break;
  }
  return false;
}
}  // namespace

__global__ void __launch_bounds__(kSearchThreads, 1) k_search(Work wk, const uint32_t* __restrict__ runs,
                                                              uint32_t nruns) {
  begin_kernel();
  extern __shared__ __align__(128) uint8_t search_sm[];
  const uint32_t* sdata = reinterpret_cast<const uint32_t*>(search_sm);
  const uint16_t* link = reinterpret_cast<const uint16_t*>(search_sm + kDataBytes);
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t next_chunk;
  __shared__ uint2 queue[kSearchThreads / 32][64];  // positions to walk: offset | length << 16, distance
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  if (blockIdx.x >= nruns) return;
  const uint32_t first = runs[2 * blockIdx.x], count = runs[2 * blockIdx.x + 1];
  const uint32_t seg = wk.tiles[first].seg;
  const Segment sg = wk.segs[seg];
  const LazyCfg cfg = c_lazy[sg.level];
  const uint32_t ts = wk.tiles[first].start, tend = min(sg.len, ts + count * T), tl = tend - ts;
  uint32_t* F = reinterpret_cast<uint32_t*>(wk.scratch + sg.toks) + ts;
  const uint32_t rs = ts > W ? ts - W : 0;  // region start; a multiple of 16 positions
  const uint64_t g0 = (sg.in_off + rs) & ~uint64_t(15);
  const uint32_t boff = uint32_t(sg.in_off + rs - g0);
  const uint32_t data16 = (boff + (min(sg.len, tend + 8) - rs) + 15) / 16;
  const uint32_t link16 = ((tend - rs) * 2 + 15) / 16;
  if (tid == 0) {
    mbar_init(&bar, 1);
    next_chunk = 0;
    mbar_expect(&bar, (data16 + link16) * 16);
    if (data16) bulk_copy(search_sm, wk.in + g0, data16 * 16, &bar);
    if (link16) bulk_copy(search_sm + kDataBytes, wk.scratch + sg.links + uint64_t(rs) * 2, link16 * 16, &bar);
  }
  __syncthreads();
  const bool staged = mbar_wait(&bar, 0, kStageWaitNs);
  if (!__syncthreads_and(staged && !(sg.flags & kSegFault))) {
    // as in k_link; the tiles are left without matches
    if (!staged && tid == 0) atomicOr(&wk.segs[seg].flags, kSegFault);
    mbar_wait(&bar, 0, kStageWaitNs);
    for (uint32_t i = tid; i < tl; i += kSearchThreads) F[i] = 0;
    return;
  }
  const SmemBytes sd{sdata, boff};
  const uint8_t* bytes = search_sm + boff;
  const uint32_t bytes_at = smem_u32(bytes), links_at = smem_u32(link);

  const uint32_t nch = (tl + 31) / 32;
  const uint32_t lt = (1u << lane) - 1;
  uint2* wq = queue[tid >> 5];
  uint32_t nq = 0;   // positions in the warp's queue
  bool more = true;  // chunks left
  uint32_t r = 0, maxm = 0, best = 0, bd = 0, pb = 0, l = 0;
  int pos = 0, pmin = 0, lim = 0, slack = 0, miss = 0;
  bool busy = false;
  bool pure = true;  // the candidate at pos has r's 4 bytes
  for (;;) {
    const uint32_t idle = __ballot_sync(kAll, !busy);
    // -- the warp's next chunks of 32 positions, one per lane: the first
    // candidate, which is all many positions have; the others are queued
    while (more && nq < uint32_t(__popc(idle))) {
      uint32_t c = 0;
      if (lane == 0) c = atomicAdd(&next_chunk, 1u);
      c = __shfl_sync(kAll, c, 0);
      if (c >= nch) {
        more = false;
        break;
      }
      const uint32_t i = c * 32 + lane, p = ts - rs + i;
      const uint32_t end = min(tl, (c * 32 / T + 1) * T);  // a chunk lies in one tile
      const uint32_t mx = i + 4 <= end ? min(258u, end - i) : 0u;
      const uint32_t l1 = mx ? uint32_t(link[p]) : kLinkDiff;
      uint32_t len = 3, dist = 0;
      bool walk = l1 > kLinkDiff;  // other 4 bytes in the bucket: the walk sorts it out
      if (l1 < kLinkDiff) {
        len = match_length(sd, p, p - l1, mx);
        dist = l1;
        walk = int(len) < cfg.nice && len < mx && !none_longer(link, p, len, l1);
      }
      if (!walk && i < tl) F[i] = dist ? (len << 16) | dist : 0u;
      const uint32_t m = __ballot_sync(kAll, walk);
      if (walk) wq[nq + __popc(m & lt)] = make_uint2(i | (len << 16), dist);
      nq += __popc(m);
      __syncwarp();
    }
    const uint32_t take = min(uint32_t(__popc(idle)), nq);
    if (!busy && uint32_t(__popc(idle & lt)) < take) {
      const uint2 e = wq[nq - 1 - __popc(idle & lt)];
      const uint32_t i = e.x & 0xFFFFu;
      busy = true;
      best = e.x >> 16;
      bd = e.y;
      r = ts - rs + i;
      maxm = min(258u, min(tl, (i / T + 1) * T) - i);
      pos = int(r - bd);
      pmin = max(int(r) - int(kMaxDist), 0);
      l = link[pos];
      pb = bytes[r + best];
      lim = cfg.chain - (bd ? 1 : 0);
      slack = cfg.chain + 64;  // 2 * chain + 64 candidates, skipped ones included
      miss = 0;
      pure = true;
    }
    nq -= take;
    __syncwarp();
    if (idle == kAll && take == 0) break;
    // -- candidates known to have the same 4 bytes: one link and one byte
    // each, no branch.  `x` is the shared address of byte `best` of the
    // candidate and `k2` turns it into its link's.  A flagged link is at least
    // 32768 and so leads below `lo` like one out of the window; a lane that
    // has stopped keeps x and loads the same link again.
    bool hit, done;
    {
      const uint32_t to_x = bytes_at + best, k2 = links_at - 2 * to_x;
      uint32_t x = uint32_t(pos) + to_x;
      const bool run = busy && pure;
      int lo = run ? pmin + int(to_x) : kStopped;
#pragma unroll
      for (int k = 0; k < kWalkSteps; ++k)
        asm("{\n"
            " .reg .pred p, q;\n .reg .s32 nx;\n .reg .u32 a, b;\n"
            " sub.s32 nx, %0, %1;\n"
            " setp.ge.s32 p, nx, %2;\n"
            " setp.gt.and.s32 p, %3, 0, p;\n"
            " @p mov.s32 %0, nx;\n"
            " @p add.s32 %3, %3, -1;\n"
            " mad.lo.u32 a, %0, 2, %4;\n"
            " ld.shared.u16 %1, [a];\n"
            " ld.shared.u8 b, [%0];\n"
            " setp.eq.and.u32 q, b, %5, p;\n"
            " @q mov.s32 %2, 0x7FFFFFFF;\n"
            "}"
            : "+r"(x), "+r"(l), "+r"(lo), "+r"(lim)
            : "r"(k2), "r"(pb));
      pos = int(x - to_x);
      hit = run && lo == kStopped;
    }
    // -- the chain's end, or other 4 bytes in the same bucket
    const int d1 = int(l & 0x7FFFu);
    // (with no candidate left to count none can be taken, whatever comes)
    done = busy && !hit && (d1 == 0 || pos - d1 < pmin || lim == 0);
    bool slow = busy && !hit && !done && (!pure || l >= kLinkDiff);
    if (__any_sync(kAll, slow)) {
      const uint32_t v4p = sd.load4(r);
#pragma unroll 1
      for (int k = 0; k < kSlowSteps && slow; ++k) {
        const int d = int(l & 0x7FFFu);
        if (d == 0 || pos - d < pmin) { done = true; break; }
        pos -= d;
        l = link[pos];
        const uint32_t v = sd.load4(uint32_t(pos));
        pure = v == v4p;
        if (!pure && hash16(v) != hash16(v4p)) {  // same 15-bit bucket, other 16-bit chain
          if (slack) --slack;
          else if (lim-- == 0) { done = true; break; }
          continue;
        }
        if (lim-- == 0) { done = true; break; }
        if (!pure) {
          if (++miss >= cfg.miss) { done = true; break; }
          continue;
        }
        miss = 0;
        hit = bytes[pos + best] == pb;
        slow = false;
      }
    }
    // -- candidates that agree at byte `best`
    if (hit && sd.load4(uint32_t(pos) + best - 3) == sd.load4(r + best - 3)) {
      const uint32_t len = match_length(sd, r, uint32_t(pos), maxm);
      if (len > best) {
        best = len;
        bd = r - uint32_t(pos);
        done = int(len) >= cfg.nice || len >= maxm || none_longer(link, r, len, bd);
        pb = bytes[r + len];
      }
    }
    if (done) {
      F[r - (ts - rs)] = bd ? (best << 16) | bd : 0u;
      busy = false;
    }
  }
}

// ---------------------------------------------------------------- k_lparse
// Parse of one tile per CTA from the matches k_search left in the tile's
// token words, which the tokens replace (0x80000000 | length << 16 | distance
// at a match's first position, 0 elsewhere), and its symbol histogram.
//
// Lazy parse (reference rule, lz77.cpp:449-493, with n = tile end): a parse
// step depends only on its start position (the head), so the heads are found
// in parallel: (1) each thread parses one part of the tile from its start; (2)
// it parses again from where the part before was left, until it meets a head of
// its own parse, after which the two are the same, and so on until no part is
// left elsewhere than before; (3) the threads emit the matches of the heads.
// With 32 parts, stitched one after the other by one lane, a tile of text took
// 40 us, now 31 with 128 threads and 15 with 512; 32 MiB of it 302 and 239.
//
// Optimal parse (levels 10-12): costs from the histogram of the lazy parse,
// then a backward pass finds, for every position, the cheapest way to the
// tile end (a literal, or the match found there shortened by up to 31 bytes),
// then the path from position 0 is read.
//
// The chains of one warp are bound by latency, so they run apart from the
// search, up to 16 tiles per SM at once, where the search CTA had one parsing
// warp and 31 waiting ones.
namespace {
constexpr uint32_t kFmWords = T / 32;
static_assert(T % 32 == 0, "tiles are whole windows of 32 positions");
template <int N>  // threads
struct ParseMem {
  uint16_t len[T];         // match length found at each position (optimal: then the token length)
  uint32_t fm[kFmWords];   // positions with a match
  uint32_t hd[kFmWords];   // heads, then the first positions of the parse's matches
  uint32_t em[kFmWords];
  uint32_t hist[320];
  uint32_t sx[N];  // where each part's parse leaves it
};
struct OptMem {
  uint32_t cost[512];      // cost to the tile end, by position mod 512
  uint32_t ring[128];      // prepared positions, by position mod 128
  uint16_t scost[320];     // symbol costs, 1/16 bit: 0-255 literals, 257+ lengths, 288+ distances
  uint16_t lcost[260];     // cost of a match length 0..258 (code + extra bits)
};
template <bool Opt, int N> struct ParseSmem { ParseMem<N> p; };
template <int N> struct ParseSmem<true, N> { ParseMem<N> p; OptMem o; };

// First position >= i where a match starts (a set bit of fm), or tl.
__device__ __forceinline__ uint32_t next_head(const uint32_t* fm, uint32_t i, uint32_t tl) {
  if (i >= tl) return tl;
  uint32_t w = i >> 5;
  uint32_t bits = fm[w] & (kAll << (i & 31));
  while (!bits && ++w < (tl + 31) / 32) bits = fm[w];
  return bits ? min(w * 32 + __ffs(bits) - 1, tl) : tl;
}

// One step of the lazy parse from head i (len[i] != 0): up to `lazy` moves to
// i + 1 while the match there is longer by two or more (the reference's lazy
// rule, lz77.cpp:449-493; the match at i + 1 is the full search of i + 1,
// where the reference searches again with half the chain).  Returns the
// match's position; its length is len there.
__device__ __forceinline__ uint32_t lazy_step(const uint16_t* len, uint32_t i, uint32_t tl, int lazy) {
  uint32_t m = len[i];
  int k = lazy;
  while (k > 0 && i + m + 1 < tl && i + 4 <= tl) {
    const uint32_t g = len[i + 1];
    if (g <= m + 1) break;
    ++i;
    m = g;
    --k;
  }
  return i;
}

// Clears the bits of positions [lo, hi).
__device__ __forceinline__ void clear_bits(uint32_t* bm, uint32_t lo, uint32_t hi) {
  while (lo < hi) {
    const uint32_t w = lo >> 5, b0 = lo & 31, n = min(32u - b0, hi - lo);
    const uint32_t mask = (n == 32 ? kAll : ((1u << n) - 1)) << b0;
    bm[w] &= ~mask;
    lo += n;
  }
}

__device__ __forceinline__ uint32_t len_sym(uint32_t len) {
  uint32_t li, ne, ev;
  length_code(len, li, ne, ev);
  return li;
}
__device__ __forceinline__ uint32_t dist_sym(uint32_t d) {
  uint32_t dc, ne, ev;
  dist_code(d, dc, ne, ev);
  return dc;
}

// Bit cost (1/16 bit) of a token with `count` in a histogram of `total`
// symbols: log2(total / count), 1..15 bits; unseen symbols cost 2 bits more
// than the rarest possible.
__device__ __forceinline__ uint16_t sym_cost(uint32_t count, uint32_t total) {
  const float b = count ? __log2f(float(total) / float(count)) : __log2f(float(total)) + 2.0f;
  return uint16_t(16.0f * fminf(fmaxf(b, 1.0f), 15.0f) + 0.5f);
}

// Histogram of the tokens whose first positions are the bits of m.em (lengths
// in m.len, distances in F's low halves); every byte no match covers is a
// literal.  With `write`, F's words become the tokens.  The warps of the CTA
// share the windows; all threads call it.
template <int N>
__device__ void parse_tokens(ParseMem<N>& m, uint32_t* F, uint32_t tl, const SegBytes& sb, uint32_t ts, bool write) {
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (uint32_t k = threadIdx.x; k < 320; k += uint32_t(N)) m.hist[k] = 0;
  __syncthreads();
  const uint32_t nwin = (tl + 31) / 32;
  const uint32_t per = (nwin + uint32_t(N) / 32 - 1) / (uint32_t(N) / 32);
  const uint32_t wa = min(nwin, wid * per), wb = min(nwin, wa + per);
  uint32_t cover = 0;  // end of the last match before the window (a match reaches 8 windows on at most)
  for (uint32_t w = wa; w > 0 && w + 9 > wa;) {
    const uint32_t bits = m.em[--w];
    if (bits) {
      const uint32_t i = w * 32 + 31 - __clz(bits);
      cover = i + m.len[i];
      break;
    }
  }
  constexpr uint32_t B = 8;  // windows whose loads are in flight together
  for (uint32_t w0 = wa; w0 < wb; w0 += B) {
    uint32_t v[B];  // the match at a token's position, the byte elsewhere
#pragma unroll
    for (uint32_t j = 0; j < B; ++j) {
      const uint32_t w = w0 + j, i = w * 32 + lane;
      const bool tok = w < wb && ((m.em[w] >> lane) & 1u);
      v[j] = tok ? F[i] : w < wb && i < tl ? sb.byte(ts + i) : 0u;
    }
#pragma unroll
    for (uint32_t j = 0; j < B; ++j) {
      const uint32_t w = w0 + j, i = w * 32 + lane;
      if (w >= wb) break;
      const uint32_t bits = m.em[w];
      const bool tok = (bits >> lane) & 1u;
      const uint32_t len = tok ? m.len[i] : 0u;
      // matches do not overlap, so the nearest one before a position decides
      const uint32_t prior = bits & ((1u << lane) - 1);
      const uint32_t pend = __shfl_sync(kAll, i + len, prior ? 31 - __clz(prior) : 0);
      const uint32_t end = prior ? pend : cover;
      if (tok) {
        atomicAdd(&m.hist[257 + len_sym(len)], 1u);
        atomicAdd(&m.hist[288 + dist_sym(v[j] & 0xFFFFu)], 1u);
      } else if (i < tl && end <= i) {
        atomicAdd(&m.hist[v[j]], 1u);
      }
      if (write && i < tl) F[i] = tok ? 0x80000000u | (len << 16) | (v[j] & 0xFFFFu) : 0u;
      if (bits) cover = __shfl_sync(kAll, i + len, 31 - __clz(bits));
    }
  }
  __syncthreads();
}
}  // namespace

template <bool Opt, int N>
__global__ void __launch_bounds__(N) k_lparse(Work wk, const uint32_t* __restrict__ list, uint32_t nlist) {
  begin_kernel();
  __shared__ ParseSmem<Opt, N> S;
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (blockIdx.x >= nlist) return;
  Tile* tp = wk.tiles + list[blockIdx.x];
  const Tile t = *tp;
  const Segment sg = wk.segs[t.seg];
  const LazyCfg cfg = c_lazy[sg.level];
  if ((cfg.opt != 0) != Opt) return;  // the other kernel's tile
  ParseMem<N>& m = S.p;
  uint32_t* F = reinterpret_cast<uint32_t*>(wk.scratch + t.tok);
  const uint32_t tl = t.len, ts = t.start;
  const uint64_t o = sg.in_off;
  const SegBytes sb{reinterpret_cast<const uint32_t*>(wk.in + (o & ~uint64_t(3))), uint32_t(o & 3)};

  // -- lengths and the match bitmap, a warp's loads of eight windows in flight
  constexpr uint32_t kWarps = uint32_t(N) / 32;
  for (uint32_t w0 = 0; w0 < kFmWords; w0 += 8 * kWarps) {
    uint32_t f[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
      const uint32_t i = (w0 + j * kWarps + wid) * 32 + lane;
      f[j] = i < tl ? F[i] : 0u;
    }
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
      const uint32_t w = w0 + j * kWarps + wid;
      const uint32_t b = __ballot_sync(kAll, f[j] != 0);
      if (w < kFmWords) {
        m.len[w * 32 + lane] = uint16_t(f[j] >> 16);
        if (lane == 0) m.fm[w] = b;
      }
    }
  }
  for (uint32_t w = tid; w < kFmWords; w += uint32_t(N)) m.hd[w] = m.em[w] = 0;
  __syncthreads();

  // -- heads of the lazy parse: thread k those from part k's first position on,
  // then again from where part k - 1 was left, until no exit changes
  {
    const uint32_t part = ((tl + 32 * uint32_t(N) - 1) / (32 * uint32_t(N))) * 32;
    const uint32_t a = min(tid * part, tl), b = min(a + part, tl);
    uint32_t entry = a;
    auto walk = [&](bool again) {
      uint32_t i = entry;
      if (again) clear_bits(m.hd, a, min(i, b));
      for (;;) {
        const uint32_t h = i < b ? next_head(m.fm, i, b) : b;
        if (h >= b) {
          m.sx[tid] = max(i, b);
          return;
        }
        const uint32_t bit = 1u << (h & 31);
        if (again && (m.hd[h >> 5] & bit)) return;  // from here on as before
        m.hd[h >> 5] |= bit;  // a part is whole words
        i = lazy_step(m.len, h, tl, cfg.lazy);
        i += m.len[i];
        if (again) clear_bits(m.hd, h + 1, min(i, b));
      }
    };
    walk(false);
    for (;;) {
      __syncthreads();
      const uint32_t e = tid ? m.sx[tid - 1] : 0u;
      const bool again = a < b && e != entry;
      if (!__syncthreads_or(again)) break;
      if (again) {
        entry = e;
        walk(true);
      }
    }
  }
  // -- the matches of the heads
  for (uint32_t w = tid; w < kFmWords; w += uint32_t(N)) {
    uint32_t bits = m.hd[w];
    while (bits) {
      const uint32_t i = lazy_step(m.len, w * 32 + __ffs(bits) - 1, tl, cfg.lazy);
      bits &= bits - 1;
      atomicOr(&m.em[i >> 5], 1u << (i & 31));
    }
  }
  __syncthreads();

  if constexpr (Opt) {
    OptMem& c = S.o;
    parse_tokens(m, F, tl, sb, ts, false);
    if (wid == 0) {
      {
        uint32_t ltot = 0, dtot = 0;
        for (uint32_t k = lane; k < 286; k += 32) ltot += m.hist[k];
        for (uint32_t k = 288 + lane; k < 318; k += 32) dtot += m.hist[k];
        ltot = __reduce_add_sync(kAll, ltot) + 1;  // EOB counts once
        dtot = __reduce_add_sync(kAll, dtot);
        for (uint32_t k = lane; k < 320; k += 32)
          c.scost[k] = k < 288 ? sym_cost(m.hist[k], ltot) : sym_cost(m.hist[k], dtot > 0 ? dtot : 1);
      }
      __syncwarp();
      for (uint32_t k = lane; k < 259; k += 32) {
        uint32_t ls = 0, lne = 0, lev;
        if (k >= 3) length_code(k, ls, lne, lev);
        c.lcost[k] = k >= 3 ? uint16_t(c.scost[257 + ls] + 16 * lne) : uint16_t(0);
      }
      for (uint32_t k = lane; k < 512; k += 32) c.cost[k] = 0;  // positions past the tile end cost nothing
      for (uint32_t k = lane; k < 128; k += 32) c.ring[k] = 0;  // positions before the tile (a last group of one or two)
      __syncwarp();
      // Positions are prepared a window at a time, one per lane: match length |
      // literal cost << 9 | distance cost << 17, in a ring of four windows; the
      // loads of the window after next are in flight meanwhile.
      uint32_t fpre = 0, bpre = 0;
      auto fetch = [&](int w) {
        const uint32_t j = uint32_t(w) * 32 + lane;
        const bool in = w >= 0 && j < tl;
        fpre = in ? F[j] : 0u;
        bpre = in ? sb.byte(ts + j) : 0u;
      };
      auto prepare = [&](int w) {
        uint32_t dc = 0, dne = 0, dev;
        if (fpre) dist_code(fpre & 0xFFFFu, dc, dne, dev);
        const uint32_t dcost = fpre ? c.scost[288 + dc] + 16 * dne : 0u;
        c.ring[(uint32_t(w) * 32 + lane) & 127] = (fpre >> 16) | (uint32_t(c.scost[bpre]) << 9) | (dcost << 17);
      };
      // cost << 9 | length of this lane's way to shorten the match of position i
      auto match_key = [&](int i, uint32_t e) {
        const uint32_t flen = e & 511u, L = flen - lane;
        return lane + 3 <= flen ? ((c.lcost[L] + (e >> 17) + c.cost[(uint32_t(i) + L) & 511]) << 9) | L : kAll;
      };
      int pw = int(tl + 31) / 32;  // windows from here on are prepared
      fetch(pw - 1);
      uint32_t next = 0;  // cost of the position after the current one
      // Three positions at a time: a match is at least 3 long, so the matches of
      // all three lead past the first and their minima do not wait for each
      // other; only the literals go from one position to the next.
      for (int i = int(tl) - 1; i >= 0; i -= 3) {
        while (pw > 0 && pw > (i >> 5) - 1) {
          prepare(--pw);
          fetch(pw - 1);
          __syncwarp();
        }
        const uint32_t e0 = c.ring[i & 127], e1 = c.ring[(i - 1) & 127], e2 = c.ring[(i - 2) & 127];
        uint32_t m0 = kAll, m1 = kAll, m2 = kAll;
        if ((e0 | e1 | e2) & 511u) {
          m0 = __reduce_min_sync(kAll, match_key(i, e0));
          m1 = __reduce_min_sync(kAll, match_key(i - 1, e1));
          m2 = __reduce_min_sync(kAll, match_key(i - 2, e2));
        }
        const uint32_t b0 = min(m0, ((((e0 >> 9) & 255u) + next) << 9) | 1u);
        const uint32_t b1 = min(m1, ((((e1 >> 9) & 255u) + (b0 >> 9)) << 9) | 1u);
        const uint32_t b2 = min(m2, ((((e2 >> 9) & 255u) + (b1 >> 9)) << 9) | 1u);
        next = b2 >> 9;
        const uint32_t v = lane == 0 ? b0 : lane == 1 ? b1 : b2;
        if (lane < 3 && i >= int(lane)) {
          c.cost[(uint32_t(i) - lane) & 511] = v >> 9;
          m.len[uint32_t(i) - lane] = uint16_t(v & 511u);
        }
        __syncwarp();
      }
      for (uint32_t w = lane; w < kFmWords; w += 32) m.em[w] = 0;
      __syncwarp();
      if (lane == 0) {
        uint32_t i = 0, word = 0, bits = 0;  // the bits of the word being filled
        while (i < tl) {
          const uint32_t n = m.len[i];
          if ((i >> 5) != word) {
            m.em[word] = bits;
            word = i >> 5;
            bits = 0;
          }
          bits |= (n >= 3 ? 1u : 0u) << (i & 31);
          i += n;
        }
        m.em[word] = bits;
      }
    }
    __syncthreads();
  }

  parse_tokens(m, F, tl, sb, ts, true);
  uint32_t* gh = reinterpret_cast<uint32_t*>(wk.scratch + sg.hist);  // the segment's, cleared by k_link
  for (uint32_t i = tid; i < 320; i += uint32_t(N))
    if (m.hist[i]) atomicAdd(&gh[i], m.hist[i]);
  if (wid == 0) {
    uint32_t nm = 0;
    for (uint32_t w = lane; w < kFmWords; w += 32) nm += __popc(m.em[w]);
    nm = __reduce_add_sync(kAll, nm);
    if (lane == 0) {
      tp->fin_matches = nm;
      tp->fix_bits = 0;
      tp->splice_bit = 0;
    }
  }
}

// ---------------------------------------------------------------- Huffman
// Code lengths, canonical codes, the block type and the code-length header of
// one segment per CTA, one thread per symbol (288 literal/length symbols in
// nine warps, 32 distance symbols in the tenth).  Only the two-queue merge is
// sequential: leaves in order of (frequency, symbol), internal nodes in
// creation order, a leaf wins a tie; one thread per alphabet, with the next
// leaves and nodes in registers so that a step does not wait for shared
// memory.  Ranks, depths, codes, run lengths and header bits are found in
// parallel.  Bound by the latency of the merge (285 steps at most).
//
// One warp did all this on one lane (and summed the tiles' histograms, now
// added up by k_lparse): 107 us for a segment of 4 KiB and 1.7 ms for one of
// 16 MiB, now 19 us and 35 us; 512 segments of 128 KiB 0.33 ms, now 0.06.
namespace {

constexpr int kHuffThreads = 320;
constexpr uint32_t kNone = 0xFFFFFFFFu;

// A Huffman tree over sorted leaf frequencies (kNone past the last).
template <int N>
struct Tree {
  uint32_t leaf[N + 4], node[N + 4];  // node weights in creation order, kNone where not made yet
  uint16_t par[2 * N];                // parent of leaf i at i, of node k at m + k
};

// The two-queue merge of m >= 2 leaves (one thread).
template <int N>
__device__ void merge_queues(Tree<N>& t, int m) {
  uint32_t l0 = t.leaf[0], l1 = t.leaf[1], l2 = t.leaf[2], l3 = t.leaf[3];
  uint32_t n0 = kNone, n1 = kNone, n2 = kNone, n3 = kNone;
  int li = 0, ni = 0;
  for (int k = 0; k < m - 1; ++k) {
    const bool a = l0 <= n0;
    const uint32_t lb = a ? l1 : l0, nb = a ? n0 : n1;
    const bool b = lb <= nb;
    const uint32_t sum = (a ? l0 : n0) + (b ? lb : nb);
    t.par[a ? li : m + ni] = uint16_t(m + k);
    li += a ? 1 : 0;
    ni += a ? 0 : 1;
    t.par[b ? li : m + ni] = uint16_t(m + k);
    li += b ? 1 : 0;
    ni += b ? 0 : 1;
    const int c = (a ? 1 : 0) + (b ? 1 : 0);  // leaves taken, of two
    l0 = c == 0 ? l0 : c == 1 ? l1 : l2;
    l1 = c == 0 ? l1 : c == 1 ? l2 : l3;
    n0 = c == 2 ? n0 : c == 1 ? n1 : n2;
    n1 = c == 2 ? n1 : c == 1 ? n2 : n3;
    l2 = t.leaf[li + 2];
    l3 = t.leaf[li + 3];
    n2 = t.node[ni + 2];
    n3 = t.node[ni + 3];
    t.node[k] = sum;
    const int at = k - ni;
    if (at == 0) n0 = sum;
    if (at == 1) n1 = sum;
    if (at == 2) n2 = sum;
    if (at == 3) n3 = sum;
  }
}

// Depth of leaf r in a tree of m >= 2 leaves.
template <int N>
__device__ __forceinline__ uint32_t leaf_depth(const Tree<N>& t, uint32_t r, uint32_t m) {
  uint32_t d = 1;
  for (uint32_t x = t.par[r]; x != 2 * m - 2; x = t.par[x]) ++d;
  return d;
}

// Adjusts the counts per length so that none exceeds `limit` (ITU-T T.81 Annex K.3; one thread).
__device__ void limit_counts(uint32_t* cnt, int limit) {
  for (int i = 63; i > limit; --i) {
    while (cnt[i] > 0) {
      int j = i - 2;
      while (cnt[j] == 0) --j;
      cnt[i] -= 2;
      cnt[i - 1] += 1;
      cnt[j + 1] += 2;
      cnt[j] -= 1;
    }
  }
}
// Length of the leaf of rank r (least frequent first) under adjusted counts:
// the longest lengths go to the least frequent symbols.
__device__ __forceinline__ uint32_t limited_length(const uint32_t* cnt, int limit, uint32_t r) {
  int l = limit;
  for (uint32_t c = cnt[l]; r >= c; c += cnt[l]) --l;
  return uint32_t(l);
}

struct HuffSmem {
  alignas(16) uint32_t freq[320];
  Tree<288> lit;
  Tree<32> dist;
  Tree<20> cl;
  uint32_t cnt[2][64], clcnt[64];    // codes per length, where a tree is too deep
  uint32_t used[2], deep[2], clused, cldeep, matches;
  uint32_t groups[10][16], next[2][16];
  uint8_t len[320], seq[320];
  uint32_t runs[10], scan[10];
  uint32_t top[2];                   // symbols up to the last used one
  uint8_t rsym[320], rext[320];      // run-length coded lengths
  uint32_t clf[19], clc[19];         // code-length code: counts, code | length << 16
  uint32_t hdr[160];
  unsigned long long sums[3];        // extra bits, fixed code, dynamic code
};

// Exclusive scan over the CTA and its total (all threads; a barrier on each side).
__device__ __forceinline__ uint32_t huff_scan(HuffSmem& S, uint32_t v, uint32_t& total) {
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const uint32_t t = __shfl_up_sync(kAll, incl, k);
    if (lane >= uint32_t(k)) incl += t;
  }
  __syncthreads();
  if (lane == 31) S.scan[wid] = incl;
  __syncthreads();
  uint32_t below = 0;
  total = 0;
  for (uint32_t k = 0; k < 10; ++k) {
    if (k < wid) below += S.scan[k];
    total += S.scan[k];
  }
  return below + incl - v;
}

// Canonical codes (RFC 1951 3.2.2), reversed for LSB-first output, of the
// thread's symbol of length `len` in its alphabet: code | length << 16.
__device__ uint32_t canon_code(HuffSmem& S, uint32_t len) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint32_t peers = kAll;  // lanes of the same length
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t bal = __ballot_sync(kAll, (len >> k) & 1u);
    peers &= (len >> k) & 1u ? bal : ~bal;
  }
  const uint32_t before = __popc(peers & ((1u << lane) - 1));
  __syncthreads();
  if (tid < 160) S.groups[tid >> 4][tid & 15] = 0;
  __syncthreads();
  if (len && !before) S.groups[wid][len] = __popc(peers);
  __syncthreads();
  if (tid < 32) {  // lane l and 16 + l: codes of length l of the two alphabets
    const uint32_t l = lane & 15;
    uint32_t n = 0;
    if (lane < 16) {
      for (int k = 0; k < 9; ++k) n += S.groups[k][l];
    } else {
      n = S.groups[9][l];
    }
    uint32_t code = 0;
    for (int k = 1; k < 16; ++k) {  // code = (code + count of the length before) << 1
      const uint32_t c = __shfl_sync(kAll, n, (lane & 16) + k - 1);
      if (uint32_t(k) <= l) code = (code + c) << 1;
    }
    S.next[lane >> 4][l] = code;
  }
  __syncthreads();
  if (!len) return 0;
  uint32_t code = S.next[wid == 9][len] + before;
  if (wid < 9)
    for (uint32_t k = 0; k < wid; ++k) code += S.groups[k][len];
  return rev_bits(code, len) | (len << 16);
}

constexpr uint32_t kLimitBits = 15, kClLimitBits = 7;
__device__ __forceinline__ uint32_t fixed_length(uint32_t tid) {
  return tid < 144 ? 8u : tid < 256 ? 9u : tid < 280 ? 7u : tid < 288 ? 8u : 5u;
}
__constant__ uint8_t c_cl_order[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

}  // namespace

__global__ void __launch_bounds__(kHuffThreads) k_huff(Work wk, const uint32_t* __restrict__ list, uint32_t nlist) {
  begin_kernel();
  __shared__ HuffSmem S;
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (blockIdx.x >= nlist) return;
  Segment* gp = wk.segs + list[blockIdx.x];
  const Segment sg = *gp;
  const uint32_t al = wid == 9 ? 1u : 0u;             // alphabet
  const uint32_t i = al ? tid - 288 : tid;            // symbol in it
  const uint32_t f = tid == 256 ? 1u : reinterpret_cast<const uint32_t*>(wk.scratch + sg.hist)[tid];  // one end of block
  S.freq[tid] = f;
  for (uint32_t k = tid; k < 292; k += kHuffThreads) S.lit.leaf[k] = S.lit.node[k] = kNone;
  if (tid < 36) S.dist.leaf[tid] = S.dist.node[tid] = kNone;
  if (tid < 24) S.cl.leaf[tid] = S.cl.node[tid] = kNone;
  if (tid < 128) S.cnt[tid >> 6][tid & 63] = 0;
  if (tid < 64) S.clcnt[tid] = 0;
  if (tid < 19) S.clf[tid] = 0;
  if (tid < 160) S.hdr[tid] = 0;
  if (tid < 2) S.used[tid] = S.deep[tid] = S.top[tid] = 0;
  if (tid < 3) S.sums[tid] = 0;
  if (tid == 0) S.cldeep = 0;
  __syncthreads();
  {
    const uint32_t n = __popc(__ballot_sync(kAll, f != 0));
    if (lane == 0) atomicAdd(&S.used[al], n);
    const bool any = __any_sync(kAll, f != 0);
    if (wid == 9 && lane == 0) S.matches = any ? 1u : 0u;  // a match has a distance
  }
  __syncthreads();
  if ((sg.flags & kSegWholeBuf) && !S.matches) {  // all-literal parse (block_compressor.cpp:60-61)
    if (tid == 0) {
      gp->block_type = kBlkStored;
      gp->hdr_bits = 0;
      gp->eob = 0;
    }
    return;
  }

  // -- code lengths
  const uint32_t m = S.used[al];
  uint32_t rank = 0;
  {
    // used symbols before this one by (frequency, symbol); f - 1 sends 0 to the end
    const uint4* fv = reinterpret_cast<const uint4*>(S.freq + (al ? 288 : 0));
    const uint32_t key = f - 1u;
    for (uint32_t k = 0; k < (al ? 8u : 72u); ++k) {
      const uint4 v = fv[k];
      rank += v.x - 1u < key || (v.x == f && 4 * k < i) ? 1 : 0;
      rank += v.y - 1u < key || (v.y == f && 4 * k + 1 < i) ? 1 : 0;
      rank += v.z - 1u < key || (v.z == f && 4 * k + 2 < i) ? 1 : 0;
      rank += v.w - 1u < key || (v.w == f && 4 * k + 3 < i) ? 1 : 0;
    }
  }
  if (f) (al ? S.dist.leaf : S.lit.leaf)[rank] = f;
  __syncthreads();
  if (tid == 0 && m >= 2) merge_queues(S.lit, int(m));
  if (tid == 288 && m >= 2) merge_queues(S.dist, int(m));
  __syncthreads();
  uint32_t len = 0;
  if (f) {
    len = m < 2 ? 1u : al ? leaf_depth(S.dist, rank, m) : leaf_depth(S.lit, rank, m);
    if (len > kLimitBits) S.deep[al] = 1;
    atomicAdd(&S.cnt[al][min(len, 63u)], 1u);
  }
  __syncthreads();
  if ((tid == 0 || tid == 288) && S.deep[al]) limit_counts(S.cnt[al], kLimitBits);
  __syncthreads();
  if (f && S.deep[al]) len = limited_length(S.cnt[al], kLimitBits, rank);
  if (tid == 288 && m == 0) len = 1;  // no distance: one code of one bit (deflate_block.cpp:347-383 conventions)
  S.len[tid] = uint8_t(len);
  if (len) atomicMax(&S.top[al], i + 1);
  __syncthreads();
  const uint32_t hlit = max(257u, S.top[0]), hdist = max(1u, S.top[1]), total = hlit + hdist;

  // -- run-length code of the lengths (deflate_block.cpp:212-242): each run of
  // equal lengths is coded by itself, up to 138 at a time: zeros (3 or more)
  // by 17 or 18; others (4 or more) once, then up to six by 16; else singly
  const uint32_t v = tid < total ? S.len[tid < hlit ? tid : 288 + tid - hlit] : 0u;
  S.seq[tid] = uint8_t(v);
  __syncthreads();
  const bool start = tid < total && (tid == 0 || S.seq[tid - 1] != v);
  const uint32_t starts = __ballot_sync(kAll, start);
  if (lane == 0) S.runs[wid] = starts;
  __syncthreads();
  uint32_t left = 0;  // length of the run that starts here
  if (start) {
    uint32_t w = wid, bits = starts & ~((2u << lane) - 1u);
    while (!bits && ++w < 10) bits = S.runs[w];
    left = (bits ? w * 32 + __ffs(bits) - 1 : total) - tid;
  }
  auto code_run = [&](uint32_t at, bool write) {  // returns the number of codes
    uint32_t n = 0;
    auto put = [&](uint32_t sym, uint32_t ext) {
      if (write) {
        S.rsym[at + n] = uint8_t(sym);
        S.rext[at + n] = uint8_t(ext);
        atomicAdd(&S.clf[sym], 1u);
      }
      ++n;
    };
    for (uint32_t rest = left; rest;) {
      const uint32_t run = min(rest, 138u);
      if (v == 0 && run >= 3) {
        put(run <= 10 ? 17 : 18, run <= 10 ? run - 3 : run - 11);
        rest -= run;
      } else if (v != 0 && run >= 4) {
        const uint32_t rep = min(run - 1, 6u);
        put(v, 0);
        put(16, rep - 3);
        rest -= 1 + rep;
      } else {
        put(v, 0);
        --rest;
      }
    }
    return n;
  };
  uint32_t ncodes;
  const uint32_t at = huff_scan(S, code_run(0, false), ncodes);
  code_run(at, true);
  __syncthreads();

  // -- the code-length code (warp 0): lengths of at most 7 bits, codes
  if (wid == 0) {
    const uint32_t cf = lane < 19 ? S.clf[lane] : 0u;
    const uint32_t n = __popc(__ballot_sync(kAll, cf != 0));
    uint32_t r = 0;
    for (int k = 0; k < 19; ++k) {
      const uint32_t o = __shfl_sync(kAll, cf, k);
      r += o - 1u < cf - 1u || (o == cf && uint32_t(k) < lane) ? 1 : 0;
    }
    if (cf) S.cl.leaf[r] = cf;
    __syncwarp();
    if (lane == 0 && n >= 2) merge_queues(S.cl, int(n));
    __syncwarp();
    uint32_t cl = !cf ? 0u : n < 2 ? 1u : leaf_depth(S.cl, r, n);
    if (__any_sync(kAll, cl > kClLimitBits)) {
      if (cf) atomicAdd(&S.clcnt[cl], 1u);
      __syncwarp();
      if (lane == 0) limit_counts(S.clcnt, kClLimitBits);
      __syncwarp();
      if (cf) cl = limited_length(S.clcnt, kClLimitBits, r);
    }
    uint32_t code = 0, mine = 0, prev = 0;
#pragma unroll
    for (uint32_t l = 1; l <= kClLimitBits; ++l) {
      code = (code + __popc(prev)) << 1;
      prev = __ballot_sync(kAll, cl == l);
      if (cl == l) mine = code + __popc(prev & ((1u << lane) - 1));
    }
    if (lane < 19) S.clc[lane] = cl ? rev_bits(mine, cl) | (cl << 16) : 0u;
  }
  __syncthreads();
  // -- header bits: HLIT, HDIST, HCLEN, the code-length code's lengths, the codes
  uint32_t hclen;
  {
    const uint32_t used = __ballot_sync(kAll, lane < 19 && S.clc[c_cl_order[lane < 19 ? lane : 0]] != 0);
    hclen = max(4u, 32u - __clz(used));
  }
  uint32_t bits = 0, nb = 0;
  if (tid < ncodes) {
    const uint32_t sym = S.rsym[tid], c = S.clc[sym];
    nb = (c >> 16) + (sym == 16 ? 2u : sym == 17 ? 3u : sym == 18 ? 7u : 0u);
    bits = (c & 0xFFFFu) | (uint32_t(S.rext[tid]) << (c >> 16));
  }
  uint32_t code_bits;
  const uint32_t pos = 14 + 3 * hclen + huff_scan(S, nb, code_bits);
  auto put_bits = [&](uint32_t at_bit, uint32_t val, uint32_t n) {
    atomicOr(&S.hdr[at_bit >> 5], val << (at_bit & 31));
    if ((at_bit & 31) + n > 32) atomicOr(&S.hdr[(at_bit >> 5) + 1], val >> (32 - (at_bit & 31)));
  };
  if (nb) put_bits(pos, bits, nb);
  if (tid < hclen) put_bits(14 + 3 * tid, S.clc[c_cl_order[tid]] >> 16, 3);
  if (tid == 0) put_bits(0, (hlit - 257) | ((hdist - 1) << 5) | ((hclen - 4) << 10), 14);
  const uint32_t hbits = 14 + 3 * hclen + code_bits;

  // -- block type on exact sizes
  {
    uint32_t x = 0;  // extra bits of the symbol
    if (!al && i >= 265 && i < 285) x = ((i - 257) >> 2) - 1;
    if (al && i >= 4 && i < 30) x = (i >> 1) - 1;
    unsigned long long e = (unsigned long long)(f) * x;
    unsigned long long fx = al && i >= 30 ? 0ull : (unsigned long long)(f) * fixed_length(tid);
    unsigned long long dy = (unsigned long long)(f) * len;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      e += __shfl_xor_sync(kAll, e, o);
      fx += __shfl_xor_sync(kAll, fx, o);
      dy += __shfl_xor_sync(kAll, dy, o);
    }
    if (lane == 0) {
      atomicAdd(&S.sums[0], e);
      atomicAdd(&S.sums[1], fx);
      atomicAdd(&S.sums[2], dy);
    }
  }
  __syncthreads();
  const uint32_t pieces = sg.len ? (sg.len + 65534) / 65535 : 1;
  const uint64_t stored_bits = (uint64_t(sg.len) + 5ull * pieces) * 8;
  const uint64_t fixed_bits = 3 + S.sums[0] + S.sums[1], dyn_bits = 3 + hbits + S.sums[0] + S.sums[2];
  const uint32_t type = stored_bits <= fixed_bits && stored_bits <= dyn_bits ? kBlkStored
                        : fixed_bits <= dyn_bits                             ? kBlkFixed
                                                                             : kBlkDynamic;
  if (type == kBlkFixed) len = fixed_length(tid);
  if (type != kBlkStored) {
    const uint32_t c = canon_code(S, len);
    reinterpret_cast<uint32_t*>(wk.scratch + sg.codes)[tid] = c;
    if (tid == 256) gp->eob = c;
  } else if (tid == 0) {
    gp->eob = 0;
  }
  if (type == kBlkDynamic && tid < 160) reinterpret_cast<uint32_t*>(wk.scratch + sg.hdr_off)[tid] = S.hdr[tid];
  if (tid == 0) {
    gp->block_type = type;
    gp->hdr_bits = type == kBlkDynamic ? hbits : 0;
  }
}

// ---------------------------------------------------------------- k_enc
// Codes of one tile per CTA.  Warps take runs of 32-position windows: a first
// pass sums each warp's bits, a scan gives its place, a second pass packs the
// codes into the tile's bits in shared memory, which are written out in order.
// A position belongs to a token unless the nearest match before it reaches it.
// One warp per tile, a window after the other with the token chain followed by
// shuffles, took 137 us for a single tile, this 24, 16 with 512 threads; 64 MiB of mixed data
// 0.44 ms and 0.38 (the packing is bound by issue, each pass once per window).
template <int N>
__global__ void __launch_bounds__(N) k_enc(Work wk, const uint32_t* __restrict__ list, uint32_t nlist) {
  begin_kernel();
  constexpr uint32_t kWarps = N / 32;
  // literal codes; per match length code and extra bits | their number << 24;
  // per distance - 1 below 256, or 256 + its bits above the 7th, the code |
  // its bits << 16 | extra bits << 20
  __shared__ uint32_t code[256], lens[259], dists[512];
  __shared__ uint32_t buf[kLazyTile / 2 + 64];  // at most 16 bits per byte (lazy_stream_bytes)
  __shared__ uint32_t warp_bits[kWarps];
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (blockIdx.x >= nlist) return;
  Tile* tp = wk.tiles + list[blockIdx.x];
  const Tile t = *tp;
  const Segment sg = wk.segs[t.seg];
  if (sg.block_type == kBlkStored) {
    if (tid == 0) { tp->spec_bits = 0; tp->spec_exit = t.start + t.len; }
    return;
  }
  const uint32_t* codes = reinterpret_cast<const uint32_t*>(wk.scratch + sg.codes);
  for (uint32_t k = tid; k < 1024; k += N) {
    if (k < 256) {
      code[k] = codes[k];
    } else if (k < 512) {
      uint32_t li, le, lv;
      length_code(k - 253, li, le, lv);  // 3 to 258
      const uint32_t c = codes[257 + li], n = c >> 16;
      lens[k - 253] = (c & 0xFFFFu) | (lv << n) | ((n + le) << 24);
    } else {
      const uint32_t i = k - 512;
      uint32_t dc, de, dv;
      dist_code((i < 256 ? i : (i - 256) << 7) + 1, dc, de, dv);
      dists[i] = codes[288 + dc] | (de << 20);
    }
  }
  for (uint32_t k = tid; k < kLazyTile / 2 + 64; k += N) buf[k] = 0;
  const uint32_t* tok = reinterpret_cast<const uint32_t*>(wk.scratch + t.tok);
  const uint64_t o = sg.in_off;
  const SegBytes sb{reinterpret_cast<const uint32_t*>(wk.in + (o & ~uint64_t(3))), uint32_t(o & 3)};
  const uint32_t nwin = (t.len + 31) / 32, per = (nwin + kWarps - 1) / kWarps;
  const uint32_t wa = min(nwin, wid * per), wb = min(nwin, wa + per);
  // end of the last match before the warp's windows (it starts at most 257 positions back)
  uint32_t cover0 = 0;
  for (uint32_t w = wa; w > 0 && w + 9 > wa;) {
    --w;
    const uint32_t tk = tok[w * 32 + lane];
    const uint32_t b = __ballot_sync(kAll, tk != 0);
    if (b) {
      const uint32_t j = 31 - __clz(b);
      cover0 = w * 32 + j + ((__shfl_sync(kAll, tk, j) >> 16) & 0x1FFu);
      break;
    }
  }
  __syncthreads();
  // walks the warp's windows; emit(token's two parts) per position
  auto walk = [&](auto&& emit) {
    uint32_t cover = cover0;
    for (uint32_t w0 = wa; w0 < wb; w0 += 4) {
      uint32_t tk4[4], by4[4];  // four windows' loads in flight
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t i = (w0 + k) * 32 + lane;
        const bool in = w0 + k < wb && i < t.len;
        tk4[k] = in ? tok[i] : 0u;
        by4[k] = in ? sb.byte(t.start + i) : 0u;
      }
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        if (w0 + k >= wb) break;
        const uint32_t i = (w0 + k) * 32 + lane, tk = tk4[k], len = (tk >> 16) & 0x1FFu;
        const uint32_t heads = __ballot_sync(kAll, tk != 0), prior = heads & ((1u << lane) - 1);
        if (!heads && cover >= (w0 + k) * 32 + 32) continue;  // within one match
        const uint32_t pend = __shfl_sync(kAll, i + len, prior ? 31 - __clz(prior) : 0);
        const uint32_t end = prior ? pend : cover;
        uint32_t a = 0, na = 0, b = 0, nb = 0;
        if (tk) {
          const uint32_t dm1 = (tk & 0xFFFFu) - 1;
          const uint32_t le = lens[len], de = dists[dm1 < 256 ? dm1 : 256 + (dm1 >> 7)];
          const uint32_t dn = (de >> 16) & 15u, dx = de >> 20;
          a = le & 0xFFFFFFu;
          na = le >> 24;
          b = (de & 0xFFFFu) | ((dm1 & ((1u << dx) - 1u)) << dn);
          nb = dn + dx;
        } else if (i < t.len && end <= i) {
          const uint32_t c = code[by4[k]];
          a = c & 0xFFFFu;
          na = c >> 16;
        }
        if (heads) cover = __shfl_sync(kAll, i + len, 31 - __clz(heads));
        emit(a, na, b, nb);
      }
    }
  };
  uint32_t mine = 0;
  walk([&](uint32_t, uint32_t na, uint32_t, uint32_t nb) { mine += na + nb; });
  mine = __reduce_add_sync(kAll, mine);
  if (lane == 0) warp_bits[wid] = mine;
  __syncthreads();
  uint32_t cursor = 0, total = 0;
  for (uint32_t k = 0; k < kWarps; ++k) {
    if (k < wid) cursor += warp_bits[k];
    total += warp_bits[k];
  }
  auto put = [&](uint32_t bp, uint32_t v, uint32_t n) {
    if (!n) return;
    atomicOr(&buf[bp >> 5], v << (bp & 31));
    if ((bp & 31) + n > 32) atomicOr(&buf[(bp >> 5) + 1], v >> (32 - (bp & 31)));
  };
  walk([&](uint32_t a, uint32_t na, uint32_t b, uint32_t nb) {
    uint32_t incl = na + nb;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t x = __shfl_up_sync(kAll, incl, s);
      if (lane >= uint32_t(s)) incl += x;
    }
    const uint32_t bp = cursor + incl - na - nb;
    put(bp, a, na);
    put(bp + na, b, nb);
    cursor += __shfl_sync(kAll, incl, 31);
  });
  __syncthreads();
  uint32_t* out = reinterpret_cast<uint32_t*>(wk.scratch + t.scratch);
  for (uint32_t k = tid; k < (total + 31) / 32; k += N) out[k] = buf[k];
  if (tid == 0) {
    tp->spec_bits = total;
    tp->spec_exit = t.start + t.len;
  }
}

int launch_lazy(const Work& wk, const LazyLists& L, cudaStream_t st, int sms, Marks* mk) {
  if (!L.n_tiles) return 0;
  static std::atomic<bool> attr_set[64];
  const int ds = device_slot();
  if (!attr_set[ds].load(std::memory_order_relaxed)) {
    constexpr auto kMaxSmem = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (cudaFuncSetAttribute(k_link, kMaxSmem, int(sizeof(LinkSmem))) == cudaSuccess &&
        cudaFuncSetAttribute(k_search, kMaxSmem, int(kSearchSmem)) == cudaSuccess)
      attr_set[ds].store(true, std::memory_order_relaxed);
  }
  launch_after(k_link, L.n_runs, 1024, sizeof(LinkSmem), st, wk, L.runs, L.n_runs);
  launch_after(k_search, L.n_groups, kSearchThreads, kSearchSmem, st, wk, L.groups, L.n_groups);
  // Where all tiles' CTAs run at once, their latency counts and they are larger.
  // k_lparse of 128 / 512 threads (us): one tile of text 31 / 15, 1 MiB 41 / 20,
  // 2 MiB (508 tiles) 42 / 26, 3 MiB 50 / 61, 64 MiB 412 / 712; k_enc of 256 / 512:
  // one tile 24 / 16, 1 MiB 27 / 22, 2 MiB 33 / 36, 64 MiB 382 / 483.
  const bool few = L.n_tiles <= 4 * uint32_t(sms), few_enc = L.n_tiles <= 2 * uint32_t(sms);
  if (L.any_lazy)
    few ? launch_after(k_lparse<false, 512>, L.n_tiles, 512, 0, st, wk, L.tiles, L.n_tiles)
        : launch_after(k_lparse<false, 128>, L.n_tiles, 128, 0, st, wk, L.tiles, L.n_tiles);
  if (L.any_opt)
    few ? launch_after(k_lparse<true, 512>, L.n_tiles, 512, 0, st, wk, L.tiles, L.n_tiles)
        : launch_after(k_lparse<true, 128>, L.n_tiles, 128, 0, st, wk, L.tiles, L.n_tiles);
  mk->mark(kPhLazyLz, st);
  launch_after(k_huff, L.n_segs, kHuffThreads, 0, st, wk, L.segs, L.n_segs);
  mk->mark(kPhLazyHuff, st);
  few_enc ? launch_after(k_enc<512>, L.n_tiles, 512, 0, st, wk, L.tiles, L.n_tiles)
          : launch_after(k_enc<256>, L.n_tiles, 256, 0, st, wk, L.tiles, L.n_tiles);
  mk->mark(kPhLazyEnc, st);
  return 4 + (L.any_lazy ? 1 : 0) + (L.any_opt ? 1 : 0);
}

}  // namespace orotb
