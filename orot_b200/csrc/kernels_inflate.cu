// kernels_inflate.cu -- DEFLATE decoding (RFC 1951) on sm_100a.
//
// Decoding a DEFLATE stream is sequential by its definition: a code's length
// is known only after the code before it is decoded, and a match copies bytes
// that earlier tokens produced.  One CTA decodes one stream (CTAs take streams
// from a counter, largest first; many short streams go to small CTAs), and both
// chains are broken up inside it:
//
//   synchronisation  A window of the stream is cut into parts of kPartBits,
//            one per thread.  Every thread decodes its part from a guessed
//            start (the part's first bit) to the first token that starts
//            beyond it, marking the token starts in a bitmap.  Huffman codes
//            mostly synchronise themselves: after a few tokens a wrong start
//            leads to the same token starts as the right one.  Then each thread
//            compares its start with the end its left neighbour found and, if
//            they differ, decodes again until it meets a token start it had
//            marked, until no thread's start changes; the first part's start is
//            right, so then all are.  Where all codes have one length that does
//            not divide a part, a wrong start stays wrong and the right one moves
//            on by a part a round (1 MiB of literals in codes of 7 bits: 16 ms,
//            in codes of 8 bits 0.4).
//   tokens   The bitmap's tokens are dealt out evenly and decoded independently
//            (kBatch at a time); output offsets come from a scan of their
//            lengths.
//   expansion  For a piece of up to kPiece output bytes the tokens set a bit
//            at their first byte and beside it the literal or the distance.
//            Every output byte finds its token by the nearest bit and becomes a
//            byte value (a literal, or a byte before the piece) or the index of
//            the byte of the piece it copies.
//   copies   Indices are followed by pointer doubling (value = value[value])
//            until all are bytes: as many rounds as the logarithm of the
//            longest chain of matches that copy from matches.
//
// Tables are looked up by 12 bits (literal/length) and 11 (distance), 10 and 8 in small CTAs; their
// entries carry all a token needs (code bits, base value, extra bits).  Longer codes are resolved by the canonical
// rule of RFC 1951 3.2.2 (codes of one length are consecutive integers and
// shorter codes precede longer ones): left-aligned, a code is below the end of
// its length's range and of no shorter one's.
// The code lengths of a dynamic block are read by one warp, 32 bit offsets at a
// time (one thread took 16 to 32 thousand cycles a block).
//
// Bound by latency: the dependent steps of a token (two table lookups in shared
// memory, shifts) times the tokens of a part times the rounds of
// synchronisation, and the lookups, history reads and barriers of a piece; so
// the CTA is as large as can be and parts are short.  1 MiB streams of zlib
// level 6 on a B200, against one warp per stream that decoded 64 bit offsets
// at a time and followed the tokens one by one (whole deflate_decompress call,
// ms): text 67.5 -> 1.9, integers (39 blocks) 3.7, 8-byte periods 1.0, zeros 0.9.
// One exit test per token and 16 consecutive bytes a thread when bytes are
// coded took the text from 2.14 to 2.03, indices reduced only where a match
// overlaps itself to 1.97, code lengths read by a warp to 1.94, tables filled by
// comparing with the ends of the lengths' ranges (held in registers) to 1.92.
// 512 threads with parts of 480 bits take 2.7 on the text, 1024 threads with
// parts of 480 bits 2.2.
// A stream of short blocks pays for each block, not for what lies behind it:
// words stay staged, the fixed code's tables stay, and the first window of a
// block is about twice the longer of the two before (1 MiB of text in blocks of 100 bytes
// each behind a flush: 717 ms with whole windows staged and decoded, now 366;
// with the fixed code 437 and 193; one warp per stream took 489 and 324).
//
// The kernel does not read the zlib / gzip framing; the host strips it and
// checks the trailer against a checksum of the output (src/formats/*:
// zlib_decompress, gzip_decompress semantics).
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>
#include "engine.cuh"
#include "kernels.cuh"

namespace orotb {

namespace {

constexpr uint32_t kAll = 0xFFFFFFFFu;
// A CTA of N threads, with tables looked up by LIT and DIST bits.
template <int N, int LIT, int DIST>
struct Inf {
  static constexpr uint32_t kThreads = N;
  // Parts of the stream per window, decoded by a thread each.  An odd number of
  // words: threads at the same place of their parts read different banks.
  static constexpr uint32_t kParts = N, kPartBits = 9 * 32;
  static constexpr uint32_t kMapWords = kParts * kPartBits / 32;
  static constexpr uint32_t kWindowWords = kMapWords + 6;  // with the bits a last token reaches past the window
  static constexpr uint32_t kBatch = 8 * N;                // tokens decoded at once
  static constexpr uint32_t kPiece = 16 * N;               // output bytes expanded at once
  static constexpr int kLitBits = LIT, kDistBits = DIST;   // table index bits
};
using InfLarge = Inf<1024, 12, 11>;  // one CTA per SM
// For many short streams (large_streams): 22 KB, eight CTAs per SM by their
// registers.  10,000 streams of 100 bytes / of 1 to 4 KiB verified, with 128
// threads and 10 + 8 bits 2.08 / 2.58 ms, 11 + 9 bits 2.13 / 2.63, 256 threads 2.28 /
// 2.76, 64 threads and 9 + 8 bits 2.03 / 2.60 (and 35% slower on streams of 64 KiB).
using InfSmall = Inf<128, 10, 8>;
constexpr uint32_t kOverBits = 48 + 96;           // a token, and what is loaded for the one behind it
constexpr uint32_t kHeaderBits = 4608 + 96;       // a dynamic block's header (3 + 14 + 19 * 3 + 316 * 14), and the same
constexpr int kClBits = 7;                        // table index bits of the code-length code

// order of the code-length code lengths in a dynamic block header (3.2.7)
__constant__ uint8_t c_cl_order[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

// Lookup-table entries (0: the code is longer than the table's index or not assigned).
//   code-length code: [0,4) code bits, [16,32) symbol
//   literal/length:   [0,4) code bits, [4,6) kind (0 literal, 1 length,
//                     2 end of block, 3 symbol 286/287), [6,11) code + extra
//                     bits, [11,14) extra bits, [16,32) literal or base length
//   distance:         [0,4) code bits, [4,8) extra bits, [8,13) code + extra
//                     bits, bit 15 symbol 30/31, [16,32) base distance
enum : uint32_t { kTabCl = 0, kTabLit = 1, kTabDist = 2 };

// Base values and extra bits by the rule behind RFC 1951 3.2.5's tables: from
// the 9th length on, four codes share a number of extra bits (the last length
// has none); from the 5th distance on, two do.
__device__ __forceinline__ uint32_t make_entry(uint32_t tab, uint32_t s, uint32_t n) {
  if (tab == kTabCl) return n | (s << 16);
  if (tab == kTabLit) {
    if (s < 256) return n | (n << 6) | (s << 16);
    if (s == 256) return n | (2u << 4) | (n << 6);
    if (s > 285) return n | (3u << 4) | (n << 6);
    const uint32_t i = s - 257;
    const uint32_t x = i < 8 || i == 28 ? 0u : (i >> 2) - 1;
    const uint32_t base = i < 8 ? 3 + i : i == 28 ? 258u : ((4 + (i & 3)) << x) + 3;
    return n | (1u << 4) | ((n + x) << 6) | (x << 11) | (base << 16);
  }
  if (s > 29) return n | 0x8000u;
  const uint32_t x = s < 4 ? 0u : (s >> 1) - 1;
  const uint32_t base = s < 4 ? s + 1 : ((2 + (s & 1)) << x) + 1;
  return n | (x << 4) | ((n + x) << 8) | (base << 16);
}

// One Huffman code: per length the first code, the number of codes and the
// index of the first symbol; the symbols in code order; `end` is the end of the
// length's codes, left-aligned to 15 bits.
struct Canon {
  uint32_t first[16], count[16], offs[16], end[16];
  uint16_t sym[288];
};

template <class C>
struct InfSmem {
  uint32_t lit[1 << C::kLitBits], dist[1 << C::kDistBits];  // the lit table holds the code-length code first
  uint32_t words[C::kWindowWords];         // the stream from the window's first word
  alignas(16) uint32_t map[C::kMapWords];  // token starts, by bit of the window
  union alignas(16) {
    uint32_t list[C::kBatch];  // bit positions of a batch's tokens
    // a piece's bytes: at a token's first byte its code, then the codes below
    uint16_t value[C::kPiece];
  };
  uint32_t bits[C::kPiece / 32];     // first bytes of tokens
  uint16_t last[C::kPiece / 32];     // the last first byte before each bitmap word
  uint32_t end[C::kParts];           // where a part's last token ends, from the window's first bit | flags
  uint32_t scan[C::kThreads / 32];
  Canon lc, dc;
  uint32_t groups[10][16];           // build: codes of each length per 32 symbols
  uint8_t lens[320], raw[320];       // code lengths: literal/length at 0, distance at 288; as read
  uint32_t job, type, bad, used, stop;
  uint64_t staged;                   // the stream's word at words[0]
  uint64_t block_at;                 // the block's first bit behind its header
  uint32_t parts[2];                 // twice the sizes of the last two blocks
  static_assert(C::kParts * C::kPartBits + kOverBits + 31 <= C::kWindowWords * 32 && kHeaderBits + 31 <= C::kWindowWords * 32,
                "a window fits from any bit of its first word");
};
// Codes of a piece's bytes: at a token's start kDone | literal or kMatch |
// distance - 1; then kDone | byte, kBefore | bytes before the piece - 1, or an index (kHistory: in registers only).
constexpr uint32_t kMatch = 0x8000u, kBefore = 0x8000u, kDone = 0x4000u, kHistory = 0x10000u;
constexpr uint32_t kEndBlock = 1u << 30, kEndBad = 1u << 31, kEndFlags = kEndBlock | kEndBad;
static_assert(InfLarge::kPiece <= kDone, "indices leave the flag bits free");
static_assert(sizeof(InfSmem<InfLarge>) <= 227 * 1024, "one CTA per SM");

// Aligned input word j of a stream whose last bit is at absolute bit `endb`
// (bits at or past it read as zero).
__device__ __forceinline__ uint32_t word_at(const uint32_t* a, uint64_t j, uint64_t endb) {
  const uint64_t b0 = j * 32;
  if (b0 >= endb) return 0;
  uint32_t v = __ldg(a + j);
  if (endb - b0 < 32) v &= (1u << uint32_t(endb - b0)) - 1u;
  return v;
}

// Table entry of the code at the low bits of `w`, one of more than `nbits` bits
// or not assigned (then 0).
__device__ __forceinline__ uint32_t long_code(const Canon& c, uint32_t w, uint32_t nbits, uint32_t tab) {
  const uint32_t code = __brev(w) >> 17;  // 15 bits, first bit on top
  for (uint32_t l = nbits + 1; l < 16; ++l)
    if (code < c.end[l]) return make_entry(tab, c.sym[(code >> (15 - l)) - c.first[l] + c.offs[l]], l);
  return 0;
}

// The token at bit `at` of the staged words: its kind (0 literal, 1 match, 2
// end of block, 3 invalid), with the literal or length in `len` and the
// distance in `dist`; returns its bits.  Both lookups are made for every kind,
// so that lanes with literals and with matches stay together.
template <class C>
__device__ __forceinline__ uint32_t token_at(const InfSmem<C>& S, uint32_t at, uint32_t& kind, uint32_t& len,
                                             uint32_t& dist) {
  constexpr int kLitBits = C::kLitBits, kDistBits = C::kDistBits;
  const uint32_t* sw = S.words + (at >> 5);
  const uint32_t x0 = sw[0], x1 = sw[1], x2 = sw[2];
  const uint32_t w = __funnelshift_r(x0, x1, at & 31u), whi = __funnelshift_r(x1, x2, at & 31u);
  uint32_t e = S.lit[w & ((1u << kLitBits) - 1)];
  if (!e) {
    e = long_code(S.lc, w, kLitBits, kTabLit);
    if (!e) e = 3u << 4;
  }
  const uint32_t tot = (e >> 6) & 31u;
  kind = (e >> 4) & 3u;
  len = (e >> 16) + ((w >> (e & 15u)) & ((1u << ((e >> 11) & 7u)) - 1u));
  const uint32_t w2 = __funnelshift_r(w, whi, tot);
  uint32_t d = S.dist[w2 & ((1u << kDistBits) - 1)];
  if (kind == 1 && !d) d = long_code(S.dc, w2, kDistBits, kTabDist);
  if (kind == 1 && (!d || (d & 0x8000u))) kind = 3;
  dist = (d >> 16) + ((w2 >> (d & 15u)) & ((1u << ((d >> 4) & 15u)) - 1u));
  return tot + (kind == 1 ? (d >> 8) & 31u : 0u);
}

// Exclusive scan over the CTA of `v`; the sum over all threads in `total`.
// Every thread calls it; the CTA has passed a barrier since the last call.
template <class C>
__device__ __forceinline__ uint32_t cta_scan(InfSmem<C>& S, uint32_t v, uint32_t& total) {
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const uint32_t t = __shfl_up_sync(kAll, incl, k);
    if (lane >= uint32_t(k)) incl += t;
  }
  if (lane == 31) S.scan[wid] = incl;
  __syncthreads();
  const uint32_t w = lane < C::kThreads / 32 ? S.scan[lane] : 0u;
  const uint32_t below = __reduce_add_sync(kAll, lane < wid ? w : 0u);
  total = __reduce_add_sync(kAll, w);
  return below + incl - v;
}

// Builds the canonical code and the lookup table of 1 << nbits entries from
// code lengths lens[0..n), n <= 320 (all threads).  Returns false for an
// over-subscribed set of lengths; an incomplete set is accepted (a code that
// is not assigned is reported when it is read).
template <class C>
__device__ bool build_code(InfSmem<C>& S, Canon& c, const uint8_t* lens, uint32_t n, uint32_t* table, uint32_t nbits,
                           uint32_t tab) {
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  constexpr uint32_t N = C::kThreads, K = (320 + N - 1) / N;  // symbols of a thread
  uint32_t len[K], before[K];
  for (uint32_t i = tid; i < 160; i += N) S.groups[i >> 4][i & 15] = 0;
  __syncthreads();
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) {
    const uint32_t s = tid + j * N;
    len[j] = s < n ? lens[s] : 0u;
    uint32_t peers = kAll;  // lanes of the same length
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t bal = __ballot_sync(kAll, (len[j] >> k) & 1u);
      peers &= (len[j] >> k) & 1u ? bal : ~bal;
    }
    before[j] = __popc(peers & ((1u << lane) - 1));
    if (len[j] && !before[j]) S.groups[s >> 5][len[j]] = __popc(peers);
  }
  __syncthreads();
  if (tid < 16) {
    uint32_t sum = 0;
    for (int k = 0; k < 10; ++k) sum += S.groups[k][tid];
    c.count[tid] = sum;  // none of length 0: groups[.][0] stays 0
  }
  __syncthreads();
  if (tid == 0) {
    int left = 1;  // codes still available at the current length
    uint32_t bad = 0, code = 0, at = 0;
    c.first[0] = c.offs[0] = 0;
    for (int l = 1; l < 16; ++l) {
      left = (left << 1) - int(c.count[l]);
      if (left < 0) bad = 1;
      c.first[l] = code;
      c.offs[l] = at;
      c.end[l] = (code + c.count[l]) << (15 - l);
      code = (code + c.count[l]) << 1;
      at += c.count[l];
    }
    S.bad = bad;
  }
  __syncthreads();
  if (S.bad) return false;
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) {
    if (!len[j]) continue;
    const uint32_t s = tid + j * N;
    uint32_t r = before[j];
    for (uint32_t k = 0; k < s >> 5; ++k) r += S.groups[k][len[j]];
    c.sym[c.offs[len[j]] + r] = uint16_t(s);
  }
  __syncthreads();
  // every index finds its code: codes are sent most significant bit first, and
  // a code is below the end of its length's range and of no shorter one's
  constexpr uint32_t kLitBits = C::kLitBits;
  uint32_t end[kLitBits];
#pragma unroll
  for (uint32_t l = 0; l < kLitBits; ++l) end[l] = l < nbits ? c.end[l + 1] : 0u;
  for (uint32_t i = tid; i < (1u << nbits); i += N) {
    const uint32_t code = __brev(i) >> 17;
    uint32_t l = 1;
#pragma unroll
    for (uint32_t k = 0; k < kLitBits; ++k) l += k < nbits && code >= end[k] ? 1u : 0u;
    table[i] = l <= nbits ? make_entry(tab, c.sym[(code >> (15 - l)) - c.first[l] + c.offs[l]], l) : 0u;
  }
  __syncthreads();
  return true;
}

// Reads a dynamic block's code lengths, from bit `at` of the staged words (all
// threads; the first warp decodes).  Returns false for an invalid header; S.used is
// the bit after it.
template <class C>
__device__ bool read_lengths(InfSmem<C>& S, uint32_t at) {
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  constexpr uint32_t N = C::kThreads;
  auto bits_at = [&](uint32_t o) { return __funnelshift_r(S.words[o >> 5], S.words[(o >> 5) + 1], o & 31u); };
  const uint32_t h = bits_at(at);
  const uint32_t hlit = (h & 31u) + 257, hdist = ((h >> 5) & 31u) + 1, hclen = ((h >> 10) & 15u) + 4;
  at += 14;
  if (hlit > 286 || hdist > 30) return false;
  for (uint32_t i = tid; i < 320; i += N) S.raw[i] = 0;
  if (tid < 19) S.lens[c_cl_order[tid]] = tid < hclen ? uint8_t(bits_at(at + 3 * tid) & 7u) : uint8_t(0);
  at += 3 * hclen;
  __syncthreads();
  if (!build_code(S, S.lc, S.lens, 19, S.lit, kClBits, kTabCl)) return false;
  if (tid < 32) {
    const uint32_t n = hlit + hdist, lt = (1u << lane) - 1;
    uint32_t i = 0, prev = 0, err = 0;
    while (i < n) {
      // lane: the symbol at bit at + lane, its bits and how many lengths it gives
      const uint32_t w = bits_at(at + lane);
      const uint32_t e = S.lit[w & ((1u << kClBits) - 1)];  // every assigned code has at most 7 bits
      const uint32_t cb = e & 15u, sym = e >> 16;
      const uint32_t xb = sym < 16 ? 0u : sym == 16 ? 2u : sym == 17 ? 3u : 7u;
      const uint32_t rep = sym < 16 ? 1u : (sym == 18 ? 11u : 3u) + ((w >> cb) & ((1u << xb) - 1u));
      const uint32_t nb = cb + xb;
      // the symbols are the lanes reached from lane 0; one that is not a code
      // or leads out leads to itself
      uint32_t to = e && lane + nb < 32 ? lane + nb : lane, path = 1u << lane;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        path |= __shfl_sync(kAll, path, to);
        to = __shfl_sync(kAll, to, to);
      }
      path |= __shfl_sync(kAll, path, to);
      const bool mine = (__shfl_sync(kAll, path, 0) >> lane) & 1u;
      uint32_t incl = mine ? rep : 0u;
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const uint32_t t = __shfl_up_sync(kAll, incl, k);
        if (lane >= uint32_t(k)) incl += t;
      }
      const uint32_t first = i + incl - rep;  // index of the symbol's first length
      const bool real = mine && first < n;
      if (__any_sync(kAll, real && (!e || first + rep > n || (sym == 16 && first == 0)))) {
        err = 1;
        break;
      }
      const uint32_t set = __ballot_sync(kAll, real && sym != 16) & lt;  // symbols that give a value
      uint32_t v = sym < 16 ? sym : 0u;
      const uint32_t pv = __shfl_sync(kAll, v, set ? 31 - __clz(set) : 0);
      if (sym == 16) v = set ? pv : prev;
      if (real && v)  // the lengths are cleared
        for (uint32_t k = 0; k < rep; ++k) S.raw[first + k] = uint8_t(v);
      const uint32_t last = 31 - __clz(__ballot_sync(kAll, real));
      prev = __shfl_sync(kAll, v, last);
      i = __shfl_sync(kAll, first + rep, last);
      at += __shfl_sync(kAll, lane + nb, last);
    }
    if (lane == 0) {
      S.bad = err;
      S.used = at;
    }
  }
  __syncthreads();
  if (S.bad) return false;
  for (uint32_t i = tid; i < 320; i += N)
    S.lens[i] = i < 288 ? (i < hlit ? S.raw[i] : 0) : i - 288 < hdist ? S.raw[hlit + i - 288] : 0;
  __syncthreads();
  return S.lens[256] != 0;  // a block needs an end-of-block code
}

}  // namespace

// status: kInfOk, kInfData (corrupt), kInfOutput (output full), kInfInput (input exhausted)
template <class C>
__global__ void __launch_bounds__(C::kThreads, 1024 / C::kThreads) k_inflate(const uint8_t* __restrict__ in, uint8_t* out,
                                                            InflateJob* jobs, const uint32_t* __restrict__ order,
                                                            uint32_t njobs, uint32_t* counter) {
  extern __shared__ __align__(16) uint8_t inf_smem[];
  InfSmem<C>& S = *reinterpret_cast<InfSmem<C>*>(inf_smem);
  constexpr uint32_t N = C::kThreads, kParts = C::kParts, kPartBits = C::kPartBits, kWindowWords = C::kWindowWords;
  constexpr uint32_t kBatch = C::kBatch, kPiece = C::kPiece;
  constexpr int kLitBits = C::kLitBits, kDistBits = C::kDistBits;
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  bool fixed_tables = false;  // the tables are those of the fixed code
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      S.job = atomicAdd(counter, 1u);
      S.staged = uint64_t(1) << 63;  // none
      S.parts[0] = S.parts[1] = kParts;
    }
    __syncthreads();
    if (S.job >= njobs) break;
    InflateJob* jp = jobs + order[S.job];
    const InflateJob job = *jp;
    uint8_t* o = out + job.out_off;
    const uint8_t* base = in + job.in_off;
    // the stream as aligned words: its first bit is bit s0 of word 0
    const uint32_t* aw = reinterpret_cast<const uint32_t*>(reinterpret_cast<uint64_t>(base) & ~uint64_t(3));
    const uint64_t s0 = (reinterpret_cast<uint64_t>(base) & 3) * 8;
    const uint64_t endb = s0 + job.in_len * 8;
    uint64_t P = 0;   // bits consumed
    uint64_t op = 0;  // output position
    int32_t status = kInfOk;
    bool last = false;
    // stages the words from bit P on unless `bits` from there are staged;
    // returns the bit of P in the staged words
    auto stage = [&](uint32_t bits) -> uint32_t {
      const uint64_t q = (s0 + P) >> 5;
      const uint32_t r = uint32_t((s0 + P) & 31u);
      const uint64_t w = q - S.staged;
      __syncthreads();  // the words staged before are no longer read
      if (w < kWindowWords && uint32_t(w) * 32 + r + bits <= kWindowWords * 32) return uint32_t(w) * 32 + r;
      if (tid == 0) S.staged = q;
      for (uint32_t k = tid; k < kWindowWords; k += N) S.words[k] = word_at(aw, q + k, endb);
      __syncthreads();
      return r;
    };
    while (!last && status == kInfOk) {
      if (s0 + P + 3 > endb) { status = kInfInput; break; }
      const uint32_t r = stage(kHeaderBits);
      const uint32_t hdr = __funnelshift_r(S.words[r >> 5], S.words[(r >> 5) + 1], r & 31u);
      last = hdr & 1u;
      const uint32_t type = (hdr >> 1) & 3u;
      if (type == 3) { status = kInfData; break; }
      if (type == 0) {
        // stored: byte-align, LEN, NLEN, LEN raw bytes
        const uint64_t src = (P + 3 + 7) >> 3;
        if (src + 4 > job.in_len) { status = kInfInput; break; }
        const uint32_t len = base[src] | (uint32_t(base[src + 1]) << 8);
        const uint32_t inv = base[src + 2] | (uint32_t(base[src + 3]) << 8);
        if ((inv ^ 0xFFFFu) != len) { status = kInfData; break; }
        if (src + 4 + len > job.in_len) { status = kInfInput; break; }
        if (op + len > job.out_cap) { status = kInfOutput; break; }
        for (uint32_t i = tid; i < len; i += N) o[op + i] = base[src + 4 + i];
        op += len;
        P = (src + 4 + len) * 8;
        continue;
      }
      uint32_t used = r + 3;
      if (type == 1) {
        if (!fixed_tables) {
          for (uint32_t i = tid; i < 320; i += N) S.lens[i] = i < 144 ? 8 : i < 256 ? 9 : i < 280 ? 7 : i < 288 ? 8 : 5;
          __syncthreads();
        }
      } else {
        fixed_tables = false;
        if (!read_lengths(S, used)) { status = kInfData; break; }
        used = S.used;
      }
      if (!fixed_tables && (!build_code(S, S.lc, S.lens, 288, S.lit, kLitBits, kTabLit) ||
                            !build_code(S, S.dc, S.lens + 288, 30, S.dist, kDistBits, kTabDist))) {
        status = kInfData;
        break;
      }
      fixed_tables = type == 1;
      P += used - r;
      // What lies behind the block is decoded for nothing, so the window of a
      // block behind short ones starts at about twice the longer of the last two
      // (of the last alone: 12% slower where blocks of 100 bytes and of 60 KB alternate).
      if (tid == 0) S.block_at = P;
      uint32_t parts = max(S.parts[0], S.parts[1]);

      bool block_end = false;
      while (!block_end) {
        if (s0 + P >= endb) { status = kInfInput; break; }
        const uint32_t r0 = stage(parts * kPartBits + kOverBits);
        const uint64_t left = endb - (s0 + P);
        const uint32_t rem = left > (1u << 20) ? 1u << 20 : uint32_t(left);  // bits left, more than a window if capped
        // -- synchronisation
        const uint32_t limit = min(rem, (tid + 1) * kPartBits);  // tokens from here on are the next part's
        const bool active = tid < parts && tid * kPartBits < rem;
        uint32_t begin = tid * kPartBits;  // where this part's first token starts, as far as known
        // One test per token ends the inner loop; what it was is found behind it,
        // so that a token is little more than its chain of lookups.
        auto decode_part = [&](auto again) {
          uint32_t pos = begin, word = tid * (kPartBits / 32), bits = 0, flag = 0;
          while (pos < limit) {
            uint32_t e, d, nb, old = 0, next = pos;
            bool out;
            do {
              pos = next;
              const uint32_t here = pos >> 5, at = r0 + pos;
              const uint32_t* sw = S.words + (at >> 5);
              const uint32_t x0 = sw[0], x1 = sw[1], x2 = sw[2];
              if constexpr (decltype(again)::value) old = S.map[here] >> (pos & 31);
              const uint32_t w = __funnelshift_r(x0, x1, at & 31u), whi = __funnelshift_r(x1, x2, at & 31u);
              e = S.lit[w & ((1u << kLitBits) - 1)];
              // the map's words before this token's: at most one has no start (a token has at most 48 bits)
              if (here != word) S.map[word] = bits;
              if (here > word + 1) S.map[word + 1] = 0;
              bits = here != word ? 0u : bits;
              word = here;
              const uint32_t tot = (e >> 6) & 31u;
              d = S.dist[__funnelshift_r(w, whi, tot) & ((1u << kDistBits) - 1)];
              const bool match = (e & 0x30u) == 0x10u;
              nb = tot + (match ? (d >> 8) & 31u : 0u);
              next = pos + nb;
              // an end or invalid, a long code, the input's end, a start marked before
              out = !e || (e & 0x20u) || (match && (!d || (d & 0x8000u))) || next > rem || (old & 1u);
              if (!out) bits |= 1u << (pos & 31);
            } while (!out && next < limit);
            if (!out) {
              pos = next;
              break;
            }
            if (old & 1u) {  // from here on as before
              S.map[word] = bits | (S.map[word] & (kAll << (pos & 31)));
              return;
            }
            uint32_t kind, len, dist;
            next = pos + token_at(S, r0 + pos, kind, len, dist);
            if (kind >= 2 || next > rem) {
              flag = kind == 2 && next <= rem ? kEndBlock : kEndBad;
              pos = next;
              break;
            }
            bits |= 1u << (pos & 31);
            pos = next;
          }
          for (; word < (tid + 1) * (kPartBits / 32); ++word) {
            S.map[word] = bits;
            bits = 0;
          }
          S.end[tid] = pos | flag;
        };
        if (active) decode_part(std::false_type{});
        for (;;) {
          __syncthreads();
          const uint32_t e = tid && active ? S.end[tid - 1] : 0u;
          // behind a neighbour that met an end the start stays open
          const bool again = active && !(e & kEndFlags) && e != begin;
          if (!__syncthreads_or(again)) break;
          if (again) {
            begin = e;
            decode_part(std::true_type{});
          }
        }
        // -- the parts up to the first that met an end count
        if (tid == 0) S.stop = min(parts, (rem + kPartBits - 1) / kPartBits) - 1;
        __syncthreads();
        if (active && (S.end[tid] & kEndFlags)) atomicMin(&S.stop, tid);
        __syncthreads();
        const uint32_t stop = S.stop, stop_end = S.end[stop];
        if (stop_end & kEndBad) {
          // past the input's end only zero bits follow: more input was needed
          status = (stop_end & ~kEndFlags) > rem ? kInfInput : kInfData;
          break;
        }
        block_end = (stop_end & kEndBlock) != 0;
        P += stop_end & ~kEndFlags;
        parts = kParts;
        if (block_end && tid == 0) {
          S.parts[1] = S.parts[0];
          S.parts[0] = uint32_t(min(uint64_t(kParts), (P - S.block_at) / (kPartBits / 2) + 4));
        }

        // -- tokens, a batch at a time
        constexpr uint32_t kPartWords = kPartBits / 32;
        const uint32_t* pm = S.map + tid * kPartWords;
        uint32_t mine = 0;
        if (tid <= stop)
          for (uint32_t k = 0; k < kPartWords; ++k) mine += __popc(pm[k]);
        uint32_t ntok;
        const uint32_t first = cta_scan(S, mine, ntok);
        for (uint32_t t0 = 0; t0 < ntok; t0 += kBatch) {
          __syncthreads();  // the list's and the scan's places are free again
          if (mine && first < t0 + kBatch && first + mine > t0) {
            uint32_t i = first;
            for (uint32_t k = 0; k < kPartWords; ++k) {
              uint32_t m = pm[k];
              while (m) {
                if (i - t0 < kBatch) S.list[i - t0] = tid * kPartBits + k * 32 + __ffs(m) - 1;
                m &= m - 1;
                ++i;
              }
            }
          }
          if (tid == 0) S.bad = 0;
          __syncthreads();
          uint32_t tok[8];  // kMatch << 16 | length << 16 | distance - 1, or the literal; length 1 for it, 0: none
          uint32_t sum = 0;
          {
            // eight in a row each, so that a scan gives their places
            const uint4 la = reinterpret_cast<const uint4*>(S.list)[2 * tid], lb = reinterpret_cast<const uint4*>(S.list)[2 * tid + 1];
            const uint32_t at[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) {
              tok[q] = 0;
              if (t0 + tid * 8 + q < ntok) {
                uint32_t kind, len, dist;
                token_at(S, r0 + at[q], kind, len, dist);
                tok[q] = kind ? (kMatch << 16) | (len << 16) | (dist - 1) : (1u << 16) | len;
              }
              sum += (tok[q] >> 16) & 0x1FFu;
            }
          }
          uint32_t total;
          uint32_t off = cta_scan(S, sum, total);
          if (op + total > job.out_cap) { status = kInfOutput; break; }
          {
            uint32_t at = off;
            bool bad = false;  // a distance that reaches before the output
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) {
              bad |= (tok[q] >> 31) && op + at < (tok[q] & 0x7FFFu) + 1;
              at += (tok[q] >> 16) & 0x1FFu;
            }
            if (bad) S.bad = 1;
          }
          // -- expansion, a piece of the batch's output at a time
          for (uint32_t b0 = 0; b0 < total; b0 += kPiece) {
            const uint32_t n = min(kPiece, total - b0);
            if (tid < kPiece / 32) S.bits[tid] = 0;
            __syncthreads();
            if (S.bad) { status = kInfData; break; }
            {
              uint32_t at = off;
#pragma unroll
              for (uint32_t q = 0; q < 8; ++q) {
                const uint32_t len = (tok[q] >> 16) & 0x1FFu;
                if (at < b0 + n && at + len > b0) {  // a match cut by a piece's start goes on from there
                  const uint32_t j = max(at, b0) - b0;
                  S.value[j] = uint16_t(tok[q] >> 31 ? kMatch | (tok[q] & 0x7FFFu) : kDone | (tok[q] & 0xFFu));
                  atomicOr(&S.bits[j >> 5], 1u << (j & 31));
                }
                at += len;
              }
            }
            __syncthreads();
            // the last token start before each bitmap word
            {
              const uint32_t bm = tid < kPiece / 32 ? S.bits[tid] : 0u;
              uint32_t m = bm ? tid * 32 + 32 - __clz(bm) : 0u;  // + 1; 0: none
#pragma unroll
              for (int k = 1; k < 32; k <<= 1) {
                const uint32_t t = __shfl_up_sync(kAll, m, k);
                if (lane >= uint32_t(k)) m = max(m, t);
              }
              if (lane == 31) S.scan[wid] = m;
              __syncthreads();
              uint32_t prev = __shfl_up_sync(kAll, m, 1);
              if (lane == 0) prev = 0;
              prev = max(prev, __reduce_max_sync(kAll, lane < wid ? S.scan[lane] : 0u));
              if (tid < kPiece / 32) S.last[tid] = uint16_t(prev ? prev - 1 : 0);
            }
            __syncthreads();
            uint8_t* ob = out + job.out_off + op + b0;
            // every thread codes 16 bytes in a row: a literal, an index of the
            // piece, or how far before the piece the byte lies
            {
              const uint32_t j0 = tid * 16;
              const uint32_t starts = (S.bits[tid >> 1] >> ((tid & 1) * 16)) & 0xFFFFu;
              const uint32_t before = tid & 1 ? S.bits[tid >> 1] & 0xFFFFu : 0u;
              uint32_t s = before ? j0 - 16 + 31 - __clz(before) : S.last[tid >> 1];
              uint32_t e = S.value[s];
              const uint4 c0 = reinterpret_cast<const uint4*>(S.value)[2 * tid], c1 = reinterpret_cast<const uint4*>(S.value)[2 * tid + 1];
              const uint32_t cw[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
              __syncthreads();  // all codes are read
              uint32_t v[8];
#pragma unroll
              for (uint32_t k = 0; k < 16; ++k) {
                const uint32_t j = j0 + k;
                if ((starts >> k) & 1u) {
                  s = j;
                  e = k & 1 ? cw[k / 2] >> 16 : cw[k / 2] & 0xFFFFu;
                }
                int src = int(j) - 1 - int(e & 0x7FFFu);
                // a match that overlaps itself repeats its first d bytes (the
                // quotient is exact: it is below 258 and the half keeps it
                // away from whole numbers)
                if ((e & kMatch) && src >= int(s)) {
                  const uint32_t i = j - s, d = (e & 0x7FFFu) + 1;
                  src -= int(d * uint32_t(__fdividef(float(i) + 0.5f, float(d))));
                }
                const uint32_t x = !(e & kMatch) ? e : src >= 0 ? uint32_t(src) : kBefore | uint32_t(~src);
                v[k / 2] = k & 1 ? v[k / 2] | (x << 16) : x;
              }
              uint4* o4 = reinterpret_cast<uint4*>(S.value) + 2 * tid;
              o4[0] = make_uint4(v[0], v[1], v[2], v[3]);
              o4[1] = make_uint4(v[4], v[5], v[6], v[7]);
            }
            __syncthreads();
            // bytes before the piece, neighbours by neighbouring threads
            uint32_t open = 0;  // bytes of this thread (tid + k * N) that are not known yet
#pragma unroll
            for (uint32_t k0 = 0; k0 < 16; k0 += 8) {
              uint32_t v[8];
#pragma unroll
              for (uint32_t k = 0; k < 8; ++k) {
                const uint32_t j = tid + (k0 + k) * N;
                v[k] = j < n ? S.value[j] : kDone;
              }
#pragma unroll
              for (uint32_t k = 0; k < 8; ++k)
                if (v[k] & kBefore) v[k] = kHistory | ob[-1 - int(v[k] & 0x7FFFu)];
#pragma unroll
              for (uint32_t k = 0; k < 8; ++k) {
                const uint32_t j = tid + (k0 + k) * N;
                if (v[k] & kHistory) S.value[j] = uint16_t(kDone | (v[k] & 255u));
                else if (!(v[k] & kDone)) open |= 1u << (k0 + k);
              }
            }
            // -- copies: follow the indices until all are bytes, eight of a thread's at a time
            while (__syncthreads_or(open != 0)) {
#pragma unroll
              for (uint32_t k0 = 0; k0 < 16; k0 += 8) {
                if (!((open >> k0) & 0xFFu)) continue;
                uint32_t w[8];
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) w[k] = (open >> (k0 + k)) & 1u ? S.value[tid + (k0 + k) * N] : 0u;
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) w[k] = S.value[w[k]];
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) {
                  if (!((open >> (k0 + k)) & 1u)) continue;
                  S.value[tid + (k0 + k) * N] = uint16_t(w[k]);
                  if (w[k] & kDone) open &= ~(1u << (k0 + k));
                }
              }
            }
            for (uint32_t j = tid; j < n; j += N) ob[j] = uint8_t(S.value[j]);
            __syncthreads();
          }
          if (status != kInfOk) break;
          op += total;
        }
        if (status != kInfOk) break;
      }
    }
    if (tid == 0) {
      const uint64_t used = (P + 7) >> 3;
      if (status == kInfOk && used > job.in_len) status = kInfInput;
      jp->out_len = op;
      jp->in_used = status == kInfOk ? used : 0;
      jp->status = status;
    }
  }
}


// Compares decoded bytes with the original input, one warp per stream.
__global__ void __launch_bounds__(256) k_inflate_compare(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b,
                                                         InflateJob* jobs, const uint64_t* __restrict__ ref_off,
                                                         const uint64_t* __restrict__ ref_len, uint32_t njobs) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (j >= njobs) return;
  InflateJob job = jobs[j];
  if (job.status != kInfOk) return;
  bool same = job.out_len == ref_len[j];
  if (same) {
    const uint8_t* x = a + job.out_off;
    const uint8_t* y = b + ref_off[j];
    for (uint64_t i = lane; i < job.out_len && same; i += 32) same = x[i] == y[i];
  }
  same = __all_sync(kAll, same);
  if (lane == 0 && !same) jobs[j].status = kInfMismatch;
}

// Framing of compressed streams (one thread per stream): zlib 78 9C header and
// big-endian Adler-32 trailer, gzip 1F 8B 08 header, little-endian CRC-32 and
// ISIZE; the trailer must carry the stream's checksum and length.
__global__ void k_frame_check(const uint8_t* __restrict__ out, const Stream* __restrict__ st, InflateJob* jobs,
                              uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Stream s = st[i];
  if (s.error || jobs[i].status != kInfOk || s.fmt == kFmtRaw) return;
  const uint8_t* o = out + s.out_off;
  const uint8_t* t = o + s.out_size;
  bool good;
  if (s.fmt == kFmtZlib) {
    const uint32_t a = (uint32_t(t[-4]) << 24) | (uint32_t(t[-3]) << 16) | (uint32_t(t[-2]) << 8) | t[-1];
    good = o[0] == 0x78 && o[1] == 0x9C && a == s.checksum;
  } else {
    const uint32_t c = uint32_t(t[-8]) | (uint32_t(t[-7]) << 8) | (uint32_t(t[-6]) << 16) | (uint32_t(t[-5]) << 24);
    const uint32_t z = uint32_t(t[-4]) | (uint32_t(t[-3]) << 8) | (uint32_t(t[-2]) << 16) | (uint32_t(t[-1]) << 24);
    good = o[0] == 0x1F && o[1] == 0x8B && o[2] == 8 && c == s.checksum && z == uint32_t(s.in_len);
  }
  if (!good) jobs[i].status = kInfMismatch;
}

void launch_frame_check(const uint8_t* out, const Stream* streams, InflateJob* jobs, uint32_t n, cudaStream_t st) {
  if (n) k_frame_check<<<(n + 255) / 256, 256, 0, st>>>(out, streams, jobs, n);
}

template <class C>
static void launch_inflate_t(const uint8_t* in, uint8_t* out, InflateJob* jobs, const uint32_t* order, uint32_t njobs,
                             uint32_t* counter, int sms, cudaStream_t st) {
  if (!njobs) return;
  static std::atomic<int> ctas_per_sm[64];
  const int ds = device_slot();
  int per_sm = ctas_per_sm[ds].load(std::memory_order_relaxed);
  if (!per_sm) {
    cudaFuncSetAttribute(k_inflate<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(InfSmem<C>)));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_inflate<C>, C::kThreads, sizeof(InfSmem<C>));
    if (per_sm < 1) per_sm = 1;
    ctas_per_sm[ds].store(per_sm, std::memory_order_relaxed);
  }
  const uint32_t most = uint32_t(sms) * uint32_t(per_sm), blocks = njobs < most ? njobs : most;
  k_inflate<C><<<blocks, C::kThreads, sizeof(InfSmem<C>), st>>>(in, out, jobs, order, njobs, counter);
}

void launch_inflate(const uint8_t* in, uint8_t* out, InflateJob* jobs, const uint32_t* order, uint32_t njobs,
                    uint32_t nlarge, uint32_t* counters, int sms, cudaStream_t st) {
  if (!njobs) return;
  cudaMemsetAsync(counters, 0, 8, st);
  launch_inflate_t<InfLarge>(in, out, jobs, order, nlarge, counters, sms, st);
  launch_inflate_t<InfSmall>(in, out, jobs, order + nlarge, njobs - nlarge, counters + 1, sms, st);
}

void launch_inflate_compare(const uint8_t* decoded, const uint8_t* ref, InflateJob* jobs, const uint64_t* ref_off,
                            const uint64_t* ref_len, uint32_t njobs, cudaStream_t st) {
  if (!njobs) return;
  k_inflate_compare<<<(njobs + 7) / 8, 256, 0, st>>>(decoded, ref, jobs, ref_off, ref_len, njobs);
}

}  // namespace orotb
