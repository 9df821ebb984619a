// kernels_common.cu -- block planning, output assembly and checksums.
//
//   k_plan_*    block type of every segment (the reference's rules,
//               src/deflate/deflate_block.cpp:389-474 and
//               src/compress/block_compressor.cpp:53-63), bit offset of every
//               block, and the list of bit-range copies that assemble the
//               stream; output size and capacity check (one warp per segment
//               or stream, see below).
//   k_ck_block  CRC-32 (slicing-by-4) and Adler-32 partial sums of 64 KiB
//               blocks, 256 bytes per thread, folded with the GF(2) shift /
//               Adler weight identities.
//   k_ck_fold   folds the blocks of each stream: runs of blocks per thread,
//               then a tree over the runs (one CTA per stream); writes the zlib
//               / gzip header and trailer bytes.
//   k_join      one warp per copy: funnel-shifted 32-bit words, plain stores
//               inside a copy, atomicOr on the two boundary words it shares.
#include <cuda_runtime.h>
#include <algorithm>
#include <mutex>
#include <cstdint>
#include "engine.cuh"
#include "deflate_device.cuh"
#include "kernels.cuh"

namespace orotb {

constexpr uint32_t kFullMask = 0xFFFFFFFFu;

__host__ __device__ inline uint32_t fmt_header_bytes(uint32_t fmt) { return fmt == kFmtZlib ? 2 : fmt == kFmtGzip ? 10 : 0; }
__host__ __device__ inline uint32_t fmt_trailer_bytes(uint32_t fmt) { return fmt == kFmtZlib ? 4 : fmt == kFmtGzip ? 8 : 0; }

// ---------------------------------------------------------------- planning
// Three kernels, so that a stream of thousands of segments (a pigz-style
// stream) or a segment of thousands of tiles (a large whole buffer) is
// planned in parallel:
//   k_plan_seg     one warp or CTA per segment: token bits and matches summed over
//                  its tiles, the block type, and the block's length when it
//                  does not depend on its bit alignment (Huffman blocks).
//   k_plan_stream  one warp per stream: block offsets in order (32 segments
//                  at a time; a stored block's padding depends on where
//                  it starts), stream size,
//                  capacity check, the closing sync point of an open part.
//   k_plan_pieces  one warp or CTA per segment: its bit-range copies, at slots the
//                  host reserved for the segment (Segment::piece_off); unused
//                  slots are left empty (nbits 0).  More CTAs clear the words
//                  the streams will occupy.

// Bits a stored block of `len` bytes starting at bit c occupies: per piece of
// at most 65535 bytes, 3 header bits, padding to a byte, LEN/NLEN and the
// bytes (deflate_block.cpp:107-132).
__device__ __forceinline__ uint64_t stored_bits_at(uint64_t c, uint32_t len) {
  const uint64_t pieces = len ? (uint64_t(len) + 65534) / 65535 : 1;
  return (((c + 3 + 7) & ~uint64_t(7)) - c) + 32 + uint64_t(len) * 8 + (pieces - 1) * 40;
}

// Warps per segment of k_plan_seg and k_plan_pieces (WPS): 8, a CTA, where the
// segments are too few to fill the chip by themselves, since a warp goes through
// 32 tiles per memory latency (16 MiB in one segment of 2,048 tiles: 29 and 66 us,
// with 8 warps 9 and 20); else 1.
constexpr uint32_t kPlanCtaSegs = 1024;

// Sum over the threads of a segment (32 * WPS of them).
template <int WPS>
__device__ __forceinline__ unsigned long long seg_sum(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
  if constexpr (WPS > 1) {
    __shared__ unsigned long long part[WPS];
    __syncthreads();  // the sum before has been read
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0;
#pragma unroll
    for (int k = 0; k < WPS; ++k) v += part[k];
  }
  return v;
}

template <int WPS>
__global__ void __launch_bounds__(256) k_plan_seg(Work wk) {
  begin_kernel();
  const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) / (32 * WPS), lane = threadIdx.x % (32 * WPS);
  if (g >= wk.nsegs) return;
  const Segment sg = wk.segs[g];
  unsigned long long tok = 0, matches = 0;
  if (sg.level > 0) {
    for (uint32_t t = sg.tile_first + lane; t < sg.tile_first + sg.tile_count; t += 32 * WPS) {
      const Tile& tl = wk.tiles[t];
      tok += uint64_t(tl.fix_bits) + (tl.spec_bits - tl.splice_bit);
      matches += tl.fin_matches;
    }
  }
  tok = seg_sum<WPS>(tok);
  matches = seg_sum<WPS>(matches);
  if (lane) return;
  uint32_t type = kBlkStored;
  uint64_t bits = 0;
  if (sg.level > 0) {
    if (sg.level >= 4) {
      type = sg.block_type;  // chosen by the lazy pipeline
    } else if ((sg.flags & kSegWholeBuf) && matches == 0) {
      type = kBlkStored;     // all-literal parse (block_compressor.cpp:60-61)
    } else {
      const uint64_t fixed_bits = 3 + tok + 7;      // header + tokens + EOB
      const uint64_t stored = (uint64_t(sg.len) + 5) * 8;
      type = stored <= fixed_bits ? kBlkStored : kBlkFixed;
    }
  }
  if (type == kBlkFixed) bits = 3 + tok + 7;                       // EOB is code 0000000
  else if (type == kBlkDynamic) bits = 3 + sg.hdr_bits + tok + (sg.eob >> 16);
  wk.segs[g].block_type = type;
  wk.segs[g].bits = bits;
}

__global__ void k_plan_stream(Work wk) {
  begin_kernel();
  const uint32_t si = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (si >= wk.nstreams) return;
  Stream s = wk.streams[si];
  const bool bare = (s.mode & kStreamBare) != 0;
  const uint32_t hdr = bare ? 0 : fmt_header_bytes(s.fmt), trl = bare ? 0 : fmt_trailer_bytes(s.fmt);
  uint64_t c = 0;  // bits from the start of the raw DEFLATE stream
  bool fault = false;  // a kernel could not finish one of the stream's segments
  // 32 segments at once, the next 32 loaded ahead.  A coded block's length is
  // known; a stored one's depends on the bit it starts at within a byte, and it
  // ends on a byte.  So the bits since the last stored block give each block
  // its phase, that its length, and those the offsets.  One segment after the
  // other took 50 us for 512 segments, now 14.
  struct Row {
    uint32_t type, len, flags;
    uint64_t bits;
  };
  const uint32_t g_end = s.seg_first + s.seg_count;
  auto load = [&](uint32_t g) {
    Row r{kBlkFixed, 0, 0, 0};
    if (g < g_end) {
      const Segment& sg = wk.segs[g];
      r = Row{sg.block_type, sg.len, sg.flags, sg.bits};
    }
    return r;
  };
  Row next = load(s.seg_first + lane);
  for (uint32_t g0 = s.seg_first; g0 < g_end; g0 += 32) {
    const Row r = next;
    next = load(g0 + 32 + lane);
    if (r.flags & kSegFault) fault = true;
    const bool stored = r.type == kBlkStored;
    const uint32_t before = __ballot_sync(kFullMask, stored) & ((1u << lane) - 1);
    uint32_t x = stored ? 0u : uint32_t(r.bits) & 7u;
    const uint32_t own = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kFullMask, x, o);
      if (lane >= uint32_t(o)) x += v;
    }
    const uint32_t since = __shfl_sync(kFullMask, x, before ? 31 - __clz(before) : 0);
    const uint32_t phase = (before ? x - own - since : uint32_t(c) + x - own) & 7u;
    uint64_t n = stored ? stored_bits_at(phase, r.len) : r.bits;
    if (r.flags & kSegLast) n += (8 - (phase + uint32_t(n))) & 7u;
    uint64_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t v = __shfl_up_sync(kFullMask, incl, o);
      if (lane >= uint32_t(o)) incl += v;
    }
    if (g0 + lane < g_end) {
      wk.segs[g0 + lane].bit_off = c + incl - n;
      wk.segs[g0 + lane].bits = n;
    }
    c += __shfl_sync(kFullMask, incl, 31);
  }
  fault = __any_sync(kFullMask, fault);
  if (lane) return;
  Piece* tail = wk.pieces + s.piece_first + s.piece_count - 2;  // the open part's sync point
  const uint64_t sync_at = c;
  if (s.mode & kStreamOpen) c = ((c + 3 + 7) & ~uint64_t(7)) + 32;  // empty stored block, BFINAL = 0
  const uint64_t size = uint64_t(hdr) + c / 8 + trl;
  s.raw_bits = c;
  s.error = fault ? kErrInternal : size > s.out_cap ? kErrCapacity : kErrNone;
  s.out_size = s.error ? 0 : size;
  if (s.mode & kStreamOpen) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(wk.out + s.out_off);
    const uint64_t base = uint64_t(hdr) * 8;
    tail[0] = Piece{nullptr, dst, 0, base + sync_at, s.error ? 0u : 3u, 0u};
    tail[1] = Piece{nullptr, dst, 0, base + ((sync_at + 3 + 7) & ~uint64_t(7)), s.error ? 0u : 32u, 0xFFFF0000u};
  }
  wk.streams[si] = s;
}

// Clears the words stream si will occupy (the join ORs boundary words), part
// `part` of `parts`, so that one large stream is cleared by many CTAs.
__device__ __forceinline__ void clear_output(const Work& wk, uint32_t si, uint32_t part, uint32_t parts) {
  const Stream& s = wk.streams[si];
  if (s.error) return;
  uint4* o = reinterpret_cast<uint4*>(wk.out + s.out_off);
  const uint64_t n16 = (s.out_size + 15) / 16;
  const uint64_t per = (n16 + parts - 1) / parts;
  const uint64_t b = per * part, e = min(n16, b + per);
  for (uint64_t i = b + threadIdx.x; i < e; i += blockDim.x) o[i] = make_uint4(0, 0, 0, 0);
}

// The CTAs after those of the segments clear the streams' words.
template <int WPS>
__global__ void __launch_bounds__(256) k_plan_pieces(Work wk, uint32_t seg_ctas, uint32_t parts) {
  begin_kernel();
  if (blockIdx.x >= seg_ctas) {
    const uint32_t x = blockIdx.x - seg_ctas;
    clear_output(wk, x / parts, x % parts, parts);
    return;
  }
  constexpr uint32_t N = 32 * WPS;  // threads of a segment
  const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) / N, lane = threadIdx.x % N;
  if (g >= wk.nsegs) return;
  const Segment sg = wk.segs[g];
  const Stream& s = wk.streams[sg.stream];
  const bool bare = (s.mode & kStreamBare) != 0;
  const uint32_t hdr = bare ? 0 : fmt_header_bytes(s.fmt);
  uint32_t* dst = reinterpret_cast<uint32_t*>(wk.out + s.out_off);
  Piece* pc = wk.pieces + s.piece_first + sg.piece_off;
  const uint32_t slots = seg_piece_slots(sg.tile_count, sg.len);
  const uint64_t c = uint64_t(hdr) * 8 + sg.bit_off;  // block start in the output slot
  const bool last = (sg.flags & kSegLast) != 0;
  // slots that stay empty: from `used` on, and the code table's of a fixed block
  const bool coded = sg.block_type != kBlkStored;
  const uint32_t used = s.error ? 0u : coded ? 2 + 2 * sg.tile_count + (sg.block_type == kBlkDynamic ? 1u : 0u)
                                             : stored_slots(sg.len);
  for (uint32_t i = used + lane; i < slots; i += N) pc[i].nbits = 0;
  if (s.error) return;
  if (lane == 0 && sg.block_type == kBlkFixed) pc[1].nbits = 0;
  if (sg.block_type == kBlkStored) {
    const uint64_t c1 = ((c + 3 + 7) & ~uint64_t(7)) + 32 + 8ull * 65535;  // start of piece 1 (if there is one)
    // per stored piece its header, its length and copies of 4 KiB at most: one
    // warp copies a Piece
    constexpr uint32_t kPer = 2 + kStoredSplit;
    for (uint32_t x = lane; x < used; x += N) {
      const uint32_t i = x / kPer, k = x % kPer;
      const uint64_t ci = i == 0 ? c : c1 + uint64_t(i - 1) * (40 + 8ull * 65535);
      const uint32_t off = i * 65535u, n = min(sg.len - off, 65535u);
      const bool fin = last && off + n == sg.len;
      const uint64_t lenpos = (ci + 3 + 7) & ~uint64_t(7);
      if (k == 0) {
        pc[x] = Piece{nullptr, dst, 0, ci, 3, fin ? 1u : 0u};
      } else if (k == 1) {
        pc[x] = Piece{nullptr, dst, 0, lenpos, 32, n | ((~n & 0xFFFFu) << 16)};
      } else {
        const uint32_t o = (k - 2) * kStoredPart;
        const uint64_t a = sg.in_off + off + o;
        pc[x] = Piece{reinterpret_cast<const uint32_t*>(wk.in + (a & ~uint64_t(3))), dst, (a & 3) * 8,
                      lenpos + 32 + 8ull * o, min(kStoredPart, n - o) * 8, 0};
      }
    }
    return;
  }
  // BFINAL + BTYPE (write_bits(type, 2) puts the low bit first), then the
  // code-length header of a dynamic block (written by the Huffman kernel)
  uint64_t at = c + 3;
  if (lane == 0) pc[0] = Piece{nullptr, dst, 0, c, 3, (last ? 1u : 0u) | (sg.block_type << 1)};
  if (sg.block_type == kBlkDynamic) {
    if (lane == 0)
      pc[1] = Piece{reinterpret_cast<const uint32_t*>(wk.scratch + sg.hdr_off), dst, 0, at, sg.hdr_bits, 0};
    at += sg.hdr_bits;
  }
  // two copies per tile (fix-up bits, then the speculative bits from the
  // splice point), at offsets from a prefix sum over the tiles
  struct Row {
    uint32_t fb, sp, bits, len;
    uint64_t words;
  };
  auto load = [&](uint32_t t) {
    Row r{0, 0, 0, 0, 0};
    if (t < sg.tile_count) {
      const Tile& tl = wk.tiles[sg.tile_first + t];
      r = Row{tl.fix_bits, tl.splice_bit, tl.spec_bits, tl.len, tl.scratch};
    }
    return r;
  };
  Row next = load(lane);
  for (uint32_t t0 = 0; t0 < sg.tile_count; t0 += N) {
    const uint32_t t = t0 + lane;
    const Row r = next;
    next = load(t + N);
    const uint32_t fb = r.fb, sp = r.sp, sb = r.bits - sp;
    unsigned long long incl = uint64_t(fb) + sb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(kFullMask, incl, o);
      if ((lane & 31) >= uint32_t(o)) incl += v;
    }
    unsigned long long total;  // of these tiles
    if constexpr (WPS > 1) {
      __shared__ unsigned long long part[WPS];
      __syncthreads();  // the sums before have been read
      if ((lane & 31) == 31) part[lane >> 5] = incl;
      __syncthreads();
      total = 0;
#pragma unroll
      for (int k = 0; k < WPS; ++k) {
        if (uint32_t(k) < lane >> 5) incl += part[k];
        total += part[k];
      }
    } else {
      total = __shfl_sync(kFullMask, incl, 31);
    }
    const uint64_t mine = at + incl - (uint64_t(fb) + sb);
    if (t < sg.tile_count) {
      const uint32_t* spec = reinterpret_cast<const uint32_t*>(wk.scratch + r.words);
      const uint32_t* fix = reinterpret_cast<const uint32_t*>(wk.scratch + r.words + tile_stream_bytes(r.len));
      pc[2 + 2 * t] = Piece{fix, dst, 0, mine, fb, 0};
      pc[3 + 2 * t] = Piece{spec, dst, sp, mine + fb, sb, 0};
    }
    at += total;
  }
  if (lane == 0 && sg.block_type == kBlkDynamic) {
    const uint32_t eob = sg.eob;  // dynamic EOB: code | (len << 16)
    pc[2 + 2 * sg.tile_count] = Piece{nullptr, dst, 0, at, eob >> 16, eob & 0xFFFFu};
  }
}

// ---------------------------------------------------------------- checksums
__constant__ uint32_t c_crc_slice[4][256];
__constant__ uint32_t c_crc_sub[9];   // x^(8*256*2^s), s = 0..8
__constant__ uint32_t c_crc_block;    // x^(8*65536)

constexpr uint32_t kAdlerMod = 65521u;
constexpr uint32_t kCkBlock = 65536u;
constexpr uint32_t kCkSub = 256u;

__global__ void __launch_bounds__(256) k_ck_block(Work wk, CrcPowers pw) {
  begin_kernel();
  __shared__ uint32_t tb[4][256];
  __shared__ uint32_t sc[256], sa[256], sb2[256], sl[256];
  for (int i = threadIdx.x; i < 1024; i += blockDim.x) tb[i >> 8][i & 255] = c_crc_slice[i >> 8][i & 255];
  __syncthreads();
  const uint32_t bi = blockIdx.x;
  if (bi >= wk.nck) return;
  CkBlock b = wk.ck[bi];
  const uint32_t t = threadIdx.x;
  const uint32_t o0 = t * kCkSub;
  const uint32_t len = o0 < b.len ? min(kCkSub, b.len - o0) : 0u;
  const uint8_t* p = wk.in + b.in_off + o0;
  uint32_t crc = 0, A = 0, B = 0;
  uint32_t i = 0;
  const uint32_t what = b.what;  // uniform over the block
  // one 32-bit word: CRC slicing-by-4; Adler A += bytes, B += 4A + 4,3,2,1-weighted bytes
  auto word = [&](uint32_t v) {
    if (what & kCkCrc) {
      crc ^= v;
      crc = tb[3][crc & 0xFF] ^ tb[2][(crc >> 8) & 0xFF] ^ tb[1][(crc >> 16) & 0xFF] ^ tb[0][crc >> 24];
    }
    if (what & kCkAdler) {
      B += 4 * A + __dp4a(v, 0x01020304u, 0u);
      A += __dp4a(v, 0x01010101u, 0u);
    }
  };
  const uint64_t ab = b.in_off + o0;
  if ((ab & 15) == 0) {
    const uint4* p16 = reinterpret_cast<const uint4*>(wk.in + ab);
    for (; i + 16 <= len; i += 16) {
      const uint4 v = __ldg(p16 + (i >> 4));
      word(v.x);
      word(v.y);
      word(v.z);
      word(v.w);
    }
  }
  // aligned words, funnel-shifted when the block does not start on a word
  const uint32_t* pw4 = reinterpret_cast<const uint32_t*>(wk.in + (ab & ~uint64_t(3)));
  const uint32_t sh = uint32_t(ab & 3) * 8;
  for (; i + 4 <= len; i += 4)
    word(sh ? __funnelshift_r(__ldg(pw4 + (i >> 2)), __ldg(pw4 + (i >> 2) + 1), sh) : __ldg(pw4 + (i >> 2)));
  for (; i < len; ++i) {
    const uint32_t by = p[i];
    crc = tb[0][(crc ^ by) & 0xFF] ^ (crc >> 8);
    A += by;
    B += A;
  }
  // B so far is sum_j (prefix sums) = sum_i (len - i) d_i, as the fold wants.
  sc[t] = crc;
  sa[t] = A % kAdlerMod;
  sb2[t] = B % kAdlerMod;
  sl[t] = len;
  __syncthreads();
  int lvl = 0;
  for (uint32_t s = 1; s < 256; s <<= 1, ++lvl) {
    if ((t & (2 * s - 1)) == 0 && t + s < 256) {
      const uint32_t lr = sl[t + s];
      if (lr) {
        if (what & kCkCrc) {
          const uint32_t shift = (lr == kCkSub * s) ? c_crc_sub[lvl] : xpow8n(pw, lr);
          sc[t] = gf2_mulmod(shift, sc[t]) ^ sc[t + s];
        }
        if (what & kCkAdler) {
          sb2[t] = uint32_t((uint64_t(sb2[t]) + uint64_t(lr % kAdlerMod) * sa[t] + sb2[t + s]) % kAdlerMod);
          sa[t] = (sa[t] + sa[t + s]) % kAdlerMod;
        }
        sl[t] += lr;
      }
    }
    __syncthreads();
  }
  if (t == 0) {
    b.crc = sc[0];
    b.a = sa[0];
    b.b = sb2[0];
    wk.ck[bi] = b;
  }
}

// Checksum partial of a byte range: the raw CRC register from 0, Adler sums
// A = sum of bytes and B = sum of (len - i) * byte_i (mod 65521), and length.
struct CkPartial {
  uint32_t crc, a, b;
  uint64_t len;
};
constexpr int kFoldThreads = 128;

// Folds blocks blk[0, n) in order into one partial: every thread of the CTA
// (kFoldThreads threads) folds a contiguous run of blocks, then the runs are
// combined in a tree (appending R multiplies the CRC register by x^(8|R|) and
// adds |R| * A to B).  Every thread must call it; thread 0 gets the result.
__device__ CkPartial fold_blocks(const CkBlock* blk, uint32_t n, uint32_t what, const CrcPowers& pw,
                                 CkPartial* sh) {
  const uint32_t t = threadIdx.x;
  const uint32_t per = (n + kFoldThreads - 1) / kFoldThreads;
  const uint32_t b0 = min(n, t * per), b1 = min(n, b0 + per);
  CkPartial p{0, 0, 0, 0};
  for (uint32_t i = b0; i < b1; ++i) {
    const CkBlock b = blk[i];
    if (what & kCkCrc) p.crc = gf2_mulmod(b.len == kCkBlock ? c_crc_block : xpow8n(pw, b.len), p.crc) ^ b.crc;
    if (what & kCkAdler) {
      p.b = uint32_t((uint64_t(p.b) + uint64_t(b.len % kAdlerMod) * p.a + b.b) % kAdlerMod);
      p.a = (p.a + b.a) % kAdlerMod;
    }
    p.len += b.len;
  }
  sh[t] = p;
  __syncthreads();
  for (uint32_t s = 1; s < uint32_t(kFoldThreads); s <<= 1) {
    if ((t & (2 * s - 1)) == 0 && t + s < uint32_t(kFoldThreads)) {
      CkPartial l = sh[t];
      const CkPartial r = sh[t + s];
      if (r.len) {
        if (what & kCkCrc) l.crc = gf2_mulmod(xpow8n(pw, r.len), l.crc) ^ r.crc;
        if (what & kCkAdler) {
          l.b = uint32_t((uint64_t(l.b) + (r.len % kAdlerMod) * l.a + r.b) % kAdlerMod);
          l.a = (l.a + r.a) % kAdlerMod;
        }
        l.len += r.len;
        sh[t] = l;
      }
    }
    __syncthreads();
  }
  return sh[0];
}

// zlib / gzip header and trailer bytes of a stream (one thread).
__device__ void write_frame(const Work& wk, const Stream& s, uint32_t check) {
  if (s.error || (s.mode & kStreamBare)) return;
  uint8_t* o = wk.out + s.out_off;
  const uint64_t end = s.out_size;
  if (s.fmt == kFmtZlib) {
    // header 78 9C (zlib_wrapper.cpp:21-22), Adler-32 big-endian trailer
    o[0] = 0x78; o[1] = 0x9C;
    for (int i = 0; i < 4; ++i) o[end - 4 + i] = uint8_t(check >> (24 - 8 * i));
  } else {
    // 1F 8B 08 00 mtime=0 XFL OS=FF (gzip_wrapper.cpp:31-43); the parallel
    // path always writes XFL 0 (parallel_compressor.cpp:96-98)
    const uint8_t xfl = s.parallel ? 0 : (s.level >= 9 ? 2 : (s.level <= 2 ? 4 : 0));
    const uint8_t h[10] = {0x1F, 0x8B, 8, 0, 0, 0, 0, 0, xfl, 0xFF};
    for (int i = 0; i < 10; ++i) o[i] = h[i];
    const uint32_t isz = uint32_t(s.in_len);
    for (int i = 0; i < 4; ++i) {
      o[end - 8 + i] = uint8_t(check >> (8 * i));
      o[end - 4 + i] = uint8_t(isz >> (8 * i));
    }
  }
}

// One CTA per stream; with `frame` the stream's output (joined before) gets its
// header and trailer.
__global__ void __launch_bounds__(kFoldThreads) k_ck_fold(Work wk, CrcPowers pw, bool frame) {
  begin_kernel();
  __shared__ CkPartial sh[kFoldThreads];
  const uint32_t si = blockIdx.x;
  if (si >= wk.nstreams) return;
  const Stream& s = wk.streams[si];
  if (s.fmt == kFmtRaw) return;
  const uint32_t what = s.fmt == kFmtGzip ? kCkCrc : kCkAdler;
  const CkPartial p = fold_blocks(wk.ck + s.ck_first, s.ck_count, what, pw, sh);
  if (threadIdx.x) return;
  uint32_t check;
  if (s.fmt == kFmtGzip) {
    // crc32(0, data) = ~(x^(8n) * ~0 + raw(data))
    check = ~(gf2_mulmod(xpow8n(pw, s.in_len), 0xFFFFFFFFu) ^ p.crc);
  } else {
    // Adler-32 from 1: s1 = 1 + A, s2 = n + B
    const uint64_t s1 = (1 + p.a) % kAdlerMod, s2 = (s.in_len % kAdlerMod + p.b) % kAdlerMod;
    check = uint32_t(s2 << 16) | uint32_t(s1);
  }
  wk.streams[si].checksum = check;
  if (frame) write_frame(wk, s, check);
}

// Single-stream checksum with an arbitrary initial value (deflate_crc32 /
// deflate_adler32): result written to *res.  One CTA.
__global__ void __launch_bounds__(kFoldThreads) k_ck_single(const CkBlock* ck, uint32_t nck, uint64_t total,
                                                            uint32_t init, int adler, CrcPowers pw, uint32_t* res) {
  __shared__ CkPartial sh[kFoldThreads];
  if (blockIdx.x) return;
  const CkPartial p = fold_blocks(ck, nck, adler ? kCkAdler : kCkCrc, pw, sh);
  if (threadIdx.x) return;
  if (adler) {
    const uint64_t a0 = (init & 0xFFFFu) % kAdlerMod, b0 = (init >> 16) % kAdlerMod;
    const uint64_t s1 = (a0 + p.a) % kAdlerMod;
    const uint64_t s2 = (b0 + (total % kAdlerMod) * a0 + p.b) % kAdlerMod;
    *res = uint32_t(s2 << 16) | uint32_t(s1);
  } else {
    *res = ~(gf2_mulmod(xpow8n(pw, total), ~init) ^ p.crc);
  }
}

// ---------------------------------------------------------------- k_join
__global__ void __launch_bounds__(256) k_join(Work wk, uint32_t* counter) {
  begin_kernel();
  const uint32_t lane = threadIdx.x & 31;
  for (;;) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(counter, 1u);
    i = __shfl_sync(kFullMask, i, 0);
    if (i >= wk.npieces) break;
    const Piece pc = wk.pieces[i];
    if (pc.nbits == 0) continue;
    uint32_t* dst = pc.dst;
    if (pc.src == nullptr) {
      if (lane == 0) {
        const uint64_t w = pc.dst_bit >> 5;
        const uint32_t sh = uint32_t(pc.dst_bit & 31);
        const uint32_t v = pc.nbits == 32 ? pc.value : (pc.value & ((1u << pc.nbits) - 1));
        atomicOr(dst + w, v << sh);
        if (sh + pc.nbits > 32) atomicOr(dst + w + 1, v >> (32 - sh));
      }
      continue;
    }
    const uint64_t d0 = pc.dst_bit, d1 = pc.dst_bit + pc.nbits;
    const uint64_t w0 = d0 >> 5, w1 = (d1 - 1) >> 5;
    const int64_t delta = int64_t(pc.src_bit) - int64_t(d0);
    // source word of destination word w0 (floor) and the shift; both sides
    // advance word by word
    const int64_t s0 = int64_t(w0) * 32 + delta;
    const uint32_t* src = pc.src + (s0 >> 5);
    const uint32_t sh = uint32_t(s0 & 31);
    const uint32_t nw = uint32_t(w1 - w0);  // the last word
    uint32_t* dw = dst + w0;
    // the words inside, four per lane in flight
    uint32_t k = lane == 0 ? 32u : lane;  // word 0 and word nw may be shared with other copies
    for (; k + 96 < nw; k += 128) {
      uint32_t lo[4], hi[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        lo[u] = __ldg(src + k + 32 * u);
        hi[u] = __ldg(src + k + 32 * u + 1);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) dw[k + 32 * u] = __funnelshift_r(lo[u], hi[u], sh);
    }
    for (; k < nw; k += 32) dw[k] = __funnelshift_r(__ldg(src + k), __ldg(src + k + 1), sh);
    if (lane == 0 || (lane == 1 && nw)) {
      const uint32_t e = lane ? nw : 0u;
      const uint64_t x0 = (w0 + e) * 32;
      const uint32_t lb = uint32_t((d0 > x0 ? d0 : x0) - x0);
      const uint32_t hb = uint32_t((d1 < x0 + 32 ? d1 : x0 + 32) - x0);
      const uint32_t lo = (s0 >> 5) + int64_t(e) >= 0 ? __ldg(src + e) : 0u;
      const uint32_t v = __funnelshift_r(lo, __ldg(src + e + 1), sh);
      if (lb == 0 && hb == 32) {
        dw[e] = v;
      } else {
        const uint32_t m = (hb - lb == 32) ? kFullMask : (((1u << (hb - lb)) - 1) << lb);
        atomicOr(dw + e, v & m);
      }
    }
  }
}

// ---------------------------------------------------------------- launchers
// The constant tables live in each device's own constant memory, so they are
// uploaded once per device (under a lock: engines of one device may be
// created by several host threads at once).
bool upload_crc_tables() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  std::lock_guard<std::mutex> lk(mu);
  if (done[dev]) return true;
  uint32_t t[4][256];
  for (uint32_t i = 0; i < 256; ++i) {
    uint32_t c = i;
    for (int k = 0; k < 8; ++k) c = (c & 1) ? (c >> 1) ^ kCrcPoly : (c >> 1);
    t[0][i] = c;
  }
  for (int s = 1; s < 4; ++s)
    for (int i = 0; i < 256; ++i) t[s][i] = (t[s - 1][i] >> 8) ^ t[0][t[s - 1][i] & 0xFF];
  CrcPowers pw = host_crc_powers();
  uint32_t sub[9];
  for (int s = 0; s < 9; ++s) sub[s] = xpow8n(pw, uint64_t(kCkSub) << s);
  const uint32_t blk = xpow8n(pw, kCkBlock);
  if (cudaMemcpyToSymbol(c_crc_slice, t, sizeof t) != cudaSuccess ||
      cudaMemcpyToSymbol(c_crc_sub, sub, sizeof sub) != cudaSuccess ||
      cudaMemcpyToSymbol(c_crc_block, &blk, sizeof blk) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  done[dev] = true;
  return true;
}

CrcPowers host_crc_powers() {
  CrcPowers pw;
  uint32_t x = 0x40000000u;  // the polynomial x
  for (int k = 0; k < 64; ++k) { pw.x2k[k] = x; x = gf2_mulmod(x, x); }
  return pw;
}

void launch_plan(const Work& wk, uint64_t max_out, cudaStream_t st) {
  if (!wk.nstreams) return;
  const bool cta = wk.nsegs <= kPlanCtaSegs;  // a CTA per segment
  const uint32_t seg_ctas = cta ? wk.nsegs : (wk.nsegs + 7) / 8;
  if (wk.nsegs) launch_after((cta ? k_plan_seg<8> : k_plan_seg<1>), seg_ctas, 256, 0, st, wk);
  launch_after(k_plan_stream, (wk.nstreams + 7) / 8, 256, 0, st, wk);
  // clearing CTAs per stream: 64 KiB of the largest stream's output each for few
  // streams (128 MiB in one: 32 us, at 1 MiB each; now 17), 1 MiB for many
  const uint64_t few = std::max<uint64_t>(1, 2048 / wk.nstreams);
  const uint64_t most = std::min<uint64_t>(256, std::max<uint64_t>(1, max_out >> 20));
  const uint32_t parts = uint32_t(std::max(most, std::min(few, max_out >> 16)));
  launch_after((cta ? k_plan_pieces<8> : k_plan_pieces<1>), seg_ctas + wk.nstreams * parts, 256, 0, st, wk, seg_ctas, parts);
}

void launch_checksums(const Work& wk, bool frame, cudaStream_t st) {
  const CrcPowers pw = host_crc_powers();
  if (wk.nck) launch_after(k_ck_block, wk.nck, 256, 0, st, wk, pw);
  if (wk.nstreams) launch_after(k_ck_fold, wk.nstreams, kFoldThreads, 0, st, wk, pw, frame);
}

void launch_ck_single(const CkBlock* ck, uint32_t nck, uint64_t total, uint32_t init, int adler, uint32_t* res,
                      const Work& wk, cudaStream_t st) {
  const CrcPowers pw = host_crc_powers();
  if (nck) launch_after(k_ck_block, nck, 256, 0, st, wk, pw);
  k_ck_single<<<1, kFoldThreads, 0, st>>>(ck, nck, total, init, adler, pw, res);
}

void launch_join(const Work& wk, uint32_t* counter, cudaStream_t st, int sms) {
  if (!wk.npieces) return;
  uint32_t blocks = uint32_t(sms) * 8;
  const uint32_t need = (wk.npieces + 7) / 8;
  if (blocks > need) blocks = need;
  launch_after(k_join, blocks, 256, 0, st, wk, counter);
}

}  // namespace orotb
