// kernels.cuh -- launch interface between the host engine and the kernels.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include "engine.cuh"
#include "deflate_device.cuh"

namespace orotb {

// Index of the calling thread's current device for per-device launch caches
// (kernel attributes and occupancy are properties of a device and never
// change, so they are set and queried on a device's first launch only).
inline int device_slot() {
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) d = 0;
  return d;
}

// The kernels of a pass are launched so that one may start while the one before
// ends (programmatic dependent launch): every kernel begins with begin_kernel(),
// which lets the next one be launched as soon as all CTAs of this one run, and
// waits until the kernels before have completed and their writes are visible.
// No kernel touches memory before that.  A pass is 8 to 13 launches, whose gaps
// were a seventh of a small call: 4 KiB at level 6 148 -> 126 us, 100 kB at level 1
// 178 -> 158; passes of many MiB take the same.
__device__ __forceinline__ void begin_kernel() {
  asm volatile("griddepcontrol.launch_dependents;\n griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Device pointers of one compression pass.
struct Work {
  const uint8_t* in;     // input arena (16-byte aligned, 64 bytes of padding)
  uint8_t* out;          // output arena
  uint8_t* scratch;      // per-tile bit buffers, records, carried hash tables
  Stream* streams;
  Segment* segs;
  Tile* tiles;
  Piece* pieces;
  CkBlock* ck;
  uint32_t nstreams, nsegs, ntiles, npieces, nck;
  uint32_t pad;
};

// Index lists for the fast-level (1-3) pipeline of one hash width.
struct FastLists {
  const uint32_t* lastocc;   // tiles that publish a last-occurrence table
  uint32_t n_lastocc;
  const uint32_t* multi;     // segments with more than one tile
  uint32_t n_multi;
  const uint32_t* chunks;    // (segment, chunk) of every chunk of kCarryChunk tiles of theirs
  uint32_t n_chunks;
  const uint32_t* chunked;   // segments of more than one chunk
  uint32_t n_chunked;
  const uint32_t* walk;      // tiles to walk
  uint32_t n_walk;
  uint32_t* counter;         // zeroed work counters
  uint32_t* ready;           // zeroed, one flag per tile of `walk` (candidates done)
};

// Index lists for the lazy-level (4-12) pipeline.
struct LazyLists {
  const uint32_t* runs;      // (first tile, tile count) of every run, count <= kLazyRun
  uint32_t n_runs;
  const uint32_t* groups;    // (first tile, tile count) of every search group, count <= kSearchTiles
  uint32_t n_groups;
  const uint32_t* tiles;     // tiles to encode
  uint32_t n_tiles;
  const uint32_t* segs;      // segments needing Huffman tables
  uint32_t n_segs;
  bool any_lazy, any_opt;    // tiles of levels 4-9 / 10-12 among them
};

// Optional per-phase CUDA events: mark(id) records an event after phase id.
enum Phase { kPhPre = 0, kPhCand, kPhWalk, kPhFix, kPhLazyLz, kPhLazyHuff, kPhLazyEnc, kPhPlan, kPhJoin, kPhCheck, kPhFrame,
             kNumPhases };
struct Marks {
  cudaEvent_t ev[kNumPhases + 1];
  int id[kNumPhases + 1];
  int n = 0;
  bool on = false;
  void mark(int phase, cudaStream_t st) {
    if (!on || n > kNumPhases) return;
    cudaEventRecord(ev[n], st);
    id[n++] = phase;
  }
};

void launch_fast(const Work& wk, const FastLists& L, int hash_bits, cudaStream_t st, int sms, Marks* mk);
// Whether launch_fast runs the candidate pass and the parse as one kernel.
bool fast_launches_fused();
int launch_lazy(const Work& wk, const LazyLists& L, cudaStream_t st, int sms, Marks* mk);
void launch_plan(const Work& wk, uint64_t max_out, cudaStream_t st);  // max_out: largest stream bound
// Checksums of every stream; `frame`: and its header and trailer (after launch_join).
void launch_checksums(const Work& wk, bool frame, cudaStream_t st);
void launch_ck_single(const CkBlock* ck, uint32_t nck, uint64_t total, uint32_t init, int adler, uint32_t* res,
                      const Work& wk, cudaStream_t st);
CrcPowers host_crc_powers();
void launch_join(const Work& wk, uint32_t* counter, cudaStream_t st, int sms);
bool upload_crc_tables();  // once per device; false on a device error

// One DEFLATE stream to decode (raw data, framing stripped by the host).
struct InflateJob {
  uint64_t in_off;   // raw DEFLATE bytes, relative to the input base
  uint64_t in_len;
  uint64_t out_off;  // output slot, relative to the output base
  uint64_t out_cap;
  uint64_t out_len;  // result: bytes written
  uint64_t in_used;  // result: bytes of input the stream occupied
  int32_t status;    // result: kInf*
  uint32_t pad;
};
constexpr int32_t kInfOk = 0, kInfData = 1, kInfOutput = 2, kInfInput = 3, kInfMismatch = 4;
// How many of the streams order[0..n) (by decreasing in_len) are decoded by large
// CTAs, one per SM; the others by small ones, eight per SM, which pay where a
// large one would wait for the same dozens of steps whatever the stream's length: for
// short streams, the longer the more rounds of large CTAs they would take, and
// most of the streams, since the small CTAs start after the large ones.
// deflate_gpu_batch_verify of text at level 6 (us), all large / small / with the one
// warp per stream that went before: 300 of 100 to 200 bytes 186 / 146 / 163, 10,000
// of them 4300 / 2080 / 2090, 10,000 of 1 to 4 KiB 5200 / 2580 / 3400, 1,000 of 32 to
// 64 KiB 1560 / 1560 / 5340.  Limits of 512 bytes a round, or without the
// majority, made mixed sizes up to 20% slower than all large.
inline uint32_t large_streams(const InflateJob* jobs, const uint32_t* order, uint32_t n, int sms) {
  auto shorter = [&](uint64_t len) {
    uint32_t k = 0;
    while (k < n && jobs[order[n - 1 - k]].in_len < len) ++k;
    return k;
  };
  const uint64_t rounds = shorter(4096) / uint32_t(sms);
  const uint32_t small = shorter(rounds < 16 ? 256 * rounds : 4096);
  return small > uint32_t(sms) && small > n / 2 ? n - small : n;
}
// Decodes jobs[order[0..n)] (one CTA per stream, a large one for the first nlarge;
// the input and output buffers carry at least 8 bytes of padding); `counters` are
// two device words.
void launch_inflate(const uint8_t* in, uint8_t* out, InflateJob* jobs, const uint32_t* order, uint32_t njobs,
                    uint32_t nlarge, uint32_t* counters, int sms, cudaStream_t st);
// Marks kInfMismatch on streams whose framing or trailer is wrong (job i is stream i).
void launch_frame_check(const uint8_t* out, const Stream* streams, InflateJob* jobs, uint32_t n, cudaStream_t st);
// Marks kInfMismatch on jobs whose decoded bytes differ from ref[ref_off[j], + ref_len[j]).
void launch_inflate_compare(const uint8_t* decoded, const uint8_t* ref, InflateJob* jobs, const uint64_t* ref_off,
                            const uint64_t* ref_len, uint32_t njobs, cudaStream_t st);

}  // namespace orotb
