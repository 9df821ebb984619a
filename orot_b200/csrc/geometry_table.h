// geometry_table.h -- pass geometry per pass-size class, read by Engine::plan.
//
// The values were set by hand from sweeps; `python -m orot_b200.tune` (the
// autotuner) times every candidate on the device and rewrites them.  A class
// applies to passes of at least min_bytes input bytes (on a 148-SM B200; other
// devices scale the bounds by their SM count).  Entries are upper limits:
//   tile12, tile14  largest fast-level tile at 12 hash bits (level 1) and
//                   14 (levels 2-3): one warp walks one tile
//                   (passes of a few MiB are cut finer, Engine::pick_tile)
//   lazy_run[g]     most tiles one CTA links or searches at levels 4-6, 7-9 and
//                   10-12 (Engine::lazy_group picks the number)
// Level 1-3 hash widths are fixed (parity with the reference); the output of
// a pass does not depend on any value here.
#pragma once
#include <cstdint>

namespace orotb {

struct GeometryRow {
  uint64_t min_bytes;
  uint32_t tile12, tile14;
  uint32_t lazy_run[3];
};

constexpr const char* kGeometrySource = "tile sweeps on NVIDIA B200, 148 SMs, 2026-12-05";
constexpr GeometryRow kGeometry[] = {
    {0ull, 4096, 4096, {32, 32, 32}},
    {8ull << 20, 4096, 8192, {32, 32, 32}},
    {16ull << 20, 8192, 8192, {32, 32, 32}},
    {32ull << 20, 8192, 16384, {32, 32, 32}},
    {64ull << 20, 16384, 16384, {32, 32, 32}},
    {256ull << 20, 16384, 32768, {32, 32, 32}},
    {1ull << 30, 32768, 65536, {32, 32, 32}},
    {4ull << 30, 65536, 65536, {32, 32, 32}},
};

}  // namespace orotb
