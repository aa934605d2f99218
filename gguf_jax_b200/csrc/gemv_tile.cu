#include "gemv_tile.cuh"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>

namespace ggq {
namespace tile {

// ---------------------------------------------------------------------------------------------
// host side

struct FormatInfo { int qt, ts, table_bytes, sum_groups, oct; bool sums, four_passes; };

template <class F>
constexpr FormatInfo info_of() { return {F::kQt, F::kTs, F::kTableBytes, F::kOct / F::kGroupOct, F::kOct, F::kSums, four_passes<F>()}; }

static bool format_of(int qtype, FormatInfo* fi) {
  switch (qtype) {
    case QT_Q4_K: *fi = info_of<tf::Q4K>(); return true;
    case QT_Q5_K: *fi = info_of<tf::Q5K>(); return true;
    case QT_Q6_K: *fi = info_of<tf::Q6K>(); return true;
    case QT_Q2_K: *fi = info_of<tf::Q2K>(); return true;
    case QT_IQ4_XS: *fi = info_of<tf::IQ4XS>(); return true;
    case QT_IQ2_XXS: *fi = info_of<tf::IQ2XXS>(); return true;
    case QT_IQ2_XS: *fi = info_of<tf::IQ2XS>(); return true;
    case QT_IQ2_S: *fi = info_of<tf::IQ2S>(); return true;
    case QT_IQ3_XXS: *fi = info_of<tf::IQ3XXS>(); return true;
    case QT_IQ3_S: *fi = info_of<tf::IQ3S>(); return true;
    case QT_IQ1_S: *fi = info_of<tf::IQ1S>(); return true;
    case QT_IQ1_M: *fi = info_of<tf::IQ1M>(); return true;
    case QT_Q3_K: *fi = info_of<tf::Q3K>(); return true;
    case QT_TQ1_0: *fi = info_of<tf::TQ10>(); return true;
    case QT_TQ2_0: *fi = info_of<tf::TQ20>(); return true;
    case QT_Q8_0: *fi = info_of<tf::Q80>(); return true;
    case QT_Q4_0: *fi = info_of<tf::Q40>(); return true;
    case QT_Q4_1: *fi = info_of<tf::Q41>(); return true;
    case QT_Q5_0: *fi = info_of<tf::Q50>(); return true;
    case QT_Q5_1: *fi = info_of<tf::Q51>(); return true;
    case QT_IQ4_NL: *fi = info_of<tf::IQ4NL>(); return true;
    case QT_MXFP4: *fi = info_of<tf::MXFP4>(); return true;
    case QT_NVFP4: *fi = info_of<tf::NVFP4>(); return true;
    default: return false;
  }
}

static int passes_of(int M) { return M <= 2 ? 1 : M <= 4 ? 2 : 4; }

// Smallest K chunk (in superblocks) the plan may use.  Eight for weights with enough (chunk, row tile)
// units to give every warp of the device at least one; smaller for small weights, so that they still
// spread over the whole device.  The scratch is sized by the same rule.
static int min_chunk_sb(int64_t N, int64_t K) {
  const int64_t RT = (N + 15) / 16, SB = K / 256;
  int chunk = 8;
  while (chunk > 1 && RT * ((SB + chunk - 1) / chunk) < 148 * kWarps) chunk /= 2;
  return chunk;
}

// Shared-memory layout and work split for one launch; false if nothing fits.
static bool plan(const FormatInfo& fi, int64_t N, int64_t K, int M, int sm_count, int nb_forced, int chunk_forced, Geo* out) {
  const int SB = (int)(K / 256);
  const int x_rows = 2 * passes_of(M);
  Geo best{};
  double best_cost = 1e30;
  for (int nb = 1; nb <= 4; nb *= 2) {
    if (nb_forced > 0 && nb != nb_forced) continue;
    for (int chunk = min_chunk_sb(N, K); ; chunk *= 2) {
      const bool whole_k = chunk >= SB;
      if (chunk % nb == 0 && (chunk_forced <= 0 || chunk == chunk_forced || whole_k)) {
        Geo g{};
        g.nb = nb;
        g.chunk_sb = whole_k ? (SB + nb - 1) / nb * nb : chunk;
        g.spu = g.chunk_sb / nb;
        g.C = (SB + g.chunk_sb - 1) / g.chunk_sb;
        g.RT = (int)((N + 15) / 16);
        g.row_skew = (int)((int64_t)SB * fi.ts % 16);
        g.S = (int64_t)g.C * g.RT * g.spu;
        const int64_t units = (int64_t)g.C * g.RT;
        g.W = (int)std::min<int64_t>((int64_t)sm_count * kWarps, units);
        g.x_rows = x_rows;
        g.x_row_bytes = g.chunk_sb * 4 * (16 * fi.oct + 16);
        g.x_row_bytes += (64 - g.x_row_bytes % 128 + 128) % 128;      // 64 (mod 128): see the staging
        g.xs_row_floats = fi.sums ? g.chunk_sb * 4 * fi.sum_groups : 0;
        // a block starts at a multiple of gcd(ts, 16) bytes in its 16-byte aligned window (ts a multiple of 16: at its start; with room for
        // the largest offset there all the same, Q8_0's ring did not fit next to eight batch rows and large weights had no plan:
        // 8192 x 12288 at 8 rows 65 to 84 us on the MMA kernel, 43 here)
        const int pieces = (16 - std::gcd(fi.ts, 16) + nb * fi.ts + 15) / 16;
        if (pieces > 48) { if (whole_k) break; continue; }     // three 16-byte pieces per lane of a half-warp and row
        g.pitch = 16 * pieces;
        if (g.pitch % 32 == 0) g.pitch += 16;          // odd multiple of 16: rows fall into different bank groups
        g.slot_bytes = 16 * g.pitch;
        // chunks a CTA's sixteen warps can touch: their steps span at most this many chunks
        const int64_t cta_steps = (g.S * kWarps + g.W - 1) / g.W + 1;
        const int64_t span = (cta_steps + (int64_t)g.RT * g.spu - 2) / ((int64_t)g.RT * g.spu) + 1;
        const int bufs = (int)std::min<int64_t>(span, g.C);
        const bool span_ok = bufs <= kMaxXBufs;
        g.xbufs = bufs;
        const int fixed = bufs * x_rows * (g.x_row_bytes + g.xs_row_floats * 4) + 64 + (fi.table_bytes + 15) / 16 * 16 + 64 * kMaxXBufs + kWarps * kMaxDepth * 8;
        const int room = kSmemLimit - fixed;
        // a ring of two slots at least; a warp that has a single step fills one (the tables of the grid formats leave no room for
        // two slots of four superblocks, and the split into smaller steps took longer: IQ2_XXS 8192 x 4096 at 8 rows 24.8 us, 22)
        const int64_t warp_steps = (g.S + g.W - 1) / g.W;
        const int fit = room / (kWarps * g.slot_bytes);
        if (span_ok && fit >= std::min<int64_t>(2, warp_steps)) {
          // (more than two slots of over 4 KB only put more weights in front of the first activations: Q8_0 14336 x 4096 at batch 1 with
          // two / three / four 19.3 / 19.9 / 19.9 us; smaller slots the same either way)
          const int most = g.slot_bytes > 4096 ? 2 : kMaxDepth;
          g.depth = std::min(most, std::max(2, fit));
          g.slots = (int)std::min<int64_t>(g.depth, warp_steps);
          g.off_x = kWarps * g.slots * g.slot_bytes;
          g.off_xs = g.off_x + bufs * x_rows * g.x_row_bytes;
          g.off_zero = g.off_xs + bufs * x_rows * g.xs_row_floats * 4;
          g.off_tab = g.off_zero + 64;
          g.off_misc = g.off_tab + (fi.table_bytes + 15) / 16 * 16;
          g.off_bar = g.off_misc + 64 * kMaxXBufs;
          g.total = g.off_bar + kWarps * kMaxDepth * 8;
          // time ~ steps of the busiest warp x (blocks per step + a fixed cost per step) + staging + a flush per
          // unit, in units of one block's multiply; the constants are fitted to B200 timings (8192 x 28672:
          // nb = 2 with chunks of 16 superblocks is the fastest split for every format).  Where steps come as TMA boxes, up to four rows, ranges
          // that end with units save a segment or two, as long as two thirds of the warps have one (us, 8192 x 8192 at batch 1 with units cut /
          // whole: IQ2_XS 20.2 / 17.8, Q8_0 19.4 / 15.4; over 112 shapes, formats and batches timed with six splits each, the split picked takes
          // 0.9 % longer than the best of them, without this term 2.5 %)
          const double steps = (double)warp_steps;
          const bool whole = g.S % ((int64_t)g.W * g.spu) == 0 && g.W >= 0.65 * sm_count * kWarps;
          const double cost = steps * (nb + 0.6) * (g.depth >= std::min(3, most) ? 1.0 : 1.03) + bufs * g.chunk_sb * x_rows * 0.02 +
                              steps / g.spu * 0.6 + (g.row_skew == 0 && M <= 4 && !whole ? 2.0 : 0.0);
          if (cost < best_cost) { best_cost = cost; best = g; }
        }
      }
      if (whole_k) break;
    }
  }
  if (best_cost >= 1e30) return false;
  *out = best;
  return true;
}

static int env_int(const char* name) {
  const char* s = getenv(name);
  return s ? atoi(s) : 0;
}
static int forced_nb() { static const int v = env_int("GGQ_TILE_NB"); return v; }
static int forced_chunk() { static const int v = env_int("GGQ_TILE_CHUNK"); return v; }

}  // namespace tile

// Most batch rows one launch takes for qtype (0: not a tile format): two passes for the formats of the batch kernel, which takes their
// larger batches, four for the others.
int gemv_tile_max_batch(int qtype) {
  tile::FormatInfo fi;
  if (!tile::format_of(qtype, &fi)) return 0;
  return fi.four_passes ? tile::kMaxBatch : 4;
}

// Every 16-row tile has an arrival counter in the counter area that the kernels share.
static bool counters_fit(int64_t N) { return kWsCounterOffset + (size_t)((N + 15) / 16) * sizeof(int) <= kWsGemmPartialOffset; }

bool gemv_tile_applicable(int qtype, int64_t N, int64_t K, int M, const void* w, const void* x, int sm_count) {
  tile::FormatInfo fi;
  if (!tile::format_of(qtype, &fi)) return false;
  if (M < 1 || M > gemv_tile_max_batch(qtype) || K <= 0 || K % 256 || N < 1 || !counters_fit(N)) return false;
  if ((uintptr_t)w % 16 || (uintptr_t)x % 16 || (K * 2) % 16) return false;
  if (N * (K / 256 * fi.ts) >= (1ll << 31)) return false;      // block offsets are 32-bit inside a row; rows are 64-bit
  tile::Geo geo;
  return tile::plan(fi, N, K, M, sm_count, 0, 0, &geo);
}

// Scratch: one arrival counter per 16-row tile in the counter area every kernel shares, and two
// 16 x batch-row float slots per (chunk, row tile) in the float area; sized for the smallest chunk
// the plan may pick.
size_t gemv_tile_workspace_bytes(int qtype, int64_t N, int64_t K, int M) {
  tile::FormatInfo fi;
  if (!tile::format_of(qtype, &fi) || M < 1 || M > tile::kMaxBatch || !counters_fit(N)) return 0;
  const int64_t RT = (N + 15) / 16;
  const int chunk = tile::min_chunk_sb(N, K);
  const int64_t C = (K / 256 + chunk - 1) / chunk;
  const size_t slots = (size_t)(RT * C) * 2 * 16 * 2 * tile::passes_of(M) * sizeof(float);
  return kWsGemmPartialOffset + (slots + 255) / 256 * 256;
}

cudaError_t gemv_tile(int qtype, const uint8_t* w, int64_t N, int64_t K, const void* x, int M, void* y, int y_dtype,
                      void* ws, size_t ws_bytes, int sm_count, int* status, const uint8_t* tab, cudaStream_t st,
                      const PeerPublish* peers) {
  using namespace tile;
  FormatInfo fi;
  if (!format_of(qtype, &fi)) return cudaErrorInvalidValue;
  Geo geo;
  if (!plan(fi, N, K, M, sm_count, forced_nb(), forced_chunk(), &geo) && !plan(fi, N, K, M, sm_count, 0, 0, &geo))
    return cudaErrorInvalidValue;
  if (!ws || ws_bytes < gemv_tile_workspace_bytes(qtype, N, K, M) || (uintptr_t)ws % 256) return cudaErrorInvalidValue;
  if (!counters_fit(N)) return cudaErrorInvalidValue;
  static const bool debug = env_int("GGQ_TILE_DEBUG") != 0;     // prints the plan of every launch (a tuning aid)
  if (debug)
    fprintf(stderr, "gemv_tile qtype %d N=%lld K=%lld M=%d: nb=%d chunk=%d spu=%d C=%d RT=%d S=%lld W=%d depth=%d pitch=%d xbufs=%d smem=%d\n",
            qtype, (long long)N, (long long)K, M, geo.nb, geo.chunk_sb, geo.spu, geo.C, geo.RT, (long long)geo.S, geo.W, geo.depth,
            geo.pitch, geo.xbufs, geo.total);
  const int MP = passes_of(M);
  PeerPublish pp = {};
  if (peers) pp = *peers;
  int* counters = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(ws) + kWsCounterOffset);
  float* slots = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws) + kWsGemmPartialOffset);
  const int grid = (geo.W + kWarps - 1) / kWarps;
  alignas(64) CUtensorMap map = {};
  // (us at batch 1 with cp.async / with boxes: 14336 x 4096 Q8_0 19.3 / 17.5, Q4_0 14.9 / 13.0, IQ4_XS 19.3 / 17.3, MXFP4 19.8 / 17.9, Q2_K 14.3 /
  // 13.3, IQ2_XS 17.9 / 17.6; at four passes, where copies are the least of it, few-row weights were up to 13 % slower with boxes)
  // GGQ_TILE_TMA=0 keeps cp.async, which is also what happens where the driver offers no encoder.
  static const bool want_tma = [] { const char* e = getenv("GGQ_TILE_TMA"); return !(e && e[0] == '0'); }();
  geo.tma = want_tma && geo.row_skew == 0 && MP <= 2 && make_weight_map(&map, w, N, K / 256 * fi.ts, geo.pitch / 4);
  const Args a{&geo, grid, MP, st, w, (int)N, (int)K, x, M, y, y_dtype, counters, slots, &pp, status, tab, &map};
  switch (qtype) {
    case QT_Q4_K: case QT_Q5_K: case QT_Q6_K: case QT_Q2_K: case QT_Q3_K: case QT_TQ1_0: case QT_TQ2_0: return launch_k(qtype, a);
    case QT_IQ4_XS: case QT_IQ2_XXS: case QT_IQ2_XS: case QT_IQ2_S: case QT_IQ3_XXS: case QT_IQ3_S: case QT_IQ1_S: case QT_IQ1_M:
      return launch_iq(qtype, a);
    default: return launch_b32(qtype, a);
  }
}

}  // namespace ggq
