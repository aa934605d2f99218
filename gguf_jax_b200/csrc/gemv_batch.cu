// Host side of the batch kernel (gemv_batch.cuh): formats, work split, launch.
#include "gemv_batch.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <numeric>

namespace ggq {
namespace batch {

struct FormatInfo { int ts, table_bytes, x_tile; };
template <class F>
constexpr FormatInfo info_of() { return {F::Base::kTs, F::Base::kTableBytes, x_tile_bytes<F>()}; }

static bool format_of(int qtype, FormatInfo* fi) {
  switch (qtype) {
    case QT_Q2_K: *fi = info_of<bf::Q2K>(); return true;
    case QT_Q3_K: *fi = info_of<bf::Q3K>(); return true;
    case QT_Q4_K: *fi = info_of<bf::Q4K>(); return true;
    case QT_Q5_K: *fi = info_of<bf::Q5K>(); return true;
    case QT_Q6_K: *fi = info_of<bf::Q6K>(); return true;
    case QT_TQ1_0: *fi = info_of<bf::TQ10>(); return true;
    case QT_TQ2_0: *fi = info_of<bf::TQ20>(); return true;
    case QT_IQ4_XS: *fi = info_of<bf::IQ4XS>(); return true;
    case QT_IQ2_XXS: *fi = info_of<bf::IQ2XXS>(); return true;
    case QT_IQ2_XS: *fi = info_of<bf::IQ2XS>(); return true;
    case QT_IQ2_S: *fi = info_of<bf::IQ2S>(); return true;
    case QT_IQ3_XXS: *fi = info_of<bf::IQ3XXS>(); return true;
    case QT_IQ3_S: *fi = info_of<bf::IQ3S>(); return true;
    case QT_IQ1_S: *fi = info_of<bf::IQ1S>(); return true;
    case QT_IQ1_M: *fi = info_of<bf::IQ1M>(); return true;
    default: return false;
  }
}

static int tiles_of(int M) { return M <= 8 ? 1 : 2; }

// Clusters of Q CTAs, one CTA per SM, that are on the current device at once: a GPC holds whole clusters only, and GPCs differ
// (148 / 74 / 33 / 15 clusters of 1 / 2 / 4 / 8 on the boxes measured).  Asked once per device.
static int clusters_of(int dev, int sm_count, int Q) {
  if (Q == 1) return sm_count;
  static std::atomic<int> known[64][4];
  const int slot = Q == 2 ? 0 : Q == 4 ? 1 : 2;
  int n = dev >= 0 && dev < 64 ? known[dev][slot].load(std::memory_order_acquire) : 0;
  if (n == 0) {
    n = max_clusters(Q);
    if (n < 1) n = sm_count / (2 * Q) > 0 ? sm_count / (2 * Q) : 1;      // no device here (the plan is still a valid one)
    if (dev >= 0 && dev < 64) known[dev][slot].store(n, std::memory_order_release);
  }
  return std::min(n, std::max(1, sm_count / Q));
}

// Work split and shared-memory layout for one launch; false if nothing fits.
static bool plan(const FormatInfo& fi, int64_t N, int64_t K, int M, int dev, int sm_count, Geo* out) {
  const int SB = (int)(K / 256), NT = tiles_of(M), x_block = NT * fi.x_tile;
  Geo best{};
  double best_cost = 1e30;
  for (int nb = 1; nb <= 2; nb++) {
    for (int Q = 1; Q <= 8; Q *= 2) {
      if (Q > sm_count || Q > SB) break;
      for (int P = 1; P <= 16; P++) {
        Geo g{};
        g.nb = nb;
        g.Q = Q;
        g.P = P;
        g.spu = ((SB + Q * P - 1) / (Q * P) + nb - 1) / nb;
        g.chunk_sb = g.spu * nb;
        if (P > 1 && Q * (P - 1) * g.chunk_sb >= SB) continue;         // fewer passes do
        g.RT = (int)((N + 15) / 16);
        g.J = std::min(clusters_of(dev, sm_count, Q), g.RT);
        g.row_skew = (int)((int64_t)SB * fi.ts % 16);
        const int pieces = (16 - std::gcd(fi.ts, 16) + nb * fi.ts + 15) / 16;
        g.pitch = 16 * pieces;
        if (g.pitch % 32 == 0) g.pitch += 16;        // odd multiple of 16: rows fall into different bank groups
        g.slot_bytes = 16 * g.pitch;
        const int tiles = (g.RT + g.J - 1) / g.J, T = tiles * g.spu;
        if ((int64_t)tiles * g.spu * kWarps >= 1ll << 30) continue;
        const int pass_steps = (T + kWarps - 1) / kWarps, warp_steps = pass_steps * P;
        const int tab_bytes = (fi.table_bytes + 15) / 16 * 16, misc = (4 * (g.chunk_sb + 1) + 15) / 16 * 16, sums = (tiles + kWarps) * 512 * NT;
        const int64_t room = (int64_t)tile::kSmemLimit - g.chunk_sb * x_block - tab_bytes - misc - sums - kWarps * kMaxDepth * 8;
        const int fit = room < 0 ? 0 : (int)(room / (kWarps * g.slot_bytes));
        if (fit < std::min(2, warp_steps)) continue;
        g.depth = std::min({fit, kMaxDepth, std::max(warp_steps, 2)});
        g.off_x = kWarps * g.depth * g.slot_bytes;
        g.off_sum = g.off_x + g.chunk_sb * x_block;
        g.off_tab = g.off_sum + sums;
        g.off_misc = g.off_tab + tab_bytes;
        g.off_bar = g.off_misc + misc;
        g.total = g.off_bar + kWarps * kMaxDepth * 8;
        // in units of one block's multiply with one column tile, fitted to timings of 250 shapes, formats and batches with every nb and Q
        // (the split picked takes on average 1.3 % longer than the best of the eight): the busiest warp's steps, staging, a pass, a segment,
        // a cluster, the sums over it
        const double step = nb * (1.0 + 0.125 * (NT - 1)) + 1.25, segs = P * ((double)pass_steps / g.spu + 1.0);
        const double cost = warp_steps * step + P * (g.chunk_sb * 0.183 * NT + 1.23) + segs * 0.85 + (Q > 1 ? 1.8 : 0.0) + Q * 0.45 +
                            tiles * 0.0104 * NT * std::sqrt((double)Q);
        if (cost < best_cost) { best_cost = cost; best = g; }
        break;                                       // more passes only cost more
      }
    }
  }
  if (best_cost >= 1e30) return false;
  *out = best;
  return true;
}

// The plan of a call: worked out once per shape and thread (a microsecond or two, on the host path of calls of 5 us).  The sums of every
// tile stay in shared memory until the end, so a weight of very many rows (from 150 to 500 thousand, by format and columns) is cut into the
// fewest parts of rows that have a plan, a launch each (us at 16 rows, tiled kernel in slices of four rows / here: IQ3_S 256000 x 2048 497 / 149,
// Q3_K 600000 x 2048 1021 / 317; parts that need not be cut are slower, IQ3_S 152064 x 8192 at 8 rows 258 in one, 270 in two).
static bool split(const FormatInfo& fi, int64_t N, int64_t K, int M, int dev, int sm_count, Geo* out) {       // the plan of all parts but the last, which may be shorter
  const int64_t tiles = (N + 15) / 16;
  Geo any;
  if (!plan(fi, 16, K, M, dev, sm_count, &any)) return false;               // no number of rows has one
  for (int64_t parts = 1; parts <= tiles; parts++)
    if (plan(fi, std::min(N, (tiles + parts - 1) / parts * 16), K, M, dev, sm_count, out)) return true;
  return false;
}
static bool plan_of(int qtype, const FormatInfo& fi, int64_t N, int64_t K, int M, int dev, int sm_count, Geo* out) {
  struct Known { int64_t N = 0, K = 0; int qtype = -1, tiles = 0, sms = 0, dev = 0; bool ok = false; Geo geo; };
  static thread_local Known table[64];
  const int tiles = tiles_of(M);
  Known& k = table[((uint64_t)N * 0x9E3779B97F4A7C15ull ^ (uint64_t)K * 0xC2B2AE3D27D4EB4Full ^ (uint64_t)(qtype * 2 + tiles) * 0x165667B19E3779F9ull) >> 58];
  if (k.N != N || k.K != K || k.qtype != qtype || k.tiles != tiles || k.sms != sm_count || k.dev != dev) {
    k.ok = split(fi, N, K, M, dev, sm_count, &k.geo);
    k.N = N; k.K = K; k.qtype = qtype; k.tiles = tiles; k.sms = sm_count; k.dev = dev;
  }
  *out = k.geo;
  return k.ok;
}

}  // namespace batch

bool gemv_batch(int qtype, const uint8_t* w, int64_t N, int64_t K, const void* x, int M, void* y, int y_dtype, int dev, int sm_count, int* status,
                const uint8_t* tab, cudaStream_t st, cudaError_t* result) {
  using namespace batch;
  FormatInfo fi;
  if (!format_of(qtype, &fi)) return false;
  if (M < 1 || M > kMaxBatch || K <= 0 || K % 256 || N < 1 || sm_count < 1) return false;
  if ((uintptr_t)w % 16 || (uintptr_t)x % 16) return false;
  if (N * (K / 256 * fi.ts) >= (1ll << 31)) return false;      // byte offsets are 32-bit
  Geo part;
  if (!plan_of(qtype, fi, N, K, M, dev, sm_count, &part)) return false;
  static const bool want_tma = [] { const char* e = getenv("GGQ_TILE_TMA"); return !(e && e[0] == '0'); }();      // "0": cp.async, as without an encoder
  alignas(64) CUtensorMap map = {};
  Geo geo = part;
  geo.tma = want_tma && geo.row_skew == 0 && make_weight_map(&map, w, N, K / 256 * fi.ts, geo.pitch / 4);
  const Args a{&geo, tiles_of(M), st, w, (int)N, (int)K, x, M, y, y_dtype, tab, status, &map};
  const int tiles = (int)((N + 15) / 16);
  cudaError_t err = cudaSuccess;
  for (; geo.tile0 < tiles && err == cudaSuccess; geo.tile0 += part.RT) {
    geo.RT = std::min(part.RT, tiles - geo.tile0);
    geo.J = std::min(part.J, geo.RT);
    switch (qtype) {
      case QT_IQ4_XS: case QT_IQ2_XXS: case QT_IQ2_XS: case QT_IQ2_S: case QT_IQ3_XXS: case QT_IQ3_S: case QT_IQ1_S: case QT_IQ1_M: err = launch_iq(qtype, a); break;
      default: err = launch_k(qtype, a);
    }
  }
  *result = err;
  return true;
}

}  // namespace ggq
