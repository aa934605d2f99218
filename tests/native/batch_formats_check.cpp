// Host-side check of gguf_jax_b200/csrc/batch_formats.cuh: for every run and octet of random blocks, the scaled operands (all planes),
// the activation order and the block's float scales must reproduce the decoded weights (given by the Python test) bit for bit.
//
// usage: batch_formats_check <qtype> <blocks.bin> <decoded_f32.bin> <table.bin> <n_blocks>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../gguf_jax_b200/csrc/batch_formats.cuh"

using namespace ggq;

static std::vector<uint8_t> slurp(const char* path) {
  FILE* f = fopen(path, "rb");
  if (!f) { fprintf(stderr, "cannot open %s\n", path); exit(2); }
  fseek(f, 0, SEEK_END);
  long n = ftell(f);
  fseek(f, 0, SEEK_SET);
  std::vector<uint8_t> v(n);
  if (fread(v.data(), 1, n, f) != (size_t)n) exit(2);
  fclose(f);
  return v;
}

template <class F>
int check(const std::vector<uint8_t>& blocks, const float* want, const tf::Tables& tb, int nb) {
  typedef typename F::Base B;
  long bad = 0, seen = 0;
  for (int b = 0; b < nb; b++) {
    std::vector<int> cover(256, 0);
    // the kernel sees blocks at addresses of the format's alignment: give the loader exactly that; this block as the first and as the
    // second row of a pair
    std::vector<uint8_t> buf(2 * (B::kTs + 48));
    uint8_t *p = buf.data() + 2 * (b % 3), *other = buf.data() + B::kTs + 48;
    if ((uintptr_t)p % B::kAlign) p += B::kAlign - (uintptr_t)p % B::kAlign;
    if ((uintptr_t)other % B::kAlign) other += B::kAlign - (uintptr_t)other % B::kAlign;
    memcpy(p, blocks.data() + (size_t)b * B::kTs, B::kTs);
    memcpy(other, blocks.data() + (size_t)(nb - 1 - b) * B::kTs, B::kTs);
    for (int t = 0; t < 4; t++) {
      typename F::Run pair[2];
      if (b & 1) bf::load_pair<F>(tf::BlockLd{other}, tf::BlockLd{p}, t, pair[1], pair[0]);
      else bf::load_pair<F>(tf::BlockLd{p}, tf::BlockLd{other}, t, pair[0], pair[1]);
      const typename F::Run& run = pair[0];
      for (int q = 0; q < 8; q++) {
        uint32_t pa[4], pb[4] = {0, 0, 0, 0};
        F::octet(run, q, tb, pa, pb);
        int qa, qb;
        F::src_quads(t, q, qa, qb);
        for (int i = 0; i < 4; i++)
          for (int h = 0; h < 2; h++) {
            const int e = B::kPairOrder == 0 ? (i < 2 ? qa : qb) + (i & 1) + 2 * h : (h ? qb : qa) + i;
            cover[e]++;
            const double code = (double)bf::half_at(pa[i], h) + (F::kPlanes == 2 ? bf::half_at(pb[i], h) : 0.0f);
            float v = tf::fmaf_(run.d, (float)std::ldexp(code, bf::kExp), 0.0f);
            if constexpr (F::kMins > 0) {
              const int grp = q * F::kMins / 8;
              v = tf::fmaf_(run.nd, bf::bhalf_at(run.mn[grp / 2], grp & 1), v);
            }
            const float ref = want[(size_t)b * 256 + e];
            seen++;
            if (!(v == ref) && !(std::isnan(v) && std::isnan(ref))) {
              if (bad < 10) fprintf(stderr, "block %d run %d octet %d weight %d: got %.9g want %.9g\n", b, t, q, e, v, ref);
              bad++;
            }
          }
      }
    }
    for (int i = 0; i < 256; i++)
      if (cover[i] != 1) { fprintf(stderr, "block %d: weight %d covered %d times\n", b, i, cover[i]); return 1; }
  }
  printf("qtype %d: %ld values checked, %ld mismatches\n", B::kQt, seen, bad);
  return bad ? 1 : 0;
}

int main(int argc, char** argv) {
  if (argc != 6) { fprintf(stderr, "usage: %s qtype blocks decoded table n_blocks\n", argv[0]); return 2; }
  const int qt = atoi(argv[1]), nb = atoi(argv[5]);
  const std::vector<uint8_t> blocks = slurp(argv[2]), dec = slurp(argv[3]), table = slurp(argv[4]);
  const float* want = reinterpret_cast<const float*>(dec.data());
  tf::Tables tb{};
  tb.grid = table.data();
  if (table.size() == 16) memcpy(tb.kv, table.data(), 16);
  switch (qt) {
    case tf::Q2K::kQt: return check<bf::Q2K>(blocks, want, tb, nb);
    case tf::Q3K::kQt: return check<bf::Q3K>(blocks, want, tb, nb);
    case tf::Q4K::kQt: return check<bf::Q4K>(blocks, want, tb, nb);
    case tf::Q5K::kQt: return check<bf::Q5K>(blocks, want, tb, nb);
    case tf::Q6K::kQt: return check<bf::Q6K>(blocks, want, tb, nb);
    case tf::IQ4XS::kQt: return check<bf::IQ4XS>(blocks, want, tb, nb);
    case tf::IQ2XXS::kQt: return check<bf::IQ2XXS>(blocks, want, tb, nb);
    case tf::IQ2XS::kQt: return check<bf::IQ2XS>(blocks, want, tb, nb);
    case tf::IQ2S::kQt: return check<bf::IQ2S>(blocks, want, tb, nb);
    case tf::IQ3XXS::kQt: return check<bf::IQ3XXS>(blocks, want, tb, nb);
    case tf::IQ3S::kQt: return check<bf::IQ3S>(blocks, want, tb, nb);
    case tf::IQ1S::kQt: return check<bf::IQ1S>(blocks, want, tb, nb);
    case tf::IQ1M::kQt: return check<bf::IQ1M>(blocks, want, tb, nb);
    case tf::TQ10::kQt: return check<bf::TQ10>(blocks, want, tb, nb);
    case tf::TQ20::kQt: return check<bf::TQ20>(blocks, want, tb, nb);
  }
  fprintf(stderr, "no batch format for qtype %d\n", qt);
  return 2;
}
