// Host check of the register pass kernels' shared-memory index maps
// (fft_reg.cuh): for every variant, each point is loaded once from where TMA
// put it, the exchange hands phase 2 the vectors phase 1 wrote, every store
// lands where the TMA store expects it, all accesses stay inside the buffer,
// what is written in place belongs to the warp that read it, and no access
// has bank conflicts.  Prints one line per variant; exit status 1 on a fault.
#include <cstdio>
#include <set>
#include <vector>

#include "../mcfft_b200/csrc/fft_reg.cuh"

using namespace mcfft;
using namespace mcfft::reg;

static int g_bad = 0;
#define CHECK(c, ...)                 \
  do {                                \
    if (!(c)) {                       \
      ++g_bad;                        \
      if (g_bad < 20) {               \
        printf("  line %d: ", __LINE__); \
        printf(__VA_ARGS__);          \
        printf("\n");                 \
      }                               \
    }                                 \
  } while (0)

// Wavefronts of one warp access of `bytes` per lane (8- and 16-byte accesses
// go by half and quarter warps).
static int wavefronts(const std::vector<uint32_t>& a, int bytes) {
  const int lanes = bytes == 4 ? 32 : bytes == 8 ? 16 : 8;
  int total = 0;
  for (size_t p = 0; p < a.size(); p += lanes) {
    std::set<uint32_t> words[32];
    size_t worst = 1;
    for (int i = 0; i < lanes; ++i)
      for (int w = 0; w < bytes / 4; ++w) {
        const uint32_t x = a[p + i] / 4 + w;
        words[x % 32].insert(x);
      }
    for (auto& s : words) worst = s.size() > worst ? s.size() : worst;
    total += (int)worst;
  }
  return total;
}

template <class P>
void check(const char* name) {
  const int bad0 = g_bad;
  const uint32_t in_bytes = P::TP * P::EI, mid_bytes = P::TP * P::EO;
  auto in_at = [](uint32_t pos, uint32_t c) {
    return P::KIND == kCC ? pos * P::RBI + c * P::EI : P::template row_base<P::EI>(pos, c);
  };
  auto out_at = [](uint32_t pos, uint32_t c) -> uint32_t {
    if (P::KIND == kRR) return P::template row_base<P::EO>(pos, c);
    if (P::KIND == kRC) return pos * P::RB + c * P::EO;
    const uint32_t k1 = pos % P::R1, k2 = pos / P::R1;  // rows [k1 high][k2][k1 low]
    return (((k1 >> P::h) * P::R2 + k2) * (1u << P::h) + (k1 & P::m)) * P::RB + c * P::EO;
  };
  int excess = 0;
  std::vector<int> seen(P::TP, 0);
  // slot -> (k1, v, c) after phase 1
  std::vector<int64_t> slot(mid_bytes / P::EO, -1);
  std::vector<int> out_seen(mid_bytes / P::EO, 0);
  for (int w = 0; w < P::NW; ++w) {
    std::set<uint32_t> read, wrote;
    for (int j = 0; j < P::V1; ++j)
      for (int n = 0; n < P::R1; ++n) {
        std::vector<uint32_t> la, sa;
        for (int l = 0; l < 32; ++l) {
          uint32_t v, c;
          P::vec1(w * 32 + l, j, v, c);
          CHECK(v < (uint32_t)P::NV && c < (uint32_t)P::C, "phase 1 vector %u %u", v, c);
          if (P::PK && j) {
            uint32_t v0, c0;
            P::vec1(w * 32 + l, 0, v0, c0);
            CHECK(v0 == v, "packed vectors share their twiddles");
          }
          const uint32_t pos = n * P::NV + v;
          const uint32_t at = (P::load1_base(v, c) ^ P::load1_x(n)) + P::load1_a(n);
          CHECK(at == in_at(pos, c), "load pos %u c %u at %u, staged at %u", pos, c, at, in_at(pos, c));
          CHECK(at + P::EI <= in_bytes && at % P::EI == 0, "load offset %u", at);
          if (at + P::EI <= in_bytes) ++seen[at / P::EI];
          const uint32_t st = (P::store1_base(v, c) ^ P::store1_x(n)) + P::store1_a(n);  // k = n
          CHECK(st + P::EO <= mid_bytes && st % P::EO == 0, "store offset %u", st);
          if (st + P::EO <= mid_bytes) {
            CHECK(slot[st / P::EO] < 0, "slot %u written twice", st);
            slot[st / P::EO] = ((int64_t)n * P::NV + v) * P::C + c;
          }
          read.insert(at);
          wrote.insert(st);
          la.push_back(at);
          sa.push_back(st);
        }
        excess += wavefronts(la, P::EI) - (P::EI == 8 ? 2 : 1) + wavefronts(sa, P::EO) - (P::EO == 8 ? 2 : 1);
      }
    if (P::EI == P::EO) CHECK(read == wrote, "phase 1 of warp %d writes other slots than it read", w);
  }
  for (int s : seen) CHECK(s == 1, "point loaded %d times", s);
  for (int w = 0; w < P::NW; ++w) {
    std::set<uint32_t> read, wrote;
    for (int j = 0; j < P::V2; ++j) {
      for (int i = 0; i < P::R2 / P::LW2; ++i) {
        std::vector<uint32_t> la;
        for (int l = 0; l < 32; ++l) {
          uint32_t k1, c;
          P::vec2(w * 32 + l, j, k1, c);
          CHECK(k1 < (uint32_t)P::R1 && c < (uint32_t)P::C, "phase 2 vector %u %u", k1, c);
          const uint32_t at = (P::load2_base(k1, c) ^ P::load2_x(i)) + P::load2_a(i);
          CHECK(at % (P::EO * P::LW2) == 0 && at + P::EO * P::LW2 <= mid_bytes, "load offset %u", at);
          for (int u = 0; u < P::LW2 && at + P::EO * P::LW2 <= mid_bytes; ++u) {
            const int64_t want = ((int64_t)k1 * P::NV + i * P::LW2 + u) * P::C + c;
            CHECK(slot[at / P::EO + u] == want, "phase 2 reads %lld for %lld", (long long)slot[at / P::EO + u],
                  (long long)want);
            read.insert(at + u * P::EO);
          }
          la.push_back(at);
        }
        const int b = P::EO * P::LW2;
        excess += wavefronts(la, b) - (b == 16 ? 4 : b == 8 ? 2 : 1);
      }
      for (int k = 0; k < P::R2; ++k) {
        std::vector<uint32_t> sa;
        for (int l = 0; l < 32; ++l) {
          uint32_t k1, c;
          P::vec2(w * 32 + l, j, k1, c);
          const uint32_t st = (P::store2_base(k1, c) ^ P::store2_x(k)) + P::store2_a(k);
          const uint32_t pos = k1 + P::R1 * k;
          CHECK(st == out_at(pos, c), "output pos %u c %u at %u, stored from %u", pos, c, st, out_at(pos, c));
          CHECK(st + P::EO <= mid_bytes && st % P::EO == 0, "store offset %u", st);
          if (st + P::EO <= mid_bytes) ++out_seen[st / P::EO];
          wrote.insert(st);
          sa.push_back(st);
        }
        excess += wavefronts(sa, P::EO) - (P::EO == 8 ? 2 : 1);
      }
    }
    if (P::KIND != kRC) CHECK(read == wrote, "phase 2 of warp %d writes other slots than it read", w);
  }
  for (int s : out_seen) CHECK(s == 1, "output slot written %d times", s);
  CHECK(excess == 0, "%d wavefronts of bank conflicts", excess);
  printf("%s %s (excess wavefronts %d)\n", g_bad == bad0 ? "ok" : "FAULT", name, excess);
}

#define V(L, R1, R2, TP, I, O, K, PT) check<RegPass<L, R1, R2, TP, I, O, K, PT, false>>(#L " " #R1 "x" #R2 " " #TP " " #I " " #O " " #K)
#define ROWS(TP, I, O, K)                                                              \
  V(64, 8, 8, TP, I, O, K, false), V(128, 8, 16, TP, I, O, K, false), V(256, 16, 16, TP, I, O, K, false), \
      V(512, 16, 32, TP, I, O, K, false), V(1024, 32, 32, TP, I, O, K, false)

int main() {
  ROWS(16384, true, true, kRR);
  ROWS(16384, true, true, kRC);
  V(64, 8, 8, 16384, true, true, kCC, false);
  V(128, 16, 8, 16384, true, true, kCC, false);
  V(256, 16, 16, 16384, true, true, kCC, false);
  V(512, 32, 16, 16384, true, true, kCC, true);
  V(1024, 32, 32, 16384, true, true, kCC, true);
  ROWS(8192, false, false, kRR);
  ROWS(8192, false, false, kRC);
  ROWS(8192, true, false, kRR);
  V(64, 8, 8, 8192, false, false, kCC, false);
  V(128, 8, 16, 8192, false, false, kCC, false);
  V(256, 16, 16, 8192, false, false, kCC, false);
  V(512, 32, 16, 8192, false, false, kCC, false);
  V(1024, 32, 32, 8192, false, false, kCC, false);
  V(64, 8, 8, 8192, true, false, kCC, true);
  V(128, 8, 16, 8192, true, false, kCC, true);
  V(256, 16, 16, 8192, true, false, kCC, true);
  V(512, 32, 16, 8192, true, false, kCC, true);
  V(1024, 32, 32, 8192, true, false, kCC, true);
  return g_bad ? 1 : 0;
}
