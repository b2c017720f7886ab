// Host check of the register pass kernels' shared-memory index maps
// (fft_reg.cuh): for every variant, each point is loaded once from where TMA
// put it, the exchange hands phase 2 the vectors phase 1 wrote, every store
// lands where the TMA store expects it, all accesses stay inside the buffer,
// what is written in place belongs to the warp that read it, and no access
// has bank conflicts.  Where TMA puts or takes a point is worked out from the
// tensor-map dimensions, not from the kernels' own formulas.  Prints one line
// per variant; exit status 1 on a fault.
#include <cstdio>
#include <set>
#include <vector>

#include "../mcfft_b200/csrc/fft_mma.cuh"
#include "../mcfft_b200/csrc/fft_rows.cuh"
#include "../mcfft_b200/csrc/reg_staging.h"

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

// Byte of (pos, c) in shared memory as the tensor map's box places it (the box
// of tile 0 over a pass of C columns): index pos * C + c.
static std::vector<uint32_t> tma_place(const layout::Staging& s, bool row) {
  std::vector<uint32_t> at((size_t)s.L * s.C, ~0u);
  uint64_t n = 1;
  for (int d = 0; d < s.ndims; ++d) n *= s.box[d];
  CHECK(s.ndims >= 3 && s.ndims <= 5 && n == at.size(), "box of %llu points", (unsigned long long)n);
  for (uint64_t i = 0; i < n; ++i) {
    uint64_t r = i, g = 0;
    for (int d = 0; d < s.ndims; ++d) {
      const uint64_t x = r % s.box[d];
      r /= s.box[d];
      CHECK(s.box[d] <= 256, "box dimension %u", s.box[d]);
      g += x * (d ? s.gstride_bytes[d] / s.elem : 1);
    }
    const uint64_t pos = row ? g % s.L : g / s.C, c = row ? g / s.L : g % s.C;
    CHECK(pos < (uint64_t)s.L && c < (uint64_t)s.C, "element %llu", (unsigned long long)g);
    uint32_t off = (uint32_t)(i * s.elem);
    off ^= ((off >> 7) & s.swz) << 4;
    if (pos < (uint64_t)s.L && c < (uint64_t)s.C) at[pos * s.C + c] = off;
  }
  for (uint32_t a : at) CHECK(a != ~0u, "a point outside the box");
  return at;
}

// The kernels without TMA copy 16 bytes of a transform to where TMA would
// (in_map, out_map: the inverse of the tensor map's placement).
template <class P>
void check_maps(const RegShape& sh, const char* name) {
  const int bad0 = g_bad;
  for (int out = 0; out < 2; ++out) {
    const uint32_t e = out ? P::EO : P::EI;
    const auto at = tma_place(out ? reg_staging_out(sh, layout::ROW, layout::ROW, e, 1, P::L, 0, P::C, 1)
                                  : reg_staging_in(sh, layout::ROW, e, 1, P::L, 0, P::C, 1), true);
    for (uint32_t c = 0; c < P::C; ++c)
      for (uint32_t p = 0; p < P::L; ++p) {
        const uint32_t x = at[p * P::C + c], a = x & ~15u;
        CHECK((out ? P::out_map(a) : P::in_map(a)) + (x & 15u) == (c * P::L + p) * e, "byte %u", x);
      }
  }
  printf("%s %s maps\n", g_bad == bad0 ? "ok" : "FAULT", name);
}

template <class P>
void check(const char* name) {
  const int bad0 = g_bad;
  const uint32_t in_bytes = P::TP * P::EI, mid_bytes = P::TP * P::EO;
  const RegShape sh{P::L, P::R1, P::C, P::h, false};
  const layout::Kind ik = P::KIND == kCC ? layout::COL : layout::ROW, ok = P::KIND == kRR ? layout::ROW : layout::COL;
  const bool ri = ik == layout::ROW, ro = ok == layout::ROW;
  const auto tin = tma_place(reg_staging_in(sh, ik, P::EI, ri ? 1 : P::C, ri ? P::L : 1, 0, P::C, 1), ri);
  const auto tout = tma_place(reg_staging_out(sh, ik, ok, P::EO, ro ? 1 : P::C, ro ? P::L : 1, 0, P::C, 1), ro);
  auto in_at = [&](uint32_t pos, uint32_t c) { return tin[pos * P::C + c]; };
  auto out_at = [&](uint32_t pos, uint32_t c) { return tout[pos * P::C + c]; };
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

template <class M>
void check_mma(const char* name) {
  const int bad0 = g_bad;
  const uint32_t bytes = M::TP * 4;
  const RegShape sh{M::L, M::R, M::C, 0, true};
  const layout::Kind ik = M::KIND == kCC ? layout::COL : layout::ROW, ok = M::KIND == kRR ? layout::ROW : layout::COL;
  const bool ri = ik == layout::ROW, ro = ok == layout::ROW;
  const auto tin = tma_place(reg_staging_in(sh, ik, 4, ri ? 1 : M::C, ri ? M::L : 1, 0, M::C, 1), ri);
  const auto tout = tma_place(reg_staging_out(sh, ik, ok, 4, ro ? 1 : M::C, ro ? M::L : 1, 0, M::C, 1), ro);
  auto at = [&](uint32_t t, uint32_t r) { return (t ^ (r & M::XM)) + (r & ~M::XM); };
  int excess = 0;
  std::vector<int> seen(M::TP, 0), out_seen(M::TP, 0);
  std::vector<int64_t> slot(M::TP, -1);
  auto tag = [](uint32_t k1, uint32_t v, uint32_t c) { return ((int64_t)k1 * M::NV + v) * M::C + c; };
  for (uint32_t w = 0; w < (uint32_t)M::NW; ++w) {
    std::set<uint32_t> read, wrote;
    for (uint32_t h = 0; h < 2; ++h)
      for (uint32_t i = 0; i < 4; ++i) {
        std::vector<uint32_t> la;
        for (uint32_t l = 0; l < 32; ++l) {
          const uint32_t x = at(M::load1_t(l, w), M::load1_r(h, i));
          CHECK(x % 16 == 0 && x + 16 <= bytes, "load %u", x);
          for (uint32_t u = 0; u < 4; ++u) {
            const auto a = M::p1(l >> 2, h, u, w);
            const uint32_t pos = ((l & 3) + 4 * i) * M::NV + a.v;
            CHECK(a.v < (uint32_t)M::NV && a.c < (uint32_t)M::C, "vector %u %u", a.v, a.c);
            CHECK(tin[pos * M::C + a.c] == x + 4 * u, "point %u %u staged at %u, read at %u", pos, a.c,
                  tin[pos * M::C + a.c], x + 4 * u);
            ++seen[pos * M::C + a.c];
            read.insert(x + 4 * u);
          }
          la.push_back(x);
        }
        excess += wavefronts(la, 16) - 4;
      }
    // stores: chunk words are the four w, or (h, p) where phase 2 reads operand slots
    for (uint32_t mt = 0; mt < 2; ++mt)
      for (uint32_t x = 0; x < 4; ++x) {  // (p, h), or w
        std::vector<uint32_t> sa;
        for (uint32_t l = 0; l < 32; ++l) {
          const uint32_t d = M::WK ? M::store1_r(mt, 0, 0, x) : M::store1_r(mt, x & 1, x >> 1, 0);
          const uint32_t s = at(M::store1_t(l, w), d);
          CHECK(s % 16 == 0 && s + 16 <= bytes, "store %u", s);
          for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t p = M::WK ? u >> 1 : x & 1, h = M::WK ? u & 1 : x >> 1, ww = M::WK ? x : u;
            const auto a = M::p1((l & 3) << 1 | p, h, ww, w);
            const uint32_t k1 = (l >> 2) + 8 * mt;
            CHECK(slot[s / 4 + u] < 0, "slot written twice");
            CHECK(M::ex_at(k1, a.v, a.c) == s + 4 * u, "exchange address");
            slot[s / 4 + u] = tag(k1, a.v, a.c);
            wrote.insert(s + 4 * u);
          }
          sa.push_back(s);
        }
        excess += wavefronts(sa, 16) - 4;
      }
    CHECK(read == wrote, "phase 1 of warp %u writes other slots than it read", w);
  }
  for (int x : seen) CHECK(x == 1, "point loaded %d times", x);
  for (uint32_t w = 0; w < (uint32_t)M::NW; ++w) {
    std::set<uint32_t> read, wrote;
    for (uint32_t j = 0; j < 8; ++j) {
      std::vector<uint32_t> la;
      for (uint32_t l = 0; l < 32; ++l) {
        const uint32_t x = at(M::load2_t(l, w), M::load2_r(j));
        CHECK(x % 16 == 0 && x + 16 <= bytes, "load %u", x);
        for (uint32_t u = 0; u < 4 && x + 16 <= bytes; ++u) {
          const uint32_t unit = M::WK ? j : (j >> 2) * 4 + u, i = M::WK ? u : j & 3;
          const auto a = M::p2(l >> 2, unit, w);
          CHECK(a.k1 < 16 && a.n3 < (uint32_t)M::R && a.c < (uint32_t)M::C, "phase 2 vector");
          const int64_t want = tag(a.k1, M::v_of((l & 3) + 4 * i, a.n3), a.c);
          CHECK(slot[x / 4 + u] == want, "phase 2 reads %lld for %lld", (long long)slot[x / 4 + u], (long long)want);
          read.insert(x + 4 * u);
        }
        la.push_back(x);
      }
      excess += wavefronts(la, 16) - 4;
    }
    // outputs, chunk by chunk as run() stores them
    auto put = [&](uint32_t d, auto who) {  // who(word) -> (mt, p, unit, k3)
      std::vector<uint32_t> sa;
      for (uint32_t l = 0; l < 32; ++l) {
        const uint32_t s = at(M::store2_t(l, w), d);
        CHECK(s % 16 == 0 && s + 16 <= bytes, "store %u", s);
        for (uint32_t u = 0; u < 4 && s + 16 <= bytes; ++u) {
          uint32_t mt, p, unit, k3;
          who(u, mt, p, unit, k3);
          const auto a = M::p2((l & 3) << 1 | p, unit, w);
          const uint32_t pos = a.k1 + 16 * ((l >> 2) + 8 * mt) + 256 * k3;
          CHECK(tout[pos * M::C + a.c] == s + 4 * u, "output %u %u taken from %u, stored at %u", pos, a.c,
                tout[pos * M::C + a.c], s + 4 * u);
          ++out_seen[pos * M::C + a.c];
          wrote.insert(s + 4 * u);
        }
        sa.push_back(s);
      }
      excess += wavefronts(sa, 16) - 4;
    };
    for (uint32_t mt = 0; mt < 2; ++mt)
      for (uint32_t x = 0; x < 4; ++x) {
        if (M::L == 256 && M::KIND == kCC)
          put(M::store2_r(mt, x & 1, 4 * (x >> 1), 0), [&](uint32_t u, uint32_t& m, uint32_t& p, uint32_t& un, uint32_t& k3) {
            m = mt, p = x & 1, un = u + 4 * (x >> 1), k3 = 0;
          });
        else if (M::L == 256)
          put(M::store2_r(mt, 0, 2 * x, 0), [&](uint32_t u, uint32_t& m, uint32_t& p, uint32_t& un, uint32_t& k3) {
            m = mt, p = u & 1, un = 2 * x + (u >> 1), k3 = 0;
          });
        else if (M::L == 512)
          put(M::store2_r(mt, x & 1, 0, x >> 1), [&](uint32_t u, uint32_t& m, uint32_t& p, uint32_t& un, uint32_t& k3) {
            m = mt, p = x & 1, un = M::KIND == kCC ? u : 2 * u, k3 = x >> 1;
          });
        else
          put(M::store2_r(mt, 0, 0, x), [&](uint32_t u, uint32_t& m, uint32_t& p, uint32_t& un, uint32_t& k3) {
            m = mt, p = M::KIND == kCC ? 0 : u & 1, un = M::KIND == kCC ? u : 4 * (u >> 1), k3 = x;
          });
      }
    if (M::KIND == kRR) CHECK(read == wrote, "phase 2 of warp %u writes other slots than it read", w);
  }
  for (int x : out_seen) CHECK(x == 1, "output written %d times", x);
  CHECK(excess == 0, "%d wavefronts of bank conflicts", excess);
  // twiddle tables: every entry set, unit modulus (phase 1)
  std::vector<float> tab(M::TWB / 4, 7.f);
  M::fill_twiddles(tab.data());
  for (size_t i = 0; i < tab.size(); i += 4)
    for (int p = 0; p < 2; ++p) {
      const double r = (double)tab[i + p] * tab[i + p] + (double)tab[i + 2 + p] * tab[i + 2 + p];
      const double want = i * 4 < (size_t)M::TW1B ? 1.0 : 1.0 / M::R / M::R;
      CHECK(r > want * 0.999 && r < want * 1.001, "twiddle entry %zu", i / 4);
    }
  printf("%s tensor cores %s (excess wavefronts %d)\n", g_bad == bad0 ? "ok" : "FAULT", name, excess);
}

// 4096-point rows, plain form: the three phases' chunks.
static void check_mma4096() {
  using M = Mma4096<false>;
  const int bad0 = g_bad;
  const RegShape sh{4096, 16, 1, 0, true};
  const auto tin = tma_place(reg_staging_in(sh, layout::ROW, 4, 1, 4096, 0, 1, 1), true);
  const auto tout = tma_place(reg_staging_out(sh, layout::ROW, layout::ROW, 4, 1, 4096, 0, 1, 1), true);
  auto at = [&](uint32_t t, uint32_t r) { return (t ^ (r & M::XM)) + (r & ~M::XM); };
  int excess = 0;
  std::vector<int> slot1(4096, -1), slot2(4096, -1), out(4096, 0), seen(4096, 0);
  auto chunk = [&](uint32_t w, auto addr, auto word) {  // one access of warp w
    std::vector<uint32_t> a;
    for (uint32_t l = 0; l < 32; ++l) {
      const uint32_t x = addr(l);
      CHECK(x % 16 == 0 && x + 16 <= 16384, "access %u", x);
      for (uint32_t u = 0; u < 4 && x + 16 <= 16384; ++u) word(l, u, x / 4 + u);
      a.push_back(x);
    }
    (void)w;
    excess += wavefronts(a, 16) - 4;
  };
  for (uint32_t w = 0; w < 4; ++w) {
    std::set<uint32_t> rd, wr;
    for (uint32_t j = 0; j < 8; ++j)
      chunk(w, [&](uint32_t l) { return at(M::load1_t(l, w), M::load1_r(j >> 2, j & 3)); },
            [&](uint32_t l, uint32_t u, uint32_t s) {
              const auto a = M::p1(l >> 2, j >> 2, u, w);
              const uint32_t pos = ((l & 3) + 4 * (j & 3)) * 256 + a.x * 16 + a.y;
              CHECK(tin[pos] == 4 * s, "point %u", pos);
              ++seen[pos];
              rd.insert(s);
            });
    for (uint32_t e = 0; e < 8; ++e)
      chunk(w, [&](uint32_t l) { return at(M::store1_t(l, w), M::store1_r(e & 1, (e >> 1) & 1, e >> 2)); },
            [&](uint32_t l, uint32_t u, uint32_t s) {
              const auto a = M::p1((l & 3) << 1 | ((e >> 1) & 1), e >> 2, u, w);
              CHECK(slot1[s] < 0, "slot written twice");
              slot1[s] = (int)(((l >> 2) + 8 * (e & 1)) * 256 + a.x * 16 + a.y);
              wr.insert(s);
            });
    CHECK(rd == wr, "phase 1 leaves its slots");
  }
  for (uint32_t w = 0; w < 4; ++w) {
    std::set<uint32_t> rd, wr;
    for (uint32_t j = 0; j < 8; ++j)
      chunk(w, [&](uint32_t l) { return at(M::load2_t(l, w), M::load2_r(j >> 2, j & 3)); },
            [&](uint32_t l, uint32_t u, uint32_t s) {
              const auto a = M::p2(l >> 2, j >> 2, u, w);
              CHECK(slot1[s] == (int)(a.x * 256 + ((l & 3) + 4 * (j & 3)) * 16 + a.y), "phase 2 load");
              rd.insert(s);
            });
    for (uint32_t e = 0; e < 8; ++e)
      chunk(w, [&](uint32_t l) { return at(M::store2_t(l, w), M::store2_r(e & 1, e >> 1)); },
            [&](uint32_t l, uint32_t u, uint32_t s) {  // words: h + 2 p is n3's upper half, stored as p + 2 h
              const auto a = M::p2((l & 3) << 1 | (u & 1), u >> 1, e >> 1, w);
              CHECK(slot2[s] < 0, "slot written twice");
              slot2[s] = (int)(a.x * 256 + ((l >> 2) + 8 * (e & 1)) * 16 + a.y);
              wr.insert(s);
            });
    CHECK(rd == wr, "phase 2 leaves its slots");
  }
  for (uint32_t w = 0; w < 4; ++w) {
    for (uint32_t j = 0; j < 8; ++j)
      chunk(w, [&](uint32_t l) { return at(M::load3_t(l, w), M::load3_r(j)); },
            [&](uint32_t l, uint32_t u, uint32_t s) {
              const auto a = M::p3(l >> 2, j, w);
              CHECK(slot2[s] == (int)(a.x * 256 + a.y * 16 + (l & 3) + 4 * u), "phase 3 load");
            });
    for (uint32_t e = 0; e < 8; ++e)
      chunk(w, [&](uint32_t l) { return at(M::store3_t(l, w), M::store3_r(e & 1, e >> 1 << 1)); },
            [&](uint32_t l, uint32_t u, uint32_t s) {
              const auto a = M::p3((l & 3) << 1 | (u & 1), (e >> 1 << 1) | u >> 1, w);
              const uint32_t pos = a.x + 16 * a.y + 256 * ((l >> 2) + 8 * (e & 1));
              CHECK(tout[pos] == 4 * s, "output %u", pos);
              ++out[pos];
            });
  }
  for (int i = 0; i < 4096; ++i) CHECK(seen[i] == 1 && out[i] == 1, "point %d: %d loads, %d stores", i, seen[i], out[i]);
  CHECK(excess == 0, "%d wavefronts of bank conflicts", excess);
  printf("%s 4096-point rows, plain\n", g_bad == bad0 ? "ok" : "FAULT");
}

// 2048-point rows, plain form.
static void check_mma2048() {
  using M = Mma2048<false>;
  const int bad0 = g_bad;
  const RegShape sh{2048, 8, 8, 0, true};
  const auto tin = tma_place(reg_staging_in(sh, layout::ROW, 4, 1, 2048, 0, 8, 1), true);
  const auto tout = tma_place(reg_staging_out(sh, layout::ROW, layout::ROW, 4, 1, 2048, 0, 8, 1), true);
  auto at = [&](uint32_t t, uint32_t r) { return (t ^ (r & M::XM)) + (r & ~M::XM); };
  int excess = 0;
  for (uint32_t c = 0; c < 8; ++c) {
    std::vector<int> slot(2048, -1), out(2048, 0), seen(2048, 0);
    for (uint32_t w = 0; w < 2; ++w) {
      std::set<uint32_t> rd, wr;
      for (uint32_t j = 0; j < 8; ++j) {
        std::vector<uint32_t> la;
        for (uint32_t l = 0; l < 32; ++l) {
          const uint32_t x = at(M::load1_t(l, w), M::load1_r(j >> 2, j & 3));
          CHECK(x % 16 == 0 && x + 16 <= 8192, "access %u", x);
          for (uint32_t u = 0; u < 4 && x + 16 <= 8192; ++u) {
            const auto a = M::p1(l >> 2, j >> 2, u, w);
            const uint32_t pos = ((l & 3) + 4 * (j & 3)) * 128 + a.x * 8 + a.y;
            CHECK(tin[pos * 8 + c] == c * 8192 + x + 4 * u, "point %u", pos);
            ++seen[pos];
            rd.insert(x + 4 * u);
          }
          la.push_back(x);
        }
        excess += wavefronts(la, 16) - 4;
      }
      for (uint32_t e = 0; e < 8; ++e) {
        std::vector<uint32_t> sa;
        for (uint32_t l = 0; l < 32; ++l) {
          const uint32_t x = at(M::store1_t(l, w), M::store1_r(e & 1, (e >> 1) & 1, e >> 2));
          CHECK(x % 16 == 0 && x + 16 <= 8192, "access %u", x);
          for (uint32_t u = 0; u < 4 && x + 16 <= 8192; ++u) {
            const auto a = M::p1((l & 3) << 1 | ((e >> 1) & 1), e >> 2, u, w);
            CHECK(slot[x / 4 + u] < 0, "slot written twice");
            slot[x / 4 + u] = (int)(((l >> 2) + 8 * (e & 1)) * 128 + a.x * 8 + a.y);
            wr.insert(x + 4 * u);
          }
          sa.push_back(x);
        }
        excess += wavefronts(sa, 16) - 4;
      }
      CHECK(rd == wr, "phase 1 leaves its slots");
    }
    for (uint32_t w = 0; w < 2; ++w) {
      for (uint32_t j = 0; j < 8; ++j) {
        std::vector<uint32_t> la;
        for (uint32_t l = 0; l < 32; ++l) {
          const uint32_t x = at(M::load2_t(l, w), M::load2_r(j >> 2, j & 3));
          CHECK(x % 16 == 0 && x + 16 <= 8192, "access %u", x);
          for (uint32_t u = 0; u < 4 && x + 16 <= 8192; ++u) {
            const auto a = M::p2(l >> 2, j >> 2, u, w);
            CHECK(slot[x / 4 + u] == (int)(a.x * 128 + ((l & 3) + 4 * (j & 3)) * 8 + a.y), "phase 2 load");
          }
          la.push_back(x);
        }
        excess += wavefronts(la, 16) - 4;
      }
      for (uint32_t e = 0; e < 16; ++e) {
        std::vector<uint32_t> sa;
        for (uint32_t l = 0; l < 32; ++l) {
          const uint32_t x = at(M::store2_t(l, w), M::store2_r(e & 1, e >> 1));
          CHECK(x % 8 == 0 && x + 8 <= 8192, "access %u", x);
          for (uint32_t p = 0; p < 2 && x + 8 <= 8192; ++p) {
            const auto a = M::p2((l & 3) << 1 | p, 0, 0, w);
            const uint32_t pos = a.x + 16 * ((l >> 2) + 8 * (e & 1)) + 256 * (e >> 1);
            CHECK(tout[pos * 8 + c] == c * 8192 + x + 4 * p, "output %u", pos);
            ++out[pos];
          }
          sa.push_back(x);
        }
        excess += wavefronts(sa, 8) - 2;
      }
    }
    for (int i = 0; i < 2048; ++i) CHECK(seen[i] == 1 && out[i] == 1, "point %d: %d loads, %d stores", i, seen[i], out[i]);
  }
  CHECK(excess == 0, "%d wavefronts of bank conflicts", excess);
  printf("%s 2048-point rows, plain\n", g_bad == bad0 ? "ok" : "FAULT");
}

// Transforms copied one by one land where a tile's own box would put them.
static void check_gather(int L, int R) {
  const int bad0 = g_bad, C = 16384 / L;
  const RegShape sh{L, R, C, 0, true};
  const std::vector<int64_t> offs{0, 3 * int64_t(L), L + 32};
  for (int out = 0; out < 2; ++out) {
    const auto want = tma_place(out ? reg_staging_out(sh, layout::ROW, layout::ROW, 4, 1, L, 0, C, 1)
                                    : reg_staging_in(sh, layout::ROW, 4, 1, L, 0, C, 1), true);
    layout::Staging g;
    std::vector<int32_t> tab;
    CHECK(reg_gather_staging(sh, out, 4, offs, &g, &tab) && tab.size() == offs.size() && g.ndims == 3, "no map");
    CHECK((int)(g.box[0] * g.box[1] * g.box[2]) == L, "box");
    for (size_t t = 0; t < offs.size(); ++t) {
      CHECK((uint64_t)tab[t] + g.box[2] <= g.gdim[2], "row %d outside the map", tab[t]);
      for (int c = 0; c < C; ++c)  // column c at byte c L 4 of the buffer
        for (int i = 0; i < L; ++i) {
          const int64_t x = i % g.box[0], y = i / g.box[0] % g.box[1], z = i / (g.box[0] * g.box[1]);
          const int64_t e = x + y * (int64_t)g.gstride_bytes[1] / 4 + (tab[t] + z) * (int64_t)g.gstride_bytes[2] / 4;
          uint32_t off = (uint32_t)(c * L + i) * 4;
          off ^= ((off >> 7) & g.swz) << 4;
          const int64_t pos = e - offs[t];
          CHECK(pos >= 0 && pos < L && want[pos * C + c] == off, "point %lld", (long long)pos);
        }
    }
  }
  layout::Staging g;
  std::vector<int32_t> tab;
  CHECK(!reg_gather_staging(sh, false, 4, {16}, &g, &tab), "offset of half a row");
  printf("%s %d-point gathered rows\n", g_bad == bad0 ? "ok" : "FAULT", L);
}

// 4096-point rows, FP32 exchange.
static void check_reg4096() {
  using M = Reg4096<false, false>;
  const int bad0 = g_bad;
  const RegShape sh{4096, 16, 1, 0, false};
  const auto tin = tma_place(reg_staging_in(sh, layout::ROW, 8, 1, 4096, 0, 1, 1), true);
  for (uint32_t p = 0; p < 4096; ++p) CHECK(tin[p] == 8 * p, "natural order");
  int excess = 0;
  std::vector<int> n1(4096, 0), out(4096, 0), slot(4096, -1);
  for (uint32_t w = 0; w < 4; ++w)
    for (uint32_t j = 0; j < 2; ++j)
      for (uint32_t k = 0; k < 16; ++k) {
        std::vector<uint32_t> a, b, c, d;
        for (uint32_t l = 0; l < 32; ++l) {
          const uint32_t t = w * 32 + l, x = M::xd(t), y = M::yd(t, j);
          a.push_back((k * 256 + y * 16 + x) * 8);            // phase 1 in and out, phase 3 out
          b.push_back((y * 256 + k * 16 + x) * 8);            // phase 2 in
          c.push_back(M::ex2_at(y, k, x));                    // phase 2 out
          CHECK(c.back() == M::ex2_at(y, 0, x) + k * 128, "phase 2 store offset");
          ++n1[a.back() / 8];
          ++out[a.back() / 8];
          CHECK(slot[c.back() / 8] < 0 && c.back() / 128 == b.back() / 128, "phase 2 slot");
          slot[c.back() / 8] = (int)(y * 256 + k * 16 + x);
        }
        excess += wavefronts(a, 8) - 2 + wavefronts(b, 8) - 2 + wavefronts(c, 8) - 2;
      }
  for (uint32_t w = 0; w < 4; ++w)
    for (uint32_t j = 0; j < 2; ++j)
      for (uint32_t n = 0; n < 8; ++n) {
        std::vector<uint32_t> a;
        for (uint32_t l = 0; l < 32; ++l) {
          const uint32_t t = w * 32 + l, k1 = M::xd(t), k2 = M::yd(t, j), x = M::ex2_at(k1, k2, 0) ^ (n << 4);
          for (uint32_t u = 0; u < 2; ++u)
            CHECK(slot[x / 8 + u] == (int)(k1 * 256 + k2 * 16 + 2 * n + u), "phase 3 load");
          a.push_back(x);
        }
        excess += wavefronts(a, 16) - 4;
      }
  for (int i = 0; i < 4096; ++i) CHECK(n1[i] == 1 && out[i] == 1, "point %d", i);
  CHECK(excess == 0, "%d wavefronts of bank conflicts", excess);
  printf("%s 4096-point rows, FP32 exchange\n", g_bad == bad0 ? "ok" : "FAULT");
}

#define W(L, K, PT) check_mma<MmaPass<L, K, PT, false>>(#L " " #K)
#define WS(L) check_mma<MmaPass<L, kRR, false, false, 4096>>(#L " small")
#define V(L, R1, R2, TP, I, O, K, PT) check<RegPass<L, R1, R2, TP, I, O, K, PT, false>>(#L " " #R1 "x" #R2 " " #TP " " #I " " #O " " #K)
#define ROWS(TP, I, O, K)                                                              \
  V(64, 8, 8, TP, I, O, K, false), V(128, 8, 16, TP, I, O, K, false), V(256, 16, 16, TP, I, O, K, false), \
      V(512, 16, 32, TP, I, O, K, false), V(1024, 32, 32, TP, I, O, K, false)

int main() {
  check_mma4096();
  check_mma2048();
  check_gather(256, 1), check_gather(512, 2), check_gather(1024, 4), check_gather(2048, 8), check_gather(4096, 16);
  check_reg4096();
#define MM(L) check_maps<MmaPass<L, kRR, false, false, 4096>>({L, L / 256, 4096 / L, 0, true}, #L)
  MM(256), MM(512), MM(1024);
  check_maps<Mma4096<false>>({4096, 16, 1, 0, true}, "4096");
  check_maps<Reg4096<true, false>>({4096, 16, 1, 0, false}, "4096 FP16 in");
  check_maps<Reg4096<false, false>>({4096, 16, 1, 0, false}, "4096 FP32");
#define RM(L, R1, I, O) check_maps<RegPass<L, R1, L / R1, 4096, I, O, kRR, false, false>>({L, R1, 4096 / L, 0, false}, #L " " #I " " #O)
  RM(64, 8, true, true), RM(128, 8, true, true);
  RM(64, 8, true, false), RM(128, 8, true, false), RM(256, 16, true, false), RM(512, 16, true, false);
  RM(64, 8, false, false), RM(128, 8, false, false), RM(256, 16, false, false), RM(512, 16, false, false);
  W(256, kRR, false), W(512, kRR, false), W(1024, kRR, false);
  WS(256), WS(512), WS(1024);
  W(256, kRC, false), W(512, kRC, false), W(1024, kRC, false);
  W(256, kCC, true), W(512, kCC, true), W(1024, kCC, true);
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
  V(64, 8, 8, 4096, true, true, kRR, false), V(128, 8, 16, 4096, true, true, kRR, false);
  V(64, 8, 8, 4096, false, false, kRR, false), V(128, 8, 16, 4096, false, false, kRR, false);
  V(256, 16, 16, 4096, false, false, kRR, false), V(512, 16, 32, 4096, false, false, kRR, false);
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
