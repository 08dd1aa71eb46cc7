// Host checks of a batch's buffers and graphs (csrc/fk_engine.cu) on the fake
// CUDA runtime.  Each check prints "<name> ok", or what went wrong.
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/fk.h"
#include "fake_cuda.h"

struct CUstream_st;
namespace fk {
struct SieveArgs;
int launch_sieve(unsigned, unsigned, unsigned, CUstream_st*, const SieveArgs&) {
  fake_kernel();
  return 0;
}
int launch_mark(unsigned, unsigned, unsigned, unsigned, CUstream_st*,
                const SieveArgs&) {
  ++fake().marks;
  fake_kernel();
  return 0;
}
int sieve_set_smem_limits() { return 0; }
int mark_set_smem_limits() { return 0; }
}  // namespace fk

namespace {

fk_engine* engine(uint32_t kind, uint32_t n, uint32_t q2, uint32_t sieve,
                  uint32_t p0 = 6) {
  fk_params p;
  std::memset(&p, 0, sizeof p);
  p.kind = kind;
  p.n = n;
  p.q2 = q2;
  p.p0 = p0;
  p.sieve = sieve;
  fk_engine* e = nullptr;
  if (fk_engine_create(&p, &e)) std::printf("create: %s\n", fk_last_error());
  return e;
}

// One run of `count` intervals of `len`; false when it fails or its result is
// not the fake's (every output in the last interval, offsets rising by one).
bool run(fk_batch* b, uint64_t count, int graph, uint64_t len = 1 << 16,
         uint64_t step = 1 << 20) {
  std::vector<fk_item> it(count);
  std::memset(it.data(), 0, count * sizeof(fk_item));
  for (uint64_t i = 0; i < count; ++i) {
    it[i].mode = 1;
    it[i].threshold = 1;
    it[i].cap = 8;
    it[i].lo[0] = 1000000007ull + i * step;
    it[i].hi[0] = it[i].lo[0] + len;
  }
  fk_batch_result r;
  if (fk_batch_run(b, it.data(), count, graph, &r)) return false;
  if (r.item_start[count] != fake().outputs) return false;
  for (uint64_t k = 0; k < fake().outputs; ++k)
    if (r.offset[k] != r.offset[0] + k || r.depth[k] != 7) return false;
  return true;
}

struct Batch {
  fk_engine* e;
  fk_batch* b = nullptr;
  explicit Batch(uint32_t q2 = 65536) : e(engine(0, 8, q2, 1)) {
    fk_batch_create(&e, 1, &b);
  }
  ~Batch() {
    fk_batch_destroy(b);
    fk_engine_destroy(e);
  }
};

// Eager runs between graph runs move buffers the graph holds.
bool growth() {
  struct Step { uint64_t count; int graph; uint64_t len; };
  // the first run sizes every buffer that goes by the expected output
  const std::vector<std::vector<Step>> lists = {
      {{684, 0, 1ull << 32}, {690, 0, 0}, {1000, 1, 0}, {1024, 0, 0}, {1000, 1, 0}},
      {{700, 0, 1ull << 32}, {750, 0, 0}, {1000, 1, 0}, {1030, 0, 0}, {1000, 1, 0}},
  };
  bool ok = true;
  for (const auto& l : lists) {
    Batch b;
    for (const Step& s : l) {
      fake().outputs = 100 + s.count % 7;
      ok &= run(b.b, s.count, s.graph, s.len ? s.len : 1 << 16);
    }
  }
  // and any order of sizes, forms and results
  uint64_t x = 88172645463325252ull;
  for (int seq = 0; seq < 12; ++seq) {
    Batch b(600);
    fake().outputs = 1;
    ok &= run(b.b, 1, 0, 1ull << 34);
    for (int k = 0; k < 40; ++k) {
      x ^= x << 13; x ^= x >> 7; x ^= x << 17;
      fake().outputs = (x >> 20) % 4000;
      fake().overflows = (x >> 50) % 8 == 0;
      ok &= run(b.b, 1 + (x >> 40) % (40u << (seq % 6)), (x >> 10) & 1,
                1 << (16 + (x >> 33) % 8));
    }
  }
  if (fake().dead) std::printf("growth: %llu uses of freed buffers\n",
                               (unsigned long long)fake().dead);
  return ok && fake().dead == 0;
}

// A batch's graph is captured once, whatever the number of its results, and
// results are whole on both sides of the length that comes back at once.
bool once() {
  Batch b;
  bool ok = true;
  for (uint64_t n : {3000u, 4000u, 0u, 1u, 2047u, 2048u, 2049u, 4096u, 2048u}) {
    fake().outputs = n;
    ok &= run(b.b, 300, 1) && run(b.b, 300, 0);
  }
  if (fake().captures != 1)
    std::printf("once: %llu captures\n", (unsigned long long)fake().captures);
  return ok && fake().captures == 1 && fake().dead == 0;
}

// A failed call is reported by the run that made it and by no other.
bool error_once() {
  Batch b;
  fake().outputs = 5;
  fake_fail_allocation(0);
  const bool first = run(b.b, 20, 0);
  return !first && run(b.b, 20, 0) && run(b.b, 20, 1) && fake().dead == 0;
}

// An allocation that fails while the buffers grow fails that run alone: the
// next one has buffers for what it does, whatever it was that was missing.
bool failed_growth() {
  bool ok = true;
  for (int graph = 0; graph < 2; ++graph)
    for (int skip = 0; skip < 40; ++skip) {
      Batch b(600);
      fake().outputs = 50;
      ok &= run(b.b, 20, graph);
      // every buffer that goes by the items or the expected output grows
      fake_fail_allocation(skip);
      const bool grown = run(b.b, 3000, graph, 1ull << 30, 1ull << 33);
      fake_fail_allocation(-1);
      // the small run again, larger ones that fit or not, and one that
      // overflows its buffers
      fake().overflows = skip % 3 == 0;
      ok &= run(b.b, 20, graph) && run(b.b, 2000, graph) &&
            run(b.b, 3000, graph, 1ull << 30, 1ull << 33);
      if (fake().dead || !ok) {
        std::printf("failed_growth: graph %d, allocation %d (%s): %llu uses "
                    "of missing buffers\n", graph, skip,
                    grown ? "passed" : "failed", (unsigned long long)fake().dead);
        return false;
      }
      if (grown) break;   // no allocation left to fail
    }
  return ok;
}

// Dickson lists of more than 2^24 entries, filling included: their offsets
// count groups of four.
bool long_lists() {
  fk_engine* e = engine(1, 3, 86000000, 1);
  const bool ok = e != nullptr;
  fk_engine_destroy(e);
  return ok;
}

// fk_stats.d2h_bytes is what a run copies back, the entries that are read
// before the result's length is known included.
bool read_back() {
  Batch b;
  bool ok = true;
  for (uint64_t n : {0u, 1u, 2047u, 2048u, 2049u, 4000u}) {
    fake().outputs = n;
    const uint64_t before = fake().d2h;
    ok &= run(b.b, 300, 0);
    fk_stats st;
    ok &= fk_batch_stats(b.b, &st) == FK_OK;
    if (st.d2h_bytes != fake().d2h - before) {
      std::printf("read_back: %llu outputs: %llu bytes, %llu copied\n",
                  (unsigned long long)n, (unsigned long long)st.d2h_bytes,
                  (unsigned long long)(fake().d2h - before));
      ok = false;
    }
  }
  return ok;
}

// fk_stats.rounds_ms covers the rounds launches of every wheel family and the
// launch that finishes what they left, mark_ms the marking launches.  (An
// event's time here is the number of kernels before it.)
bool stage_times() {
  fk_engine* e[3] = {engine(0, 8, 600, 1), engine(0, 8, 600, 1, 7),
                     engine(0, 8, 600, 2)};
  fk_batch* b = nullptr;
  bool ok = fk_batch_create(e, 3, &b) == FK_OK;
  for (int used = 1; used < 8; ++used)
    for (int graph = 0; graph < 2; ++graph) {
      std::vector<fk_item> it;
      for (uint32_t i = 0; i < 3; ++i) {
        if (!((used >> i) & 1)) continue;
        fk_item x;
        std::memset(&x, 0, sizeof x);
        x.engine = i;
        x.lo[0] = 1000000007ull;
        x.hi[0] = x.lo[0] + (1 << 24);
        it.push_back(x);
      }
      fake().outputs = 3;
      fk_batch_result r;
      fk_stats st;
      ok &= fk_batch_run(b, it.data(), it.size(), graph, &r) == FK_OK &&
            fk_batch_stats(b, &st) == FK_OK;
      const int rounds = (used & 1) + (used >> 1 & 1);
      const float want = rounds ? rounds + 1 : 0, marks = used >> 2;
      if (st.rounds_ms != want || st.mark_ms != marks) {
        std::printf("stage_times: engines %d graph %d: rounds %g, not %g; marks "
                    "%g\n", used, graph, st.rounds_ms, want, st.mark_ms);
        ok = false;
      }
    }
  fk_batch_destroy(b);
  for (fk_engine* x : e) fk_engine_destroy(x);
  return ok;
}

// A replayed graph's statistics are its own, whatever ran in between.
bool replay_stats() {
  Batch b(600);
  fake().outputs = 3;
  fk_item dense;
  std::memset(&dense, 0, sizeof dense);
  dense.mode = 2;
  dense.lo[0] = 2;
  dense.hi[0] = 1000;
  dense.cap = 8;
  fk_stats first, eager, again;
  fk_batch_result r;
  bool ok = run(b.b, 20, 1) && fk_batch_stats(b.b, &first) == FK_OK;
  ok &= fk_batch_run(b.b, &dense, 1, 0, &r) == FK_OK &&
        fk_batch_stats(b.b, &eager) == FK_OK;
  ok &= run(b.b, 20, 1) && fk_batch_stats(b.b, &again) == FK_OK;
  ok &= first.launches != eager.launches && eager.rounds_ms == 0;
  if (again.launches != first.launches || again.rounds_ms != first.rounds_ms) {
    std::printf("replay_stats: %llu launches, not %llu; rounds %g, not %g\n",
                (unsigned long long)again.launches,
                (unsigned long long)first.launches, again.rounds_ms,
                first.rounds_ms);
    ok = false;
  }
  return ok;
}

// Two settings of classify_ctas_per_sm that launch the same grids share a
// graph; one that does not has its own.
bool class_grids() {
  Batch b(600);
  fake().outputs = 3;
  bool ok = run(b.b, 20, 1);
  fk_tuning t;
  std::memset(&t, 0, sizeof t);
  for (uint32_t v : {2u, 4u, 16u, 32u}) {
    t.classify_ctas_per_sm = v;
    ok &= fk_batch_set_tuning(b.b, &t) == FK_OK && run(b.b, 20, 1);
  }
  const uint64_t same = fake().captures;
  t.classify_ctas_per_sm = 1;
  ok &= fk_batch_set_tuning(b.b, &t) == FK_OK && run(b.b, 20, 1);
  if (same != 1 || fake().captures != 2)
    std::printf("class_grids: %llu and %llu captures\n",
                (unsigned long long)same, (unsigned long long)fake().captures);
  return ok && same == 1 && fake().captures == 2;
}

// Which sieve an interval takes alone, and beside milliseconds of other work: a
// few blocks of a weak filter, thousands of tests each, are marked when nothing
// else fills the time those would take -- but not where most primes lie past
// the marked ones; strong filters and long intervals go by the SMs' cycles.
bool lone_items() {
  struct Case { uint32_t kind, n, q2, p0; uint64_t lo, len; bool alone, among; };
  const Case cases[] = {
      {0, 3, 40000, 6, 38956, 4415233, true, false},
      {0, 2, 65536, 6, 1000000000, 1 << 20, true, false},
      {1, 1, 4096, 7, 1758209, 42006, true, true},
      {0, 3, 1 << 18, 6, 1000000000, 1 << 16, false, false},
      {0, 5, 65536, 6, 300000, 1 << 20, false, false},     // about even
      {0, 8, 65536, 6, 1000000000, 1000000000, false, false},
      {1, 12, 65536, 6, 1000000000, 1 << 24, false, false},
      {0, 3, 65536, 7, 1000000000, 1ull << 36, true, true},
  };
  bool ok = true;
  for (const Case& c : cases) {
    fk_engine* e[2] = {engine(c.kind, c.n, c.q2, 0, c.p0),
                       engine(0, 12, 65536, 1, 7)};
    fk_batch* b = nullptr;
    ok &= fk_batch_create(e, 2, &b) == FK_OK;
    fake().outputs = 0;
    fk_item it[2];
    std::memset(it, 0, sizeof it);
    it[0].lo[0] = c.lo;
    it[0].hi[0] = c.lo + c.len;
    it[1].engine = 1;                  // milliseconds of rounds
    it[1].hi[0] = 1ull << 44;
    fk_batch_result r;
    const uint64_t m0 = fake().marks;
    ok &= fk_batch_run(b, it, 1, 0, &r) == FK_OK;
    const bool marked = fake().marks != m0;
    if (marked != c.alone) {
      std::printf("lone_items: kind %u n %u length %llu: marked %d\n", c.kind,
                  c.n, (unsigned long long)c.len, marked);
      ok = false;
    }
    const uint64_t m1 = fake().marks;
    ok &= fk_batch_run(b, it, 2, 0, &r) == FK_OK;
    const bool among = fake().marks != m1;
    if (among != c.among) {
      std::printf("lone_items: kind %u n %u length %llu: marked %d in a batch\n",
                  c.kind, c.n, (unsigned long long)c.len, among);
      ok = false;
    }
    fk_batch_destroy(b);
    for (fk_engine* x : e) fk_engine_destroy(x);
  }
  return ok;
}

// Up to about a thousand items nothing grows but the residue table: growing
// under load waits for whatever else runs on the device.
bool steady_items() {
  Batch b(600);
  fake().outputs = 10;
  bool ok = run(b.b, 1, 0, 1ull << 34);
  for (uint64_t n : {2u, 10u, 40u, 160u, 640u, 700u}) {
    const uint64_t before = fake().allocations;
    ok &= run(b.b, n, 0);
    const uint64_t grown = fake().allocations - before;
    if (grown > 1) {
      std::printf("steady_items: %llu items: %llu allocations\n",
                  (unsigned long long)n, (unsigned long long)grown);
      ok = false;
    }
  }
  return ok;
}

}  // namespace

int main(int argc, char** argv) {
  const struct { const char* name; bool (*check)(); } checks[] = {
      {"growth", growth},
      {"once", once},
      {"error_once", error_once},
      {"failed_growth", failed_growth},
      {"long_lists", long_lists},
      {"read_back", read_back},
      {"replay_stats", replay_stats},
      {"class_grids", class_grids},
      {"lone_items", lone_items},
      {"steady_items", steady_items},
      {"stage_times", stage_times},
  };
  for (const auto& c : checks)
    if (argc > 1 && std::strcmp(argv[1], c.name) == 0)
      std::printf("%s %s\n", c.name, c.check() ? "ok" : "failed");
  return 0;
}
