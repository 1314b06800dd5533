// Scheme and tile selection for the FP64-accurate Ozaki GEMMs.
//
// Order of precedence for each choice: an environment variable, then the
// tuning table (PHPC_TUNE_TABLE, or tune_table.txt next to the library;
// autotune.py writes one), then a built-in default. The table is measured on
// square problems; three rules go by the call's own shape and stand above it,
// below the environment: modular_bn and f32_narrow take 128-wide tiles where the
// table says 256, and pairs_fit refuses CTA pairs where the table has them.
// Schemes: the modular one
// (PHPC_MODULI = 8..15 residue GEMMs; built-in default: the fewest moduli
// whose operand grid has at least 51 bits, Frobenius error about 2e-15 on
// inputs whose exponents spread over 2^+-20 inside a row) or, with
// PHPC_MODULI=0 or a table entry of 0 moduli, the digit scheme (PHPC_SLICES =
// 2..8 slices, default 7: 55-bit digit grids).
#include <dlfcn.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "phpc_host.hpp"

namespace phpc {
namespace {

constexpr int kMinModuliCount = 8, kMaxModuliCount = 15;  // range of the modular scheme

struct TuneEntry {
  long long max_mnk;  // entry applies to problems with m*n*k <= max_mnk (first match wins)
  int slices;
  int bn;
  int group_rows;     // L2 raster height of the persistent tile order (0 = default 8)
  int cluster;        // CTAs per cluster sharing B (1 or 2; 0 = default 1)
  int moduli;         // modular scheme with this many moduli; 0 = digit scheme; -1 = built-in rule
  int stages;         // K-stages of the tcgen05 ring (0 = the deepest that fits)
};

// "f32 max_mnk bn group_rows stages": the 3xBF16 FP32 GEMM; "plain max_mnk
// stages": the plain FP64 GEMM's ring depth.
struct F32Entry {
  long long max_mnk;
  int bn, group_rows, stages;
};
struct PlainEntry {
  long long max_mnk;
  int stages;
};
// "digits max_mnk bn cluster": the digit GEMM of single problems.
struct DigitEntry {
  long long max_mnk;
  int bn, cluster;
};

std::once_flag g_once;
std::vector<TuneEntry> g_table;    // single-problem entries
std::vector<TuneEntry> g_grouped;  // grouped-call entries (lines starting with "grouped")
std::vector<F32Entry> g_f32;       // 3xBF16 entries (lines starting with "f32")
std::vector<PlainEntry> g_plain;   // plain FP64 entries (lines starting with "plain")
std::vector<DigitEntry> g_digits;  // digit-scheme entries (lines starting with "digits")

std::string library_dir() {
  Dl_info info;
  if (dladdr(reinterpret_cast<void*>(&library_dir), &info) && info.dli_fname) {
    std::string p(info.dli_fname);
    const size_t s = p.rfind('/');
    if (s != std::string::npos) return p.substr(0, s);
  }
  return ".";
}

// Table format (text): one entry per line, "max_mnk slices bn [group_rows
// [cluster [moduli [stages]]]]" for single problems, "grouped max_mean_mnk
// slices bn [stages]" for grouped calls, "f32 max_mnk bn group_rows stages"
// for the 3xBF16 GEMM, "plain max_mnk stages" for the plain FP64 GEMM and
// "digits max_mnk bn cluster" where the digit GEMM's choice is not that of the
// single-problem entry; '#' starts a comment line; the first entry whose
// max_mnk covers the problem applies.
void load_table() {
  const char* env = getenv("PHPC_TUNE_TABLE");
  const std::string path = env ? std::string(env) : library_dir() + "/tune_table.txt";
  FILE* f = fopen(path.c_str(), "r");
  if (!f) return;
  char line[256];
  while (fgets(line, sizeof line, f)) {
    if (line[0] == '#') continue;
    TuneEntry e{};
    if (strncmp(line, "grouped", 7) == 0) {
      const int got = sscanf(line + 7, "%lld %d %d %d", &e.max_mnk, &e.slices, &e.bn, &e.stages);
      if (got >= 3 && e.slices >= 2 && e.slices <= 8 && (e.bn == 128 || e.bn == 256)) {
        if (got < 4 || e.stages < 2) e.stages = 0;
        g_grouped.push_back(e);
      }
      continue;
    }
    if (strncmp(line, "f32", 3) == 0) {
      F32Entry f{};
      if (sscanf(line + 3, "%lld %d %d %d", &f.max_mnk, &f.bn, &f.group_rows, &f.stages) == 4 &&
          (f.bn == 128 || f.bn == 256) && f.group_rows >= 1 && f.group_rows <= 64 && (f.stages == 0 || f.stages >= 2))
        g_f32.push_back(f);
      continue;
    }
    if (strncmp(line, "plain", 5) == 0) {
      PlainEntry pe{};
      if (sscanf(line + 5, "%lld %d", &pe.max_mnk, &pe.stages) == 2 && pe.stages >= 2 && pe.stages <= 6)
        g_plain.push_back(pe);
      continue;
    }
    if (strncmp(line, "digits", 6) == 0) {
      DigitEntry de{};
      if (sscanf(line + 6, "%lld %d %d", &de.max_mnk, &de.bn, &de.cluster) == 3 && (de.bn == 128 || de.bn == 256) &&
          (de.cluster == 1 || de.cluster == 2))
        g_digits.push_back(de);
      continue;
    }
    const int got = sscanf(line, "%lld %d %d %d %d %d %d", &e.max_mnk, &e.slices, &e.bn, &e.group_rows, &e.cluster,
                           &e.moduli, &e.stages);
    if (got >= 3 && e.slices >= 2 && e.slices <= 8 && (e.bn == 128 || e.bn == 256)) {
      if (got < 4 || e.group_rows < 1 || e.group_rows > 64) e.group_rows = 0;
      if (got < 5 || (e.cluster != 1 && e.cluster != 2)) e.cluster = 0;
      if (got < 6 || (e.moduli != 0 && (e.moduli < kMinModuliCount || e.moduli > kMaxModuliCount))) e.moduli = -1;
      if (got < 7 || e.stages < 2) e.stages = 0;
      g_table.push_back(e);
    }
  }
  fclose(f);
}

const TuneEntry* lookup(int m, int k, int n) {
  std::call_once(g_once, load_table);
  const long long mnk = (long long)m * n * k;
  for (const TuneEntry& e : g_table)
    if (mnk <= e.max_mnk) return &e;
  return nullptr;
}

// Tile width and CTAs per cluster of the digit GEMM (0: not set): the first
// "digits" entry that covers the problem, else its single-problem entry. The
// two schemes part where tiles are few: the residue GEMM has a CTA per (tile,
// modulus), the digit GEMM one per tile, so N = 512 to 1448 wants twice as many
// tiles half as wide.
DigitEntry digit_entry(int m, int k, int n) {
  const TuneEntry* e = lookup(m, k, n);
  const long long mnk = (long long)m * n * k;
  for (const DigitEntry& d : g_digits)
    if (mnk <= d.max_mnk) return d;
  return e ? DigitEntry{e->max_mnk, e->bn, e->cluster} : DigitEntry{};
}

// The tile width PHPC_OZAKI_BN names (0: none), the cluster PHPC_CLUSTER names.
int env_bn() {
  const char* env = getenv("PHPC_OZAKI_BN");
  const int b = env ? atoi(env) : 0;
  return b == 128 || b == 256 ? b : 0;
}
int env_cluster() {
  const char* env = getenv("PHPC_CLUSTER");
  const int c = env ? atoi(env) : 0;
  return c == 1 || c == 2 ? c : 0;
}

}  // namespace

int default_slices(int m, int k, int n) {
  const char* env = getenv("PHPC_SLICES");
  if (env) {
    const int s = atoi(env);
    if (s >= 2 && s <= 8) return s;
  }
  if (const TuneEntry* e = lookup(m, k, n)) return e->slices;
  return 7;
}

int default_moduli(int m, int k, int n) {
  const char* env = getenv("PHPC_MODULI");
  if (env) {
    const int q = atoi(env);
    if (q == 0 || (q >= kMinModuliCount && q <= kMaxModuliCount)) return q;
  }
  if (const TuneEntry* e = lookup(m, k, n))
    if (e->moduli >= 0) return e->moduli;
  for (int q = kMinModuliCount; q < kMaxModuliCount; ++q)
    if (ozaki2_bits(q, k) >= 51) return q;
  return kMaxModuliCount;
}

int default_bn(int m, int k, int n) {
  if (const int b = env_bn()) return b;
  if (const TuneEntry* e = lookup(m, k, n)) return e->bn;
  return 256;
}

int digit_bn(int m, int k, int n) {
  if (const int b = env_bn()) return b;
  const DigitEntry d = digit_entry(m, k, n);
  return d.bn ? d.bn : 256;
}

int digit_cluster(int m, int k, int n) {
  if (const int c = env_cluster()) return c;
  return digit_entry(m, k, n).cluster == 2 ? 2 : 1;
}

// Tile width of a modular call's residue GEMM: default_bn, but 128 where the
// table says 256 and the (128-wide tile, modulus) units all run at once, so
// that the call waits for one unit's drain and stores of half the columns, or
// where columns beyond n <= 128 would only be padding. Whole calls, 256 / 128:
// 86 x 1343 x 615 33.5 us, 31.4; 235 x 3167 x 169 48.0, 45.6; 124 x 2991 x 1317
// (143 units) 89.9, 87.1; 336 x 4001 x 72 50.4, 47.1; 8000 x 1000 x 100 143, 137;
// N = 256 17.8, 16.4 as a graph. With more units than SMs the wide tile's fewer
// operand bytes count: GEMM of 664 x 1420 x 668 22.8, 35.0; so does its K split
// where that is much the finer one (residue_wide_split). Exact either way.
int modular_bn(int m, int k, int n, int moduli) {
  const int bn = default_bn(m, k, n);
  if (bn == 128 || getenv("PHPC_OZAKI_BN")) return bn;
  if (n <= 128) return 128;
  const DeviceInfo* dev = current_device();
  return dev && (int64_t)ceil_div(m, 128) * ceil_div(n, 128) * moduli <= dev->sm_count &&
                 !residue_wide_split(m, k, n, moduli, dev)
             ? 128
             : bn;
}

namespace {

// Whether CTA pairs suit a residue GEMM where the table has them. A pair stages
// 32 KB a K-step and SM against 48, but its units cost more to start and to
// drain (GEMM alone in us, single / pairs, 13 moduli unless named):
//  - fewer than 80 K-steps an SM: N = 1024 (44 an SM) 25.4, 29.1; 1024 x 1536 x
//    1024 (66) 39.1, 39.2; 1024 x 2048 x 1024 (88) 47.5, 47.2; 2048 x 512 x 2048
//    (88) 52.5, 48.2; 8 moduli, 1024 x 2048 x 1024 (54) 30.9, 33.5; 1500^3 (91)
//    47.4, 47.2; 10 moduli, 1536 x 1500 x 1024 (76) 47.2, 47.3; 15, N = 1024 (51)
//    33.7, 37.0;
//  - a last accumulator chunk (of 8 K-steps) that is half empty or emptier, or
//    a single short one, leaves the MMAs waiting for the drain of the pair's
//    other chunk: 4096 x K x 4096 with K = 256 110, 148; 384 144, 145; 512
//    171, 156; 520 208, 235; 700 227, 244; 830 258, 256; 1000 318, 285; 1100
//    344, 362; 2000 548, 526;
//  - an odd number of tile rows pads the last pair: 14 shapes of 5 to 11 rows
//    from 0.93 to 1.17 of the single CTAs' time, 1.03 on average; 26 of 13 to
//    27 rows 0.94 to 1.11, 0.99 on average.
bool pairs_fit(int m, int k, int n, int moduli) {
  const DeviceInfo* dev = current_device();
  const int64_t pairs = dev ? dev->sm_count / 2 : 76;
  const int64_t rows = ceil_div(m, 128), steps = ceil_div(k, 64), units = (rows + 1) / 2 * ceil_div(n, 256) * moduli;
  const bool full = steps % 8 == 0 || steps % 8 > 4 || steps > 32;
  return full && steps >= 8 && units * steps >= 80 * pairs && (rows % 2 == 0 || rows > 12);
}

}  // namespace

// CTAs per cluster of the single-problem residue GEMM (1, or 2 = a CTA pair
// computing one 256-row tile with cta_group::2 MMAs, each CTA loading its own
// half of the operands): PHPC_CLUSTER, else the table's choice where pairs
// suit the shape, else 1.
int default_cluster(int m, int k, int n, int moduli) {
  if (const int c = env_cluster()) return c;
  if (const TuneEntry* e = lookup(m, k, n))
    if (e->cluster == 2 && pairs_fit(m, k, n, moduli)) return 2;
  return 1;
}

int default_group_rows(int m, int k, int n) {
  const char* env = getenv("PHPC_GROUP_ROWS");
  if (env && atoi(env) > 0 && atoi(env) <= 64) return atoi(env);
  if (const TuneEntry* e = lookup(m, k, n))
    if (e->group_rows > 0) return e->group_rows;
  return 8;
}

// Tile width of the grouped slice GEMM: PHPC_GROUPED_BN, else the tuning
// table's entry for the batch's mean problem size, else 128 (small problems
// waste less of a 128-wide tile).
int default_grouped_bn(const phpc_gemm_problem* problems, int count) {
  const char* env = getenv("PHPC_GROUPED_BN");
  if (env) {
    const int b = atoi(env);
    if (b == 128 || b == 256) return b;
  }
  double mnk = 0;
  for (int i = 0; i < count; ++i) mnk += (double)problems[i].m * problems[i].n * problems[i].k;
  if (count > 0) {
    std::call_once(g_once, load_table);
    const long long mean = (long long)(mnk / count);
    for (const TuneEntry& e : g_grouped)
      if (mean <= e.max_mnk) return e.bn;
  }
  return 128;
}

// K-stages of the tcgen05 ring: PHPC_STAGES (>= 2; the launcher caps it at
// what fits), else the table, else 0 (the deepest ring that fits).
int default_stages(int m, int k, int n) {
  const char* env = getenv("PHPC_STAGES");
  if (env && atoi(env) >= 2) return atoi(env);
  if (const TuneEntry* e = lookup(m, k, n)) return e->stages;
  return 0;
}

int default_grouped_stages(const phpc_gemm_problem* problems, int count) {
  const char* env = getenv("PHPC_STAGES");
  if (env && atoi(env) >= 2) return atoi(env);
  double mnk = 0;
  for (int i = 0; i < count; ++i) mnk += (double)problems[i].m * problems[i].n * problems[i].k;
  if (count > 0) {
    std::call_once(g_once, load_table);
    const long long mean = (long long)(mnk / count);
    for (const TuneEntry& e : g_grouped)
      if (mean <= e.max_mnk) return e.stages;
  }
  return 0;
}

namespace {

// Where the 3xBF16 GEMM takes 128-wide tiles although its table entry says
// 256: a call that K is not split for and whose 128 x 128 tiles all run at
// once takes as long as one tile, half of it the C += AB of a warp's columns,
// 32 at a time; and columns beyond n <= 128 are only padding. Replayed graphs,
// 256 / 128: 500 x 94 x 500 18.5 us, 12.5; 1000 x 300 x 1000 24.1, 18.4; 1000 x
// 440 x 2000 (128 tiles) 28.8, 22.7; 584 x 495 x 84 15.8, 12.5. The same holds
// with K split, whose shares then exchange half as much, while the clusters of
// the narrow tiles still run at once (calls: 132 x 3857 x 268, 6 clusters of 8,
// 35.0, 30.0; 611 x 2534 x 279, 15 clusters, 31.2, 26.4; but 16: 250 x 600 x 900
// 20.8, 27.1). With a second wave the wide tile's fewer operand bytes count:
// 4868 x 216 x 605 (195 tiles) 28.4, 30.7; 1000 x 777 x 1530 28.4, 43.3.
bool f32_narrow(int m, int k, int n) {
  if (n <= 128) return true;
  const DeviceInfo* dev = current_device();
  if (!dev) return false;
  if (6 * ceil_div(k, 64) < kF32SplitSteps) return (int64_t)ceil_div(m, 128) * ceil_div(n, 128) <= dev->sm_count;
  return f32_narrow_split(m, k, n, dev);
}

}  // namespace

F32Tune default_f32(int m, int k, int n) {
  F32Tune t{256, 8, 0};
  std::call_once(g_once, load_table);
  const long long mnk = (long long)m * n * k;
  for (const F32Entry& e : g_f32)
    if (mnk <= e.max_mnk) {
      t = {e.bn, e.group_rows, e.stages};
      break;
    }
  if (t.bn == 256 && f32_narrow(m, k, n)) t.bn = 128;
  if (const char* env = getenv("PHPC_F32_BN"))
    if (atoi(env) == 128 || atoi(env) == 256) t.bn = atoi(env);
  if (const char* env = getenv("PHPC_GROUP_ROWS"))
    if (atoi(env) > 0 && atoi(env) <= 64) t.group_rows = atoi(env);
  if (const char* env = getenv("PHPC_STAGES"))
    if (atoi(env) >= 2) t.stages = atoi(env);
  return t;
}

// Ring depth of the plain FP64 GEMM: PHPC_DMMA_STAGES (2 .. 6), else the
// table, else 4.
int default_plain_stages(int m, int k, int n) {
  const char* env = getenv("PHPC_DMMA_STAGES");
  if (env && atoi(env) >= 2 && atoi(env) <= 6) return atoi(env);
  std::call_once(g_once, load_table);
  const long long mnk = (long long)m * n * k;
  for (const PlainEntry& e : g_plain)
    if (mnk <= e.max_mnk) return e.stages;
  return 4;
}

}  // namespace phpc

extern "C" int phpc_default_slices(int m, int k, int n) { return phpc::default_slices(m, k, n); }

extern "C" int phpc_tuning(int m, int k, int n, int* cfg) {
  using namespace phpc;
  if (!cfg || m < 0 || k < 0 || n < 0) return PHPC_ERR_ARG;
  const F32Tune f = default_f32(m, k, n);
  const int q = default_moduli(m, k, n);
  const int v[10] = {q, default_slices(m, k, n), q ? modular_bn(m, k, n, q) : digit_bn(m, k, n),
                     default_group_rows(m, k, n), q ? default_cluster(m, k, n, q) : digit_cluster(m, k, n),
                     default_stages(m, k, n),
                     f.bn, f.group_rows, f.stages, default_plain_stages(m, k, n)};
  for (int i = 0; i < 10; ++i) cfg[i] = v[i];
  return PHPC_OK;
}
