// Plain FP64 GEMM: C[M x N] += A[M x K] * B[K x N].
//
// Replaces the reference's SIMT kernel (src/phpc_gemm.cu:6-57, shared-memory
// tiles of tile_width^2 doubles, one DFMA per shared load pair) with:
//  - one CTA per output tile, numbered through the logical SUMMA block grid
//    (grid_width x grid_height blocks of C, src/phpc_summa.c:36-44) block by
//    block, so the CTAs working at one time share A row panels and B column
//    panels in L2;
//  - a producer warp that streams the k-panels of A and B into a shared-memory
//    ring of 2-6 stages (4 unless PHPC_DMMA_STAGES or the tuning table's
//    "plain" entry says otherwise) with TMA (the on-device form of the reference's
//    per-panel row/column broadcasts, src/phpc_summa.c:63-89);
//  - consumer warps computing 8 x 4 to 16 x 16 outputs each with FP64
//    accumulation in registers over the whole K range, on the scalar FP64 pipe (DFMA, the
//    default: 1.245 TFLOP/s at N = 16384, the GPU's FP64 rate) or on the FP64
//    tensor cores (mma.sync.m16n8k4.f64, PHPC_FP64_PIPE=dmma: 1.089 TFLOP/s);
//    both give the same bits, those of the reference's kernel;
//  - an epilogue that adds the tile into C, as the reference does (C +=, line 55).
// Out-of-range rows/columns of A and B are zero-filled by TMA, which plays the
// role of the reference's zero padding (src/phpc_gemm.cu:38-46).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "phpc_dev.cuh"
#include "phpc_host.hpp"

namespace phpc {
namespace {

constexpr int kBK = 16;         // doubles of K per stage (one 128-byte row of A)
constexpr int kMaxStages = 6;   // ring depth bounds (PHPC_DMMA_STAGES, tuning table)

struct SummaGrid {
  int tm, tn;   // tiles along M and N
  int gh, gw;   // logical block grid (rows x cols of C blocks)
};

// Tile index -> (tile row, tile col) in block-major order: blocks of the
// logical SUMMA grid in row-major order, tiles row-major inside a block.
// Block (bi, bj) owns tile rows [bi*tm/gh, (bi+1)*tm/gh) and tile columns
// [bj*tn/gw, (bj+1)*tn/gw).
// Computed, not searched: block (bi, .) is the last whose first tile row is at
// or before tile row t / tn (gh <= tm, gw <= tn).
__device__ __forceinline__ void tile_coords(const SummaGrid& g, int t, int& rm, int& rn) {
  const int bi = static_cast<int>(((int64_t)(t / g.tn + 1) * g.gh - 1) / g.tm);
  const int r0 = (int)((int64_t)bi * g.tm / g.gh), r1 = (int)((int64_t)(bi + 1) * g.tm / g.gh);
  t -= r0 * g.tn;
  const int bj = static_cast<int>(((int64_t)(t / (r1 - r0) + 1) * g.gw - 1) / g.tn);
  const int c0 = (int)((int64_t)bj * g.tn / g.gw), c1 = (int)((int64_t)(bj + 1) * g.tn / g.gw);
  t -= (r1 - r0) * c0;
  rm = r0 + t / (c1 - c0);
  rn = c0 + t % (c1 - c0);
}

// Tiles of BT x BT outputs (8: 8 x 16), warps of WM x WN. Each of the SM's
// four quarters has its own FP64 pipe (half an FMA a clock), so all tiles give
// every quarter a warp (8 x 4 outputs each in the 8 x 16 tile; FP64 tensor-core
// warps are at least 16 x 8). Larger tiles buy nothing, since the pipe, not
// shared memory or L2, is the limit: 64 x 64 tiles took 14.4 ms at N = 2048
// against 13.8 for 16 x 16, 128 x 128 tiles 895 ms at N = 8192 against 883 for
// 32 x 32, and a call that leaves SMs idle at 64 x 64 is up to 8x slower (250 x
// 514 x 302: 566 us against 72.2 with 8 x 16).
template <int BT, bool DFMA>
struct DmmaCfg {
  static_assert(BT != 8 || DFMA, "an FP64 tensor-core warp has 16 rows");
  static constexpr int BM = BT, BN = BT == 8 ? 16 : BT;
  static constexpr int WM = BT == 32 ? 16 : DFMA ? 8 : 16;
  static constexpr int WN = BT == 32 ? 16 : BT == 8 ? 4 : 8;
  static constexpr int kWarpsN = BN / WN;
  static constexpr int kConsumers = (BM / WM) * kWarpsN;
  static constexpr int kThreads = (kConsumers + 1) * 32;
  static constexpr int kStageA = BM * kBK * 8;
  static constexpr int kStageB = kBK * BN * 8;
  static constexpr int kStageBytes = kStageA + kStageB;  // a multiple of 1024: A's swizzle atoms stay aligned
  static constexpr size_t smem(int stages) { return (size_t)stages * kStageBytes + 1024 /*align*/ + 256 /*barriers*/; }
};

// A's rows of 16 doubles are stored with the 128-byte swizzle: element (row,
// k) is at 16-byte chunk (k / 2) ^ (row % 8) of its row, so that the eight
// rows a warp reads at one k lie in different banks. Chunk c of row `row`:
__device__ __forceinline__ const double* a_chunk(const double* sA, int row, int c) {
  return sA + row * kBK + 2 * (c ^ (row & 7));
}

// DFMA = false: mma.sync.m16n8k4.f64 (FP64 tensor cores); true: the same
// outputs per thread computed with scalar FP64 FMAs. Both sum every output
// over k in increasing order with one rounding per FMA, so they give the same
// bits (and the same bits as the reference's SIMT kernel).
template <int BT, bool DFMA>
__global__ void __launch_bounds__(DmmaCfg<BT, DFMA>::kThreads)
    dmma_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, double* C,
                     int64_t ldc, int M, int N, int K, int kpanel, SummaGrid grid, int stages, int* status) {
  using Cfg = DmmaCfg<BT, DFMA>;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, WM = Cfg::WM, WN = Cfg::WN;
  // a thread's outputs: rows g + 8 r, columns 8 j + NV tig .. + NV - 1
  constexpr int NR = WM / 8, NJ = (WN + 7) / 8, NV = WN >= 8 ? 2 : 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int S = stages;  // ring depth, 2 .. kMaxStages (checked by the launcher)
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * Cfg::kStageBytes);
  uint64_t* empty = full + S;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int rm, rn;
  tile_coords(grid, blockIdx.x, rm, rn);
  const int ksteps = (K + kBK - 1) / kBK;
  const int kp_steps = max(1, kpanel / kBK);  // BK steps per SUMMA k-panel

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], Cfg::kConsumers);
    }
    fence_mbar_init();
  }
  __syncthreads();

  if (warp == Cfg::kConsumers) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0;
      bool ok = true;
      // SUMMA k-panels, each streamed as kp_steps TMA stages.
      for (int p0 = 0; p0 < ksteps && ok; p0 += kp_steps) {
        const int p1 = min(ksteps, p0 + kp_steps);
        for (int ks = p0; ks < p1; ++ks) {
          if (!wait_parity(&empty[stage], phase ^ 1, status, 1)) { ok = false; break; }
          mbar_arrive_expect_tx(&full[stage], Cfg::kStageBytes);
          uint8_t* sa = smem + stage * Cfg::kStageBytes;
          tma_load_2d(sa, &tmA, ks * kBK, rm * BM, &full[stage]);
          tma_load_2d(sa + Cfg::kStageA, &tmB, rn * BN, ks * kBK, &full[stage]);
          ++issued;
          if (++stage == S) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // Let the copies already in flight land before the CTA exits.
        int s = stage;
        uint32_t ph = phase;
        for (int i = 0; i < min(issued, S); ++i) {
          if (--s < 0) { s = S - 1; ph ^= 1; }
          const uint32_t addr = smem_u32(&full[s]);
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(addr, ph) && globaltimer_ns() - t0 < PHPC_WAIT_LIMIT_NS) {}
        }
      }
    }
  } else {
    // ------------------------------------------------------------ consumers
    const int wm = warp / Cfg::kWarpsN, wn = warp % Cfg::kWarpsN;
    const int g = lane >> 2, tig = lane & 3;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    double acc[NR][NJ][NV];
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[r][j][v] = 0.0;

    for (int ks = 0; ks < ksteps; ++ks) {
      // all lanes must agree before the warp-collective mma.sync below
      ok = __all_sync(0xffffffffu, wait_parity(&full[stage], phase, status, 2));
      if (!ok) break;
      const double* sA = reinterpret_cast<const double*>(smem + stage * Cfg::kStageBytes);  // [BM][16]
      const double* sB = reinterpret_cast<const double*>(smem + stage * Cfg::kStageBytes + Cfg::kStageA);  // [16][BN]
      if constexpr (DFMA) {
#pragma unroll 2
        for (int c = 0; c < kBK / 2; ++c) {
          double2 a[NR];
#pragma unroll
          for (int r = 0; r < NR; ++r)
            a[r] = *reinterpret_cast<const double2*>(a_chunk(sA, wm * WM + 8 * r + g, c));
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            double b[NJ][NV];
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
              const double* src = &sB[(2 * c + h) * BN + wn * WN + j * 8 + NV * tig];
              if constexpr (NV == 2) {
                const double2 w = *reinterpret_cast<const double2*>(src);
                b[j][0] = w.x;
                b[j][1] = w.y;
              } else {
                b[j][0] = *src;
              }
            }
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
              for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int v = 0; v < NV; ++v) acc[r][j][v] = fma(h ? a[r].y : a[r].x, b[j][v], acc[r][j][v]);
          }
        }
      } else {
#pragma unroll
        for (int kk = 0; kk < kBK; kk += 4) {
          double a[NR], b[NJ];
#pragma unroll
          for (int r = 0; r < NR; ++r) a[r] = a_chunk(sA, wm * WM + 8 * r + g, (kk + tig) >> 1)[tig & 1];
#pragma unroll
          for (int j = 0; j < NJ; ++j) b[j] = sB[(kk + tig) * BN + wn * WN + j * 8 + g];
#pragma unroll
          for (int r = 0; r + 1 < NR; r += 2)
#pragma unroll
            for (int j = 0; j < NJ; ++j)
              asm volatile(
                  "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                  : "+d"(acc[r][j][0]), "+d"(acc[r][j][1]), "+d"(acc[r + 1][j][0]), "+d"(acc[r + 1][j][1])
                  : "d"(a[r]), "d"(a[r + 1]), "d"(b[j]));
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
      if (++stage == S) { stage = 0; phase ^= 1; }
    }
    if (!ok) return;
    // Epilogue: C += tile.
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int64_t row = (int64_t)rm * BM + wm * WM + 8 * r + g;
      if (row >= M) continue;
      double* crow = C + row * ldc;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int col = rn * BN + wn * WN + j * 8 + NV * tig;
#pragma unroll
        for (int v = 0; v < NV; ++v)
          if (col + v < N) crow[col + v] += acc[r][j][v];
      }
    }
  }
}

template <int BT, bool DFMA>
int launch_dmma(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, double* dC,
                int64_t ldc, int gw, int gh, int kpanel, cudaStream_t stream) {
  using Cfg = DmmaCfg<BT, DFMA>;
  constexpr int BM = Cfg::BM, BN = Cfg::BN;
  const DeviceInfo* dev = current_device();
  if (!dev) return PHPC_ERR_CUDA;
  CUtensorMap tmA, tmB;
  const uint64_t dimsA[2] = {(uint64_t)k, (uint64_t)m};
  const uint64_t strA[1] = {(uint64_t)lda * 8};
  const uint32_t boxA[2] = {kBK, BM};
  const uint64_t dimsB[2] = {(uint64_t)n, (uint64_t)k};
  const uint64_t strB[1] = {(uint64_t)ldb * 8};
  const uint32_t boxB[2] = {BN, kBK};
  if (!encode_tiled(&tmA, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, dA, dimsA, strA, boxA, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !encode_tiled(&tmB, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, dB, dimsB, strB, boxB, CU_TENSOR_MAP_SWIZZLE_NONE))
    return PHPC_ERR_CUDA;
  SummaGrid g;
  g.tm = ceil_div(m, BM);
  g.tn = ceil_div(n, BN);
  g.gh = std::min(gh, g.tm);
  g.gw = std::min(gw, g.tn);
  const int ntiles = g.tm * g.tn;
  auto kern = dmma_gemm_kernel<BT, DFMA>;
  const int stages = default_plain_stages(m, k, n);
  if (stages < 2 || stages > kMaxStages) return PHPC_ERR_ARG;
  const size_t smem = Cfg::smem(stages);
  static PerDevice ready;
  if (!ready.get(dev->ordinal)) {
    PHPC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::smem(kMaxStages)));
    ready.set(dev->ordinal, 1);
  }
  // One CTA per tile: the hardware gives an SM its next tile when one is done.
  // A persistent grid with tiles c, c + grid, ... left some SMs 8 % more work
  // (N = 1024 1806 us against 1745, 2048 14.05 ms against 13.84), and a CTA's
  // set-up is hidden by the seven others on its SM.
  kern<<<ntiles, Cfg::kThreads, smem, stream>>>(tmA, tmB, dC, ldc, m, n, k, kpanel, g, stages, device_status_ptr());
  PHPC_CUDA_TRY(cudaGetLastError());
  return PHPC_OK;
}

}  // namespace

// The FP64 pipe of the plain GEMM: the scalar FMA units (DFMA, default) or the
// FP64 tensor cores (PHPC_FP64_PIPE=dmma); same bits either way.
bool fp64_pipe_is_dfma() {
  const char* pipe = getenv("PHPC_FP64_PIPE");
  return !(pipe && strcmp(pipe, "dmma") == 0);
}

// Tile side: a call takes as long as the SM with the most outputs (padding
// included), ceil(tiles / SMs) x BT^2, so the smaller tile is never behind by
// load (N = 1024 in 64 x 64 tiles: 2104 us, 2 tiles on some SMs, 1 on others;
// in 16 x 16: 1745). From 100 tiles of 32 x 32 an SM that difference is under
// 1 % and the larger tile's fewer loads count for more (N = 3000, 58 tiles an
// SM, K = 500: 16 7.49 ms, 32 7.55; N = 4096, 108 an SM: 110.4 and 110.15).
// Below that, 8 x 16 tiles (DFMA only; one output a thread) where they load the
// fullest SM less, or as much with at most eight 16 x 16 tiles on it (16 / 8:
// 64 x 2048 x 64 172.5 us, 103.1; 148 x 266 x 73 29.1, 18.8; 68 x 1384 x 1617
// 359, 317; 582 x 1605 x 336 617, 562; 250 x 514 x 302, as much, 74.1, 72.2; but
// N = 1024, as much with 27 tiles, 1733, 1739).
// PHPC_DMMA_TILE = 8 or 16 forces these, any other number 32.
int plain_tile(int m, int n, int sms) {
  if (const char* force = getenv("PHPC_DMMA_TILE")) {
    const int t = atoi(force);
    return t == 16 || t == 8 ? t : 32;
  }
  if ((int64_t)ceil_div(m, 32) * ceil_div(n, 32) >= (int64_t)100 * sms) return 32;
  const int64_t load16 = ((int64_t)ceil_div(m, 16) * ceil_div(n, 16) + sms - 1) / sms * 2;
  const int64_t load8 = ((int64_t)ceil_div(m, 8) * ceil_div(n, 16) + sms - 1) / sms;
  return load8 < load16 || (load8 == load16 && load16 <= 16) ? 8 : 16;
}

int dgemm_dmma(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, double* dC,
               int64_t ldc, int gw, int gh, int kpanel, cudaStream_t stream) {
  const DeviceInfo* dev = current_device();
  if (!dev) return PHPC_ERR_CUDA;
  if (dev->cc_major != 10 || dev->cc_minor != 3) return PHPC_ERR_UNSUPPORTED;
  auto launch = [&](auto tile) {
    constexpr int T = decltype(tile)::value;
    return fp64_pipe_is_dfma() ? launch_dmma<T, true>(m, k, n, dA, lda, dB, ldb, dC, ldc, gw, gh, kpanel, stream)
                               : launch_dmma<T == 8 ? 16 : T, false>(m, k, n, dA, lda, dB, ldb, dC, ldc, gw, gh,
                                                                     kpanel, stream);
  };
  switch (plain_tile(m, n, dev->sm_count)) {
    case 8: return launch(std::integral_constant<int, 8>());
    case 16: return launch(std::integral_constant<int, 16>());
    default: return launch(std::integral_constant<int, 32>());
  }
}

}  // namespace phpc

extern "C" int phpc_dgemm_dmma_dev(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb,
                                   double* dC, int64_t ldc, int grid_width, int grid_height, int kpanel,
                                   void* stream) {
  using namespace phpc;
  int rc = PHPC_OK;
  if (m < 0 || k < 0 || n < 0 || grid_width < 1 || grid_height < 1 || kpanel < 0 || (kpanel % kBK) != 0) {
    rc = PHPC_ERR_ARG;
  } else if (m == 0 || n == 0 || k == 0) {
    rc = PHPC_OK;  // C += 0
  } else if (!dA || !dB || !dC || lda < k || ldb < n || ldc < n) {
    rc = PHPC_ERR_ARG;
  } else if (!aligned16(dA) || !aligned16(dB) || (lda & 1) || (ldb & 1)) {
    rc = PHPC_ERR_ALIGN;
  } else {
    rc = dgemm_dmma(m, k, n, dA, lda, dB, ldb, dC, ldc, grid_width, grid_height, kpanel ? kpanel : 256,
                    static_cast<cudaStream_t>(stream));
  }
  set_last_error(rc);
  return rc;
}

extern "C" const char* phpc_fp64_pipe_name(void) { return phpc::fp64_pipe_is_dfma() ? "dfma" : "dmma"; }
