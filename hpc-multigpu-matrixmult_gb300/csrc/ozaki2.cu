// FP64-accurate GEMM by the modular (Chinese-remainder) Ozaki scheme on
// tcgen05 BF16 tensor cores.
//
// C += A * B (the reference's semantics, src/phpc_gemm.cu:55) computed as:
//  1. Scans: ea[i] = max_k e(A[i][k]), eb[j] = max_k e(B[k][j]) (as in
//     ozaki.cu), and each row's (column's) grid width ba[i] (bb[j]) from an
//     upper bound of its Euclidean norm (residue.cuh, grid_bits).
//  2. Residue split: each element becomes the integer
//     A'[i][k] = sign * round(|A[i][k]| * 2^(ba[i] - ea[i])) (B' likewise
//     with eb[j], bb[j]), and then its symmetric residues modulo n pairwise
//     coprime moduli m_1..m_n <= 363: integers with |r| <= 181, exact in BF16
//     (residue.cuh). Planes A_i = [n][M][ldp], B_i = [n][N][ldp] (transposed,
//     K-major).
//  3. n residue GEMMs on the tcgen05 engine (tc_gemm.cuh, kResidue): A_i * B_i^T
//     mod m_i (exact f32 chunks of 512 products, each reduced mod m_i in FP32
//     and summed exactly), one 16-bit residue per element, into plane i of R.
//  4. CRT (this file): C_int = sum_i r_i * W_i mod M, W_i = (M/m_i) *
//     ((M/m_i)^-1 mod m_i), M = prod m_i (crt.cuh: on FP32 limbs when the
//     grids guarantee |C_int| / M <= 1/2 - 1/32, else in 160-bit integers);
//     the grids keep |A'_i| |B'_j| <= M (1/2 - 1/32), so the symmetric
//     representative of C_int is the exact integer product A' * B'^T.
//     C += round_to_double(C_int) * 2^(ea[i] - ba[i] + eb[j] - bb[j]).
//
// Compared with the digit scheme (s slices, s(s+1)/2 slice products) the
// tensor-core work is n GEMMs with no triangular truncation. With the
// worst-case grid (2 K 2^(2b) < M) n = 14 gives b = 51 at K = 16384; the
// norm-based grids add what the data allow (about 1.3 bits for uniform
// entries, 3.7 for entries spread over 2^-20 .. 2^20).
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "ozaki_digits.cuh"
#include "phpc_host.hpp"
#include "residue.cuh"
#include "tc_gemm.cuh"

namespace phpc {

namespace {

// The A side (rows) and the B side (columns) of one operand preparation.
// Either may be empty (rows / cols = 0): the two kernels below run one side
// or both in one launch, A's blocks first.
struct PrepRows {
  const double* A;
  int64_t lda;
  int rows;
  int* ea;
  int* ba;
  uint16_t* planes;  // [n][.][ldp]
  int64_t plane_stride;
};
struct PrepCols {
  const double* B;
  int64_t ldb;
  int cols;
  int64_t ldpart;
  int* pe;
  float* ps;
  int* eb;
  int* bb;
  uint16_t* planes;  // [n][.][ldp], transposed
  int64_t plane_stride;
  int merge;  // the split merges the scan's chunks itself
};

constexpr int kPrepThreads = 256;
constexpr int kOneStreamK = 2560;  // ozaki2_prepare_on
constexpr int kScanRowsPerBlock = kPrepThreads / 32;  // one warp per row

// Row blocks: one warp per row of A: ea[i] = max_k e(A[i][k]) and the row's
// grid width. Column blocks (scan part 1): strip of 32 columns, chunk of 256
// rows; warp w sums rows 32 w .. + 31 of the chunk, and warp 0 merges the eight
// slices in order into pe / ps [chunk][n]. A column's chain is 32 FMAs with 16
// loads in flight, and even N = 256 has 8 blocks; one thread per column and
// 256 rows took 53-59 us at every size up to N = 4096 (the chain's latency)
// and 410 us at N = 16384, against 4 us at N = 256, 5.5 at 1024, 22 at 4096
// and 292 at 16384 (7.3 TB/s) for this.
__global__ void __launch_bounds__(kPrepThreads) scan_kernel(const PrepRows a, const PrepCols b, int row_blocks,
                                                            int strips, int K, float logT, int* status) {
  __shared__ int se[8][32];
  __shared__ float ss[8][32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  pdl_trigger();
  NormAcc acc;
  bool nf = false;
  if (static_cast<int>(blockIdx.x) < row_blocks) {
    const int64_t row = (int64_t)blockIdx.x * kScanRowsPerBlock + w;
    if (row >= a.rows) return;
    norm_row_lane(a.A + row * a.lda, K, l, acc, nf);
    acc = norm_warp(acc);
    if (l == 0) {
      a.ea[row] = acc.e;
      a.ba[row] = grid_bits(acc.s, K, logT);
    }
    if (__any_sync(0xffffffffu, nf) && l == 0) record_error(status, PHPC_ERR_NONFINITE);
    return;
  }
  const int blk = blockIdx.x - row_blocks, chunk = blk / strips;
  const int64_t col = (int64_t)(blk - chunk * strips) * 32 + l;
  const int k0 = chunk * kNormChunk + w * kNormSlice;
  if (col < b.cols && k0 < K) norm_col_slice(b.B, b.ldb, col, k0, K, acc, nf);
  se[w][l] = acc.e;
  ss[w][l] = acc.s;
  if (nf) record_error(status, PHPC_ERR_NONFINITE);
  __syncthreads();
  if (w != 0 || col >= b.cols) return;
  acc = NormAcc{};
#pragma unroll
  for (int u = 0; u < 8; ++u) norm_merge(acc, NormAcc{se[u][l], ss[u][l]});
  b.pe[chunk * b.ldpart + col] = acc.e;
  b.ps[chunk * b.ldpart + col] = acc.s;
}

// Column scan, part 2: a block merges the chunks of 32 columns, warp p those
// numbered p, p + 8, ..., into eb[j] and bb[j].
// (No __restrict__ on what the scan writes: see launch_dependent.)
__global__ void __launch_bounds__(256) scan_cols_merge_kernel(int K, int N, int64_t ldpart, const int* pe,
                                                              const float* ps, int* eb, int* bb, float logT) {
  __shared__ int se[8][32];
  __shared__ float ss[8][32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int64_t col = (int64_t)blockIdx.x * 32 + l;
  const int chunks = (K + kNormChunk - 1) / kNormChunk;
  pdl_trigger();
  pdl_wait();
  NormAcc acc = norm_merge_strided(pe, ps, ldpart, col, col < N ? chunks : 0, w);
  se[w][l] = acc.e;
  ss[w][l] = acc.s;
  __syncthreads();
  if (w != 0 || col >= N) return;
  NormAcc q[8];
#pragma unroll
  for (int p = 0; p < 8; ++p) q[p] = NormAcc{se[p][l], ss[p][l]};
  acc = norm_merge_tree(q);
  eb[col] = acc.e;
  bb[col] = grid_bits(acc.s, K, logT);
}

// Up to this many chunks (K <= 1024) the split merges them itself: a merge
// kernel is 3-4 us of a small call, the merge in every block of the
// split 0.6 us of 11 at N = 1024 (but 22 us of 120 at N = 4096, 0.9 ms of
// 2.4 at 16384).
constexpr int kMergeInSplit = 4;

// Row blocks: A residue planes [n][M][ldp], a thread per row piece (8
// consecutive k of one row). A block takes 256 consecutive pieces of a row,
// rows first (the rows' pieces of one range of k together: 1.43 ms at N =
// 16384 against 1.44-1.65 with a row's ranges together); what is left of the
// rows, or rows shorter than that, is numbered row by row, so that the blocks
// are full. Column blocks: B residue planes, transposed
// ([n][N][ldp]), one kColBlockK x kColBlockJ block each (residue.cuh); with
// b.merge the eight threads of a column merge its chunks into the exponent
// and grid width, and the first row of blocks stores them in eb / bb for the
// CRT; without, eb / bb are there.
template <int NMOD>
__global__ void __launch_bounds__(kPrepThreads, 4)
    residue_split_kernel(const PrepRows a, const PrepCols b, int row_blocks, int strips, int K, int64_t ldp,
                         const __grid_constant__ ModTable T) {
  __shared__ double tile[kColBlockK][kColBlockJ];
  pdl_trigger();
  pdl_wait();
  if (static_cast<int>(blockIdx.x) < row_blocks) {
    const int per_row = (K + 7) >> 3, ranges = per_row / kPrepThreads, left = per_row - ranges * kPrepThreads;
    const int64_t blk = blockIdx.x, full = (int64_t)a.rows * ranges;
    int64_t row, piece;
    if (blk < full) {
      const int range = static_cast<int>(blk / a.rows);
      row = blk - (int64_t)range * a.rows;
      piece = range * kPrepThreads + threadIdx.x;
    } else {
      const int64_t t = (blk - full) * kPrepThreads + threadIdx.x, pieces = (int64_t)a.rows * left;
      if (t >= pieces) return;
      row = pieces <= UINT32_MAX ? static_cast<uint32_t>(t) / static_cast<uint32_t>(left) : t / left;
      piece = ranges * kPrepThreads + (t - row * left);
    }
    residue_row_piece<NMOD>(a.A + row * a.lda, K, a.ea[row], a.ba[row], T, a.planes + row * ldp, a.plane_stride,
                            piece * 8);
    return;
  }
  const int blk = blockIdx.x - row_blocks, kb = blk / strips;
  const int64_t j0 = (int64_t)(blk - kb * strips) * kColBlockJ, col = j0 + (threadIdx.x >> 3);
  int e, bits;
  if (b.merge) {
    const int chunks = (K + kNormChunk - 1) / kNormChunk;
    const NormAcc acc = norm_merge_chunks8(b.pe, b.ps, b.ldpart, col, col < b.cols ? chunks : 0, threadIdx.x & 7);
    e = acc.e;
    bits = grid_bits(acc.s, K, T.logT);
    if (kb == 0 && col < b.cols && (threadIdx.x & 7) == 0) {
      b.eb[col] = e;
      b.bb[col] = bits;
    }
  } else {
    e = col < b.cols ? b.eb[col] : 0;
    bits = col < b.cols ? b.bb[col] : 0;
  }
  residue_col_block<NMOD>(b.B, b.ldb, K, b.cols, j0, (int64_t)kb * kColBlockK, e, bits, T, b.planes, ldp,
                          b.plane_stride, tile);
}

// C[i][j] += C_int * 2^(ea[i] - ba[i] + eb[j] - bb[j]), C_int recovered from
// the residues. (No __restrict__ on what earlier grids write: see launch_dependent.)
template <int NMOD>
__global__ void __launch_bounds__(128, crt_min_blocks(NMOD, false))
    crt_kernel(const uint16_t* R, int64_t ldr, int64_t rplane, int M, int N, const int* ea, const int* ba,
               const int* eb, const int* bb, const __grid_constant__ ModTable T, double* C, int64_t ldc) {
  const int64_t row = blockIdx.x;
  const int64_t c0 = ((int64_t)blockIdx.y * blockDim.x + threadIdx.x) * kCrtCols;
  pdl_wait();
  if (row >= M || c0 >= N) return;
  crt_cols<NMOD>(R + row * ldr + c0, rplane, T.crt, T.crt.fast, static_cast<int>(min(static_cast<int64_t>(kCrtCols), N - c0)),
           max(ea[row], -20000) - ba[row], eb + c0, bb + c0, C + row * ldc + c0);
}

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct Ozaki2Layout {
  int64_t ldp, ldr, ldpart;
  size_t off_ea, off_eb, off_ba, off_bb, off_pe, off_ps, off_pa, off_pb, off_r, total;
};

// Workspace: ea[m], eb[n], ba[m], bb[n], the column scan's chunk partials
// pe / ps [ceil(k / 256)][n], A planes, B planes, residues.
Ozaki2Layout ozaki2_layout(int m, int k, int n, int nmod, bool padded = true) {
  Ozaki2Layout L;
  L.ldp = plane_ld(k, padded);
  L.ldr = ((int64_t)n + 15) / 16 * 16;
  L.ldpart = n;
  const size_t chunks = (static_cast<size_t>(k) + kNormChunk - 1) / kNormChunk;
  L.off_ea = 0;
  L.off_eb = align256(sizeof(int) * (size_t)m);
  L.off_ba = align256(L.off_eb + sizeof(int) * (size_t)n);
  L.off_bb = align256(L.off_ba + sizeof(int) * (size_t)m);
  L.off_pe = align256(L.off_bb + sizeof(int) * (size_t)n);
  L.off_ps = align256(L.off_pe + sizeof(int) * chunks * n);
  L.off_pa = align256(L.off_ps + sizeof(float) * chunks * n);
  L.off_pb = align256(L.off_pa + (size_t)nmod * m * L.ldp * 2);
  L.off_r = align256(L.off_pb + (size_t)nmod * n * L.ldp * 2);
  L.total = align256(L.off_r + (size_t)nmod * m * L.ldr * 2);
  return L;
}

struct Ozaki2Views {
  int* ea;
  int* eb;
  int* ba;
  int* bb;
  int* pe;
  float* ps;
  uint16_t* pa;
  uint16_t* pb;
  uint16_t* R;
};

int ozaki2_views(int m, int k, int n, int nmod, const void* ws, size_t ws_bytes, Ozaki2Layout& L, Ozaki2Views& V) {
  const DeviceInfo* dev = current_device();
  if (!dev) return PHPC_ERR_CUDA;
  if (dev->cc_major != 10 || dev->cc_minor != 3) return PHPC_ERR_UNSUPPORTED;
  L = ozaki2_layout(m, k, n, nmod);
  if (ws_bytes < L.total) L = ozaki2_layout(m, k, n, nmod, false);
  if (!ws || ws_bytes < L.total || !aligned16(ws)) return PHPC_ERR_WORKSPACE;
  uint8_t* base = static_cast<uint8_t*>(const_cast<void*>(ws));
  V.ea = reinterpret_cast<int*>(base + L.off_ea);
  V.eb = reinterpret_cast<int*>(base + L.off_eb);
  V.ba = reinterpret_cast<int*>(base + L.off_ba);
  V.bb = reinterpret_cast<int*>(base + L.off_bb);
  V.pe = reinterpret_cast<int*>(base + L.off_pe);
  V.ps = reinterpret_cast<float*>(base + L.off_ps);
  V.pa = reinterpret_cast<uint16_t*>(base + L.off_pa);
  V.pb = reinterpret_cast<uint16_t*>(base + L.off_pb);
  V.R = reinterpret_cast<uint16_t*>(base + L.off_r);
  return PHPC_OK;
}

}  // namespace

size_t ozaki2_workspace_bytes(int m, int k, int n, int nmod) { return ozaki2_layout(m, k, n, nmod).total; }

int ozaki2_bits(int nmod, int k) { return make_table(nmod, k).bits; }

namespace {

// Scans and residue splits of a's rows and b's columns (either side may be
// empty): two launches, three when the chunks of the column scan are merged
// between them.
int prepare_operands(const PrepRows& a, PrepCols b, int k, int64_t ldp, const ModTable& T, cudaStream_t stream) {
  const int strips = ceil_div(b.cols, 32), chunks = ceil_div(k, kNormChunk);
  const int scan_rows = ceil_div(a.rows, kScanRowsPerBlock);
  const int ranges = ceil_div(k, 8) / kPrepThreads, left = ceil_div(k, 8) - ranges * kPrepThreads;
  const int split_rows = a.rows * ranges + ceil_div((int64_t)a.rows * left, kPrepThreads);
  b.merge = chunks <= kMergeInSplit;
  const bool both = a.rows > 0 && b.cols > 0;  // one side: another stream's kernels share the SMs
  scan_kernel<<<scan_rows + strips * chunks, kPrepThreads, 0, stream>>>(a, b, scan_rows, strips, k, T.logT,
                                                                        device_status_ptr());
  PHPC_CUDA_TRY(cudaGetLastError());
  if (b.cols > 0 && !b.merge)
    PHPC_CUDA_TRY(launch_dependent(both, scan_cols_merge_kernel, strips, 256, 0, stream, k, b.cols, b.ldpart, b.pe,
                                   b.ps, b.eb, b.bb, T.logT));
  cudaError_t e = cudaSuccess;
  with_crt_moduli(T.n, [&](auto nm) {
    e = launch_dependent(both, residue_split_kernel<decltype(nm)::value>, split_rows + strips * ceil_div(k, kColBlockK),
                         kPrepThreads, 0, stream, a, b, split_rows, strips, k, ldp, T);
  });
  PHPC_CUDA_TRY(e);
  return PHPC_OK;
}
static_assert(kColBlockJ == 32, "scan strips are the split's column blocks");

PrepRows prep_rows(int m, int r0, int rows, const double* dA, int64_t lda, const Ozaki2Layout& L,
                   const Ozaki2Views& V) {
  return PrepRows{dA + (int64_t)r0 * lda, lda,         rows, V.ea + r0, V.ba + r0, V.pa + (int64_t)r0 * L.ldp,
                  (int64_t)m * L.ldp};
}

PrepCols prep_cols(int n, int c0, int cols, const double* dB, int64_t ldb, const Ozaki2Layout& L,
                   const Ozaki2Views& V) {
  return PrepCols{dB + c0,   ldb,       cols,      L.ldpart, V.pe + c0, V.ps + c0,
                  V.eb + c0, V.bb + c0, V.pb + (int64_t)c0 * L.ldp, (int64_t)n * L.ldp, 0};
}

}  // namespace

// Rows [r0, r0 + rows) of A (an m x k operand, dA its row 0): exponent and
// grid scan, and residue split into the planes of the full problem.
int ozaki2_prepare_a_rows(int m, int r0, int rows, int k, int n, const double* dA, int64_t lda, int nmod, void* ws,
                          size_t ws_bytes, cudaStream_t stream) {
  Ozaki2Layout L;
  Ozaki2Views V;
  const int rc = ozaki2_views(m, k, n, nmod, ws, ws_bytes, L, V);
  if (rc != PHPC_OK) return rc;
  if (r0 < 0 || rows <= 0 || r0 + rows > m) return PHPC_ERR_ARG;
  return prepare_operands(prep_rows(m, r0, rows, dA, lda, L, V), PrepCols{}, k, L.ldp, make_table(nmod, k), stream);
}

// Columns [c0, c0 + cols) of B (k x n, dB its column 0): exponent and grid
// scan, and residue split into the planes of the full problem.
int ozaki2_prepare_b_cols(int m, int k, int n, int c0, int cols, const double* dB, int64_t ldb, int nmod, void* ws,
                          size_t ws_bytes, cudaStream_t stream) {
  Ozaki2Layout L;
  Ozaki2Views V;
  const int rc = ozaki2_views(m, k, n, nmod, ws, ws_bytes, L, V);
  if (rc != PHPC_OK) return rc;
  if (c0 < 0 || cols <= 0 || c0 + cols > n) return PHPC_ERR_ARG;
  return prepare_operands(PrepRows{}, prep_cols(n, c0, cols, dB, ldb, L, V), k, L.ldp, make_table(nmod, k), stream);
}

// B (k x n): exponent and grid scan, and residue split.
int ozaki2_prepare_b(int m, int k, int n, const double* dB, int64_t ldb, int nmod, void* ws, size_t ws_bytes,
                     cudaStream_t stream) {
  return ozaki2_prepare_b_cols(m, k, n, 0, n, dB, ldb, nmod, ws, ws_bytes, stream);
}

// Exponent scans and residue splits: A's on stream_a, B's on stream_b.
int ozaki2_prepare2(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, int nmod,
                    void* ws, size_t ws_bytes, cudaStream_t stream_a, cudaStream_t stream_b) {
  int rc = ozaki2_prepare_a_rows(m, 0, m, k, n, dA, lda, nmod, ws, ws_bytes, stream_a);
  if (rc == PHPC_OK) rc = ozaki2_prepare_b(m, k, n, dB, ldb, nmod, ws, ws_bytes, stream_b);
  return rc;
}

// The same on one caller stream. Small operands (below 32 MB together, and K
// <= 2560) share the two or three launches: the fork and join cost more than
// the overlap gives (prepare alone, two streams / one: N = 256 13.5, 8.7 us;
// 664 x 1420 x 668 26.8, 22.9; 1537 x 1000 x 2311 40.3, 37.3; but 4096 x 1024 x
// 4096 72.1, 74.2). With longer rows a warp's scan of one row, which B's work
// on the other stream hides, takes as long as they do (569 x 3453 x 178 31.3,
// 33.1; 387 x 5556 x 580 53.7, 59.8; 256 x 8192 x 256 47.6, 55.8). Above,
// B's scans and split run on this thread's side stream beside A's (both are
// memory-bound; run together, one's ramp-up and tail overlap the other's), and
// the caller's stream waits for them.
// *joined: whether another stream's work joined it (then the next launch does
// not directly follow a kernel).
int ozaki2_prepare_on(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, int nmod,
                      void* ws, size_t ws_bytes, cudaStream_t stream, bool* joined = nullptr) {
  if (joined) *joined = false;
  if (k <= kOneStreamK && ((int64_t)m + n) * k < (4 << 20)) {
    Ozaki2Layout L;
    Ozaki2Views V;
    const int rc = ozaki2_views(m, k, n, nmod, ws, ws_bytes, L, V);
    if (rc != PHPC_OK) return rc;
    return prepare_operands(prep_rows(m, 0, m, dA, lda, L, V), prep_cols(n, 0, n, dB, ldb, L, V), k, L.ldp,
                            make_table(nmod, k), stream);
  }
  const cudaStream_t side = side_stream();
  if (!side || !stream_fork(stream, side)) return ozaki2_prepare2(m, k, n, dA, lda, dB, ldb, nmod, ws, ws_bytes, stream, stream);
  if (joined) *joined = true;
  int rc = ozaki2_prepare2(m, k, n, dA, lda, dB, ldb, nmod, ws, ws_bytes, stream, side);
  if (!stream_fork(side, stream) && rc == PHPC_OK) rc = PHPC_ERR_CUDA;
  return rc;
}

// The residue GEMMs of the block rows [r0, r0 + rows) x columns [c0, c0 +
// cols): plane i of R = (A_i * B_i^T) mod m_i, one 16-bit residue per element.
// Tile width, cluster and raster are those of the full m x k x n problem.
int ozaki2_multiply_block(int m, int r0, int rows, int c0, int cols, int k, int n, int nmod, const void* ws,
                          size_t ws_bytes, cudaStream_t stream, int bn, bool dependent) {
  Ozaki2Layout L;
  Ozaki2Views V;
  const int rc = ozaki2_views(m, k, n, nmod, ws, ws_bytes, L, V);
  if (rc != PHPC_OK) return rc;
  if (r0 < 0 || rows <= 0 || r0 + rows > m || c0 < 0 || cols <= 0 || c0 + cols > n || c0 % 8) return PHPC_ERR_ARG;
  const ModTable T = make_table(nmod, k);
  PairList pl{};
  pl.n = nmod;
  for (int i = 0; i < nmod; ++i) {
    pl.a[i] = static_cast<uint8_t>(i);
    pl.b[i] = static_cast<uint8_t>(i);
    pl.g[i] = static_cast<uint8_t>(i);
    pl.mod[i] = static_cast<uint16_t>(T.m[i]);
    pl.invm[i] = T.invm[i].x;
  }
  const int64_t rplane = (int64_t)m * L.ldr;
  const uint16_t* pa = V.pa + (int64_t)r0 * L.ldp;
  const uint16_t* pb = V.pb + (int64_t)c0 * L.ldp;
  uint16_t* R = V.R + (int64_t)r0 * L.ldr + c0;
  TcGemmOpts opt;
  opt.a_plane_rows = m;
  opt.b_plane_rows = n;
  opt.cfg_m = m;
  opt.cfg_n = n;
  opt.cfg_k = k;
  opt.dependent = dependent;
  return bn == 128 ? launch_tc_slice_gemm<128, kResidue>(pa, pb, nmod, nmod, L.ldp, rows, cols, k, pl, nullptr, 0,
                                                          nullptr, nullptr, stream, R, L.ldr, rplane, opt)
                   : launch_tc_slice_gemm<256, kResidue>(pa, pb, nmod, nmod, L.ldp, rows, cols, k, pl, nullptr, 0,
                                                          nullptr, nullptr, stream, R, L.ldr, rplane, opt);
}

// The residue GEMMs of rows [r0, r0 + rows), all columns.
int ozaki2_multiply_rows(int m, int r0, int rows, int k, int n, int nmod, const void* ws, size_t ws_bytes,
                         cudaStream_t stream, int bn) {
  return ozaki2_multiply_block(m, r0, rows, 0, n, k, n, nmod, ws, ws_bytes, stream, bn);
}

int ozaki2_multiply(int m, int k, int n, int nmod, const void* ws, size_t ws_bytes, cudaStream_t stream, int bn) {
  return ozaki2_multiply_rows(m, 0, m, k, n, nmod, ws, ws_bytes, stream, bn);
}

// Rows [r0, r0 + rows) of C (dC its row 0) += CRT(R) * 2^(ea - ba + eb - bb).
int ozaki2_reconstruct_rows(int m, int r0, int rows, int k, int n, double* dC, int64_t ldc, int nmod, const void* ws,
                            size_t ws_bytes, cudaStream_t stream, bool dependent) {
  Ozaki2Layout L;
  Ozaki2Views V;
  const int rc = ozaki2_views(m, k, n, nmod, ws, ws_bytes, L, V);
  if (rc != PHPC_OK) return rc;
  if (r0 < 0 || rows <= 0 || r0 + rows > m) return PHPC_ERR_ARG;
  const ModTable T = make_table(nmod, k);
  if (T.crt.L.np != crt_digits(T.n)) return PHPC_ERR_UNSUPPORTED;  // the kernels' digit count per modulus count
  cudaError_t e = cudaSuccess;
  with_crt_moduli(T.n, [&](auto nm) {
    e = launch_dependent(dependent, crt_kernel<decltype(nm)::value>, dim3(rows, ceil_div(n, 128 * kCrtCols)), 128, 0,
                         stream, V.R + (int64_t)r0 * L.ldr, L.ldr, (int64_t)m * L.ldr, rows, n, V.ea + r0, V.ba + r0,
                         V.eb, V.bb, T, dC + (int64_t)r0 * ldc, ldc);
  });
  PHPC_CUDA_TRY(e);
  return PHPC_OK;
}

// Copies the grids of the last scans (exponents and grid widths of the rows
// of A and the columns of B) to host arrays (synchronous).
int ozaki2_grids(int m, int k, int n, int nmod, const void* ws, size_t ws_bytes, int* ea, int* eb, int* ba, int* bb) {
  Ozaki2Layout L;
  Ozaki2Views V;
  const int rc = ozaki2_views(m, k, n, nmod, ws, ws_bytes, L, V);
  if (rc != PHPC_OK) return rc;
  PHPC_CUDA_TRY(cudaMemcpy(ea, V.ea, sizeof(int) * m, cudaMemcpyDeviceToHost));
  PHPC_CUDA_TRY(cudaMemcpy(eb, V.eb, sizeof(int) * n, cudaMemcpyDeviceToHost));
  PHPC_CUDA_TRY(cudaMemcpy(ba, V.ba, sizeof(int) * m, cudaMemcpyDeviceToHost));
  PHPC_CUDA_TRY(cudaMemcpy(bb, V.bb, sizeof(int) * n, cudaMemcpyDeviceToHost));
  return PHPC_OK;
}

int ozaki2_reconstruct(int m, int k, int n, double* dC, int64_t ldc, int nmod, const void* ws, size_t ws_bytes,
                       cudaStream_t stream) {
  return ozaki2_reconstruct_rows(m, 0, m, k, n, dC, ldc, nmod, ws, ws_bytes, stream);
}

// In a short call each launch after the first comes up while the one before it
// finishes (the GEMM's set-up of 208 KB of shared memory, barriers and TMEM
// among it): N = 256 24.6 -> 20 us.
int dgemm_ozaki2(int m, int k, int n, const double* dA, int64_t lda, const double* dB, int64_t ldb, double* dC,
                 int64_t ldc, int nmod, void* ws, size_t ws_bytes, cudaStream_t stream, int bn) {
  const DeviceInfo* dev = current_device();
  if (!dev) return PHPC_ERR_CUDA;
  bool joined = false;
  const bool is_short = short_gemm(m, n, (int64_t)nmod * ceil_div(k, 64), dev->sm_count);
  int rc = ozaki2_prepare_on(m, k, n, dA, lda, dB, ldb, nmod, ws, ws_bytes, stream, &joined);
  if (rc == PHPC_OK) rc = ozaki2_multiply_block(m, 0, m, 0, n, k, n, nmod, ws, ws_bytes, stream, bn, !joined);
  if (rc == PHPC_OK) rc = ozaki2_reconstruct_rows(m, 0, m, k, n, dC, ldc, nmod, ws, ws_bytes, stream, is_short);
  return rc;
}

}  // namespace phpc

extern "C" size_t phpc_ozaki2_workspace_bytes(int m, int k, int n, int moduli) {
  if (m <= 0 || k <= 0 || n <= 0 || moduli < phpc::kMinModuli || moduli > phpc::kMaxModuli) return 0;
  return phpc::ozaki2_workspace_bytes(m, k, n, moduli);
}

namespace {

// Shared argument checks of the device entry points: PHPC_OK when the call
// may proceed (the callers skip empty problems).
int ozaki2_args(int m, int k, int n, int moduli, bool need_a, const double* dA, int64_t lda, bool need_b,
                const double* dB, int64_t ldb, bool need_c, const double* dC, int64_t ldc) {
  using namespace phpc;
  if (m < 0 || k < 0 || n < 0 || moduli < kMinModuli || moduli > kMaxModuli) return PHPC_ERR_ARG;
  if (m == 0 || n == 0 || k == 0) return PHPC_OK;
  if ((need_a && (!dA || lda < k)) || (need_b && (!dB || ldb < n)) || (need_c && (!dC || ldc < n)))
    return PHPC_ERR_ARG;
  if (m > 65535 * 128 || k > 65535 * 32) return PHPC_ERR_ARG;  // launch-grid limits of the split kernels
  return PHPC_OK;
}

}  // namespace

extern "C" int phpc_default_moduli(int m, int k, int n) { return phpc::default_moduli(m, k, n); }

extern "C" int phpc_ozaki2_prepare_dev(int m, int k, int n, const double* dA, int64_t lda, const double* dB,
                                       int64_t ldb, int moduli, void* workspace, size_t workspace_bytes,
                                       void* stream) {
  int rc = ozaki2_args(m, k, n, moduli, true, dA, lda, true, dB, ldb, false, nullptr, 0);
  if (rc == PHPC_OK && m > 0 && n > 0 && k > 0) {
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    rc = phpc::ozaki2_prepare_on(m, k, n, dA, lda, dB, ldb, moduli, workspace, workspace_bytes, st);
  }
  phpc::set_last_error(rc);
  return rc;
}

extern "C" int phpc_ozaki2_multiply_dev(int m, int k, int n, int moduli, void* workspace, size_t workspace_bytes,
                                        void* stream) {
  int rc = ozaki2_args(m, k, n, moduli, false, nullptr, 0, false, nullptr, 0, false, nullptr, 0);
  if (rc == PHPC_OK && m > 0 && n > 0 && k > 0)
    rc = phpc::ozaki2_multiply(m, k, n, moduli, workspace, workspace_bytes, static_cast<cudaStream_t>(stream),
                               phpc::modular_bn(m, k, n, moduli));
  phpc::set_last_error(rc);
  return rc;
}

extern "C" int phpc_ozaki2_reconstruct_dev(int m, int k, int n, double* dC, int64_t ldc, int moduli, void* workspace,
                                           size_t workspace_bytes, void* stream) {
  int rc = ozaki2_args(m, k, n, moduli, false, nullptr, 0, false, nullptr, 0, true, dC, ldc);
  if (rc == PHPC_OK && m > 0 && n > 0 && k > 0)
    rc = phpc::ozaki2_reconstruct(m, k, n, dC, ldc, moduli, workspace, workspace_bytes,
                                  static_cast<cudaStream_t>(stream));
  phpc::set_last_error(rc);
  return rc;
}

extern "C" int phpc_dgemm_ozaki2_dev(int m, int k, int n, const double* dA, int64_t lda, const double* dB,
                                     int64_t ldb, double* dC, int64_t ldc, int moduli, void* workspace,
                                     size_t workspace_bytes, void* stream) {
  int rc = ozaki2_args(m, k, n, moduli, true, dA, lda, true, dB, ldb, true, dC, ldc);
  if (rc == PHPC_OK && m > 0 && n > 0 && k > 0)
    rc = phpc::dgemm_ozaki2(m, k, n, dA, lda, dB, ldb, dC, ldc, moduli, workspace, workspace_bytes,
                            static_cast<cudaStream_t>(stream), phpc::modular_bn(m, k, n, moduli));
  phpc::set_last_error(rc);
  return rc;
}

extern "C" int phpc_ozaki2_grids(int m, int k, int n, int moduli, const void* workspace, size_t workspace_bytes,
                                 int* ea, int* eb, int* ba, int* bb) {
  int rc = PHPC_OK;
  if (m <= 0 || k <= 0 || n <= 0 || moduli < phpc::kMinModuli || moduli > phpc::kMaxModuli || !ea || !eb || !ba ||
      !bb)
    rc = PHPC_ERR_ARG;
  if (rc == PHPC_OK) rc = phpc::ozaki2_grids(m, k, n, moduli, workspace, workspace_bytes, ea, eb, ba, bb);
  phpc::set_last_error(rc);
  return rc;
}
