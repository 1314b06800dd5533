// One tile of the 3xBF16 GEMM with K split over a cluster of two CTAs, built
// with a short wait limit, for test_gpu_ksplit_giveup.py.
//
// short_rows > 0: B's tensor map has boxes that many rows short of a stage, so
// every load stays inside its plane and its buffer but brings fewer bytes than
// the stage's barrier expects: the MMA issuer's wait runs out, the kernel
// records it in the status word, waits for its copies and returns.
#include <cuda_bf16.h>

#include <vector>

#include "tc_gemm.cuh"

using namespace phpc;

namespace {
constexpr int kM = 128, kN = 128, kK = 512, kPlanes = 3, kSplit = 2;

template <class T>
bool upload(T** dev, const std::vector<T>& host) {
  return cudaMalloc(reinterpret_cast<void**>(dev), host.size() * sizeof(T)) == cudaSuccess &&
         cudaMemcpy(*dev, host.data(), host.size() * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess;
}
}  // namespace

// c[128 * 128], in and out; *status: the device status word afterwards.
// Planes of all ones: without a shortage every c grows by 6 * 512.
extern "C" int ksplit_tile(int short_rows, float* c, int* status) {
  constexpr auto kern = tc_slice_gemm_kernel<128, kF32, false, 1, true>;
  const DeviceInfo* dev = current_device();
  if (!dev || tc_ready<kern>(dev, TcCfg<128>::kSmem) != PHPC_OK) return 1;
  const std::vector<uint16_t> ones(static_cast<size_t>(kPlanes) * 128 * kK, 0x3F80);
  uint16_t *pa = nullptr, *pb = nullptr;
  float* dC = nullptr;
  if (!upload(&pa, ones) || !upload(&pb, ones) || !upload(&dC, std::vector<float>(c, c + kM * kN))) return 2;
  CUtensorMap tmA, tmB;
  const uint64_t dims[3] = {kK, 128, kPlanes}, strides[2] = {kK * 2, kK * 2 * 128};
  const uint32_t boxA[3] = {kTcBK, 128, 1}, boxB[3] = {kTcBK, 128u - static_cast<uint32_t>(short_rows), 1};
  if (!encode_tiled(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, pa, dims, strides, boxA, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !encode_tiled(&tmB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, pb, dims, strides, boxB, CU_TENSOR_MAP_SWIZZLE_128B))
    return 3;
  PairList pairs{};
  const int a[6] = {2, 1, 0, 1, 0, 0}, b[6] = {0, 1, 2, 0, 1, 0};
  pairs.n = 6;
  for (int i = 0; i < 6; ++i) {
    pairs.a[i] = static_cast<uint8_t>(a[i]);
    pairs.b[i] = static_cast<uint8_t>(b[i]);
  }
  TcArgs args{};
  args.M = kM;
  args.N = kN;
  args.K = kK;
  args.tm = args.tn = 1;
  args.group_rows = 8;
  args.C = dC;
  args.ldc = kN;
  args.status = device_status_ptr();
  args.ksplit = kSplit;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kSplit;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kSplit, 1, 1);
  cfg.blockDim = dim3(kTcThreads, 1, 1);
  cfg.dynamicSmemBytes = TcCfg<128>::kSmem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int rc = 0;
  if (cudaLaunchKernelEx(&cfg, kern, tmA, tmB, CUtensorMap{}, pairs, args, TcGroupTable{}) != cudaSuccess ||
      cudaDeviceSynchronize() != cudaSuccess ||
      cudaMemcpy(c, dC, sizeof(float) * kM * kN, cudaMemcpyDeviceToHost) != cudaSuccess)
    rc = 4;
  *status = phpc_device_status();
  cudaFree(pa);
  cudaFree(pb);
  cudaFree(dC);
  return rc;
}
