// Checks of the block kernel that need its own launch words: runs that begin with an error word or with a small visit cap,
// and a wait for a copy that nobody issued.  Built by tests/test_gpu_block_failure.py.
#include <cstdint>
#include <cstring>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include "dtb_block.cuh"

using namespace dtb;

namespace {

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess) return nullptr;
  return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
}

bool encode(CUtensorMap* tm, const void* base, uint64_t w, uint64_t h, uint64_t pitch, uint32_t box_w, uint32_t box_h) {
  static const auto fn = encoder();
  cuuint64_t dims[2] = {w, h}, strides[1] = {pitch};
  cuuint32_t box[2] = {box_w, box_h}, estr[2] = {1, 1};
  return fn && fn(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

__global__ void wait_for_nothing(QueueHdr* hdr, uint32_t* out) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
  Queue q{};
  q.hdr = hdr;
  uint32_t bits = 0;
  const bool ok = tma_wait(&bar, bits, 1u, q, 77u);
  if (threadIdx.x == 0) {
    out[0] = ok;
    out[1] = bits & STAGE_LOST ? 1u : 0u;
  }
}

}  // namespace

// One gray image through ggdt_block<BLOCK_CTAS>; out: error word, its detail, tile visits, blocks.  Negative: set-up failed.
extern "C" __attribute__((visibility("default"))) int block_run(const uint8_t* img, int64_t img_pitch, const uint8_t* mask,
                                                                int64_t mask_pitch, float* dist, int64_t dist_pitch, int w, int h,
                                                                float g2, float v, uint32_t error, uint32_t max_visits,
                                                                uint32_t* out) {
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0) != cudaSuccess) return -1;
  ImgDesc d{};
  d.img = img;
  d.mask = mask;
  d.dist = dist;
  d.img_pitch = img_pitch;
  d.mask_pitch = mask_pitch;
  d.dist_pitch = dist_pitch;
  d.width = w;
  d.height = h;
  d.channels = 1;
  d.tiles_x = (w + TILE - 1) / TILE;
  d.tiles_y = (h + TILE - 1) / TILE;
  d.blocks_x = (w + BLOCK_W - 1) / BLOCK_W;
  d.blocks_y = (h + BLOCK_H - 1) / BLOCK_H;
  d.g2 = g2;
  d.v = v;
  d.mode = MODE_NS;
  const uint32_t blocks = (uint32_t)(d.blocks_x * d.blocks_y);
  const uint32_t grid = blocks < (uint32_t)(sms * BLOCK_CTAS) ? blocks : (uint32_t)(sms * BLOCK_CTAS);
  if (blocks > grid * (uint32_t)BLOCK_OWNED_MAX) return -2;
  CUtensorMap tm[2];
  if (!encode(&tm[0], img, (uint64_t)w, (uint64_t)h, (uint64_t)img_pitch, IMG_BOX_GRAY, IMG_BOX_ROWS) ||
      !encode(&tm[1], mask, (uint64_t)w, (uint64_t)h, (uint64_t)mask_pitch, TILE, TILE))
    return -3;
  const size_t o_msg = (sizeof(QueueHdr) + 255) / 256 * 256, o_desc = (o_msg + 32ull * blocks + 255) / 256 * 256,
               o_tm = o_desc + 256, o_base = o_tm + 256, bytes = o_base + 256;
  uint8_t* dev = nullptr;
  if (cudaMalloc(&dev, bytes) != cudaSuccess) return -4;
  QueueHdr hdr{};
  hdr.error.v = error;
  const uint32_t base[2] = {0, blocks};
  bool ok = cudaMemset(dev, 0, bytes) == cudaSuccess &&
            cudaMemcpy(dev, &hdr, sizeof(hdr), cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(dev + o_desc, &d, sizeof(d), cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(dev + o_tm, tm, sizeof(tm), cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(dev + o_base, base, sizeof(base), cudaMemcpyHostToDevice) == cudaSuccess;
  BlockRun a{};
  a.hdr = reinterpret_cast<QueueHdr*>(dev);
  a.msg = reinterpret_cast<uint2*>(dev + o_msg);
  a.base = reinterpret_cast<const uint32_t*>(dev + o_base);
  a.n = 1;
  a.total = blocks;
  a.max_visits = max_visits;
  a.timeout_ns = 2000000000ull;
  const void* fn = (const void*)ggdt_block<BLOCK_CTAS>;
  ok = ok && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BLOCK_SMEM) == cudaSuccess;
  const ImgDesc* descs = reinterpret_cast<const ImgDesc*>(dev + o_desc);
  const CUtensorMap* tmaps = reinterpret_cast<const CUtensorMap*>(dev + o_tm);
  void* args[3] = {(void*)&descs, (void*)&tmaps, (void*)&a};
  ok = ok && cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(BLOCK_WARPS * 32), args, BLOCK_SMEM, nullptr) == cudaSuccess &&
       cudaDeviceSynchronize() == cudaSuccess && cudaMemcpy(&hdr, dev, sizeof(hdr), cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(dev);
  if (!ok) return -5;
  out[0] = hdr.error.v;
  out[1] = hdr.err_info.v;
  out[2] = hdr.progress.v;
  out[3] = blocks;
  return 0;
}

// A wait on a barrier that no copy was issued on; out: its result, STAGE_LOST, error word, its detail.
extern "C" __attribute__((visibility("default"))) int lost_copy(uint32_t* out) {
  uint8_t* dev = nullptr;
  if (cudaMalloc(&dev, sizeof(QueueHdr) + 256) != cudaSuccess) return -4;
  QueueHdr hdr{};
  uint32_t* dout = reinterpret_cast<uint32_t*>(dev + sizeof(QueueHdr));
  bool ok = cudaMemset(dev, 0, sizeof(QueueHdr) + 256) == cudaSuccess;
  wait_for_nothing<<<1, 32>>>(reinterpret_cast<QueueHdr*>(dev), dout);
  ok = ok && cudaDeviceSynchronize() == cudaSuccess && cudaMemcpy(&hdr, dev, sizeof(hdr), cudaMemcpyDeviceToHost) == cudaSuccess &&
       cudaMemcpy(out, dout, 8, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(dev);
  if (!ok) return -5;
  out[2] = hdr.error.v;
  out[3] = hdr.err_info.v;
  return 0;
}
