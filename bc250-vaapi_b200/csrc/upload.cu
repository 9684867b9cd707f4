// upload.cu - small and pitched transfers between page-locked host memory and the
// device by kernels that address the host memory directly.
//
// The copy engine moves a frame whose rows lie together on both sides at the
// bus's rate, and then it is what gpu_compute_upload_nv12 uses: the bus bounds
// both (640x480: 15.9 us, this kernel 14.5; 3840x2160: 232 and 248), and the
// engine leaves the SMs to the other streams. With a pitch on either side it takes
// rows one by one, and its time is the rows': 176x144 39 us, 720x576 109,
// 1366x768 159, 2558x1440 320. Warps that read 512 bytes of a row each keep the
// bus full at any pitch: 6.2, 18.6, 39 and 124 us.
#include <cuda.h>

#include <algorithm>

#include "b200enc_internal.h"
#include "common.cuh"

namespace b200enc {

// A warp per 512-byte segment of a row. A lane reads the aligned 16 bytes that
// hold its first byte (never a 16-byte unit without one of the row's bytes, so
// never another page) and takes the next lane's for the rest: 16 bytes of the
// row, stored at once; the row's last unit by bytes.
struct UploadPlane {
  const uint8_t* src;
  uint8_t* dst;
  int src_pitch, dst_pitch, rows;
};
__global__ void __launch_bounds__(128) upload_nv12_kernel(UploadPlane y, UploadPlane uv, int width, int segs) {
  const int lane = threadIdx.x & 31;
  const int total = segs * (y.rows + uv.rows);
  for (int item = blockIdx.x * 4 + (threadIdx.x >> 5); item < total; item += gridDim.x * 4) {
    int row = item / segs;
    const int c = (item - row * segs) * 512 + 16 * lane;
    const bool chroma = row >= y.rows;
    if (chroma) row -= y.rows;
    const UploadPlane& p = chroma ? uv : y;
    const uint8_t* s = p.src + (size_t)row * p.src_pitch + c;
    const int off = (int)(reinterpret_cast<uintptr_t>(s) & 15u), left = width - c;  // bytes of the row from here
    const uint4* a = reinterpret_cast<const uint4*>(s - off);
    uint4 v = make_uint4(0u, 0u, 0u, 0u), n;
    if (left > 0) v = __ldcs(a);
    n.x = __shfl_down_sync(0xffffffffu, v.x, 1);
    n.y = __shfl_down_sync(0xffffffffu, v.y, 1);
    n.z = __shfl_down_sync(0xffffffffu, v.z, 1);
    n.w = __shfl_down_sync(0xffffffffu, v.w, 1);
    if (left <= 0) continue;
    // no next lane with bytes of this row, but bytes in the next unit
    if ((lane == 31 || left <= 16) && min(left, 16) > 16 - off) n = __ldcs(a + 1);
    uint32_t t[8] = {v.x, v.y, v.z, v.w, n.x, n.y, n.z, n.w};
    if (off & 4) {
#pragma unroll
      for (int i = 0; i < 7; ++i) t[i] = t[i + 1];
    }
    if (off & 8) {
#pragma unroll
      for (int i = 0; i < 5; ++i) t[i] = t[i + 2];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = __funnelshift_r(t[i], t[i + 1], (off & 3) * 8);
    uint8_t* d = p.dst + (size_t)row * p.dst_pitch + c;
    if (left >= 16 && (reinterpret_cast<uintptr_t>(d) & 15u) == 0) {
      *reinterpret_cast<uint4*>(d) = make_uint4(t[0], t[1], t[2], t[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < left) d[j] = (uint8_t)(t[j >> 2] >> (8 * (j & 3)));
    }
  }
}

// A frame's motion field and its two status words to page-locked host memory
// (where no entropy coder runs, whose first kernel stores them on its way): three
// copy-engine commands of a few bytes each took 3.3 us apiece.
__global__ void __launch_bounds__(256) stage_mv_kernel(const uint4* __restrict__ mv, uint4* __restrict__ mv_host, int mbs,
                                                       const uint32_t* __restrict__ s0, const uint32_t* __restrict__ s1,
                                                       uint32_t* __restrict__ status_host) {
  pdl_wait();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < mbs) mv_host[i] = mv[i];
  if (i == 0) {
    status_host[0] = *s0;
    status_host[1] = s1 ? *s1 : 0u;  // null: no deblocking pass, no word of its own
  }
}
}  // namespace b200enc

using namespace b200enc;

// What the driver knows of `bytes` bytes of memory from p on. The row kernel reads
// them all, so the whole range has to lie in the object (a cudaHostAlloc, a
// registration) its first byte lies in: a buffer registered in part, or in parts,
// goes to the copy engine. One query per plane, as the type alone took.
HostRange b200enc_host_range(const void* p, size_t bytes) {
  using Fn = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
  static const Fn fn = []() -> Fn {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<Fn>(f);
  }();
  HostRange r{false, nullptr};
  unsigned type = 0, managed = 0;
  CUdeviceptr dev = 0, start = 0;
  size_t size = 0;
  CUpointer_attribute what[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                 CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                 CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void* to[5] = {&type, &managed, &dev, &start, &size};
  if (!fn || fn(5, what, to, reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS) {
    // no driver query, or a thread that has made no runtime call yet
    cudaPointerAttributes a{};
    r.locked = cudaPointerGetAttributes(&a, p) == cudaSuccess && a.type == cudaMemoryTypeHost;
    if (!r.locked) cudaGetLastError();
    return r;
  }
  r.locked = type == CU_MEMORYTYPE_HOST && !managed;
  const size_t off = (size_t)(reinterpret_cast<CUdeviceptr>(p) - start);
  if (r.locked && dev && off <= size && bytes <= size - off) r.dev = reinterpret_cast<const uint8_t*>(dev);
  return r;
}

// Both planes of an NV12 frame, `width` bytes of each row, from page-locked host
// memory at device addresses y, uv. 148 CTAs keep the bus full.
int upload_nv12_launch(const uint8_t* y, int y_pitch, const uint8_t* uv, int uv_pitch, uint8_t* dst_y,
                       uint8_t* dst_uv, int dst_pitch, int width, int height, cudaStream_t st) {
  const int segs = (width + 511) / 512, rows = height + height / 2;
  const UploadPlane py{y, dst_y, y_pitch, dst_pitch, height}, pc{uv, dst_uv, uv_pitch, dst_pitch, height / 2};
  const long long warps = (long long)segs * rows;
  // the launch's own result, as a copy's: an error another call left behind is not this one's
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = (unsigned)std::min<long long>((warps + 3) / 4, 148);
  cfg.blockDim = 128;
  cfg.stream = st;
  return cudaLaunchKernelEx(&cfg, upload_nv12_kernel, py, pc, width, segs) == cudaSuccess ? 0 : -1;
}

int stage_mv_launch(const void* mv, void* mv_host, int mbs, const uint32_t* s0, const uint32_t* s1,
                    uint32_t* status_host, cudaStream_t st) {
  return launch_early(stage_mv_kernel, (mbs + 255) / 256, 256, 0, st, static_cast<const uint4*>(mv),
                      static_cast<uint4*>(mv_host), mbs, s0, s1, status_host) == cudaSuccess ? 0 : -1;
}
