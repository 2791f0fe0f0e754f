// Weight container management for the W4A16 path: allocation, the load-time
// repack from the checkpoint's on-disk layout into the private block layout, and
// the row dequantiser that anchors bit-exactness on the GPU.
//
// Replaces awq_alloc_fused / awq_repack_into / awq_free
// (src/kernels/gemv_w4a16.cu:308-334 of the reference project) and
// w4a16_dequant_rows (src/kernels/gemm_w4a16.cu:15-38,56-61).
#include <cstring>
#include <atomic>
#include <climits>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace w4a16 {

// ------------------------------------------------------------------ errors
static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
}

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
  return code;
}

// ------------------------------------------------------------------ device info
constexpr int kMaxDevices = 64;
static DeviceInfo g_dev[kMaxDevices];
static std::mutex g_dev_mu;
static std::atomic<bool> g_dev_ready[kMaxDevices];  // g_dev[i] is filled in and does not change any more
static std::mutex g_ww_mu;
// Streams with a weight write that no executed matmul call has followed yet, and the last capture in which a call has.
struct WeightWrite {
  cudaStream_t stream;
  unsigned long long followed_in;
};
static std::vector<WeightWrite> g_ww;
static std::atomic<int> g_ww_count{0};

__device__ int g_status_word = 0;

const DeviceInfo* device_info() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    set_error("no current CUDA device");
    return nullptr;
  }
  DeviceInfo& d = g_dev[dev];
  if (g_dev_ready[dev].load(std::memory_order_acquire)) return &d;
  std::lock_guard<std::mutex> lk(g_dev_mu);
  if (d.device != dev) {
    int sms = 0, smem = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
      set_error("cudaDeviceGetAttribute failed");
      return nullptr;
    }
    int* st = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&st), g_status_word) != cudaSuccess) {
      set_error("cudaGetSymbolAddress(status word) failed");
      return nullptr;
    }
    d.sms = sms;
    d.smem_optin = smem;
    d.status = st;
    d.device = dev;
    g_dev_ready[dev].store(true, std::memory_order_release);
  }
  return &d;
}

// ------------------------------------------------------------------ kernels
namespace {

// Physical row of logical row o: the identity, or - for a gate|up layer repacked for the fused SwiGLU epilogue
// (inter > 0) - gate row o at 2 o and up row o - inter at 2 (o - inter) + 1.
__device__ __forceinline__ int physical_row(int o, int inter) {
  return inter <= 0 ? o : (o < inter ? 2 * o : 2 * (o - inter) + 1);
}

// Packed word on disk (k-offset c at nibble c) -> stream word (k-offset c at nibble nib_pos(c)): the even nibbles
// close up into the low half, the odd ones into the high half.
__device__ __forceinline__ uint32_t stream_word(uint32_t w) {
  uint32_t e = w & 0x0F0F0F0Fu, o = (w >> 4) & 0x0F0F0F0Fu;
  e |= e >> 4;
  o |= o >> 4;
  return __byte_perm(e, o, 0x6420);
}

// Checkpoint tensors -> stream. A CTA takes 128 source rows x kRepackGroups k groups: a warp loads 8 rows x 64
// bytes (two whole sectors of each row) and stores 128 contiguous bytes of each of the group's four chunks; the eight
// groups of a row are in flight together. Scales and zero points go along in the same launch, their stores
// contiguous over the rows. Bound by HBM. One thread per 16 bytes with consecutive threads on consecutive ROWS,
// and a second kernel with consecutive threads on consecutive groups (2-byte stores 8576 bytes apart), took
// 72.3 us for 34816 x 5120; this takes 35.4 us (92.6 MB in, 93.3 MB out: 5.25 TB/s).
constexpr int kRepackGroups = 8, kRepackThreads = 256;
__global__ void __launch_bounds__(kRepackThreads) k_repack(uint8_t* __restrict__ dst, const uint32_t* __restrict__ sq,
                                                           const uint16_t* __restrict__ ss, const uint32_t* __restrict__ sz,
                                                           int out_f, int G, int row_offset, int inter) {
  const int gblocks = (G + kRepackGroups - 1) / kRepackGroups;
  const int so0 = static_cast<int>(blockIdx.x / gblocks) * kTileRows, g0 = static_cast<int>(blockIdx.x % gblocks) * kRepackGroups;
  const int ng = min(kRepackGroups, G - g0);
  const int c = threadIdx.x & 3;
#pragma unroll
  for (int pass = 0; pass < kTileRows / (kRepackThreads / 4); ++pass) {
    const int so = so0 + pass * (kRepackThreads / 4) + static_cast<int>(threadIdx.x >> 2);
    if (so >= out_f) continue;
    const uint4* src = reinterpret_cast<const uint4*>(sq) + (static_cast<size_t>(so) * G + g0) * 4 + c;
    uint4 v[kRepackGroups];
#pragma unroll
    for (int j = 0; j < kRepackGroups; ++j)
      if (j < ng) v[j] = __ldcs(src + 4 * j);
    const int o = physical_row(so + row_offset, inter);
    uint8_t* d = dst + tile_group_offset(o, g0, G) + c * kChunkBytes + weight_slot(o % kTileRows, c) * 16;
#pragma unroll
    for (int j = 0; j < kRepackGroups; ++j)
      if (j < ng)
        *reinterpret_cast<uint4*>(d + static_cast<size_t>(j) * kTileGroupBytes) =
            make_uint4(stream_word(v[j].x), stream_word(v[j].y), stream_word(v[j].z), stream_word(v[j].w));
  }
  const int so = so0 + static_cast<int>(threadIdx.x % kTileRows);
  if (so >= out_f) return;
  const int o = physical_row(so + row_offset, inter), r = o % kTileRows;
  for (int j = threadIdx.x / kTileRows; j < ng; j += kRepackThreads / kTileRows) {
    uint8_t* blk = dst + tile_group_offset(o, g0 + j, G);
    reinterpret_cast<uint16_t*>(blk + kTgScaleOff)[r] = ss[static_cast<size_t>(so) * G + g0 + j];
    const uint32_t zw = sz[static_cast<size_t>(so >> 3) * G + g0 + j];
    blk[kTgZpOff + r] = static_cast<uint8_t>((zw >> ((so & 7) * 4)) & 0xFu);
  }
}

// Stream -> bf16 rows. A warp takes 16 rows of one k group, two rows at a time: a lane expands ONE packed word (8 k),
// so that sixteen lanes store a row's 256 contiguous bytes and the loads are the two rows' neighbouring slots.
// (128 + q) - (128 + zp) is exact in bf16 and the product is rounded once, so this is bf16(float(q - zp) *
// float(s)) for every scale. Bound by HBM writes. One thread per 64 bytes of output (four 16-byte stores, 64
// bytes apart across the warp) took 117.5 us for 34816 x 5120; this takes 77.2 us (93.3 MB in, 356.5 MB out: 5.83 TB/s).
constexpr int kDequantRows = 16;
__global__ void __launch_bounds__(256) k_dequant_rows(uint16_t* __restrict__ dst, const uint8_t* __restrict__ stream, int row0,
                                                      int nrows, int K, int G) {
  const int lane = threadIdx.x & 31, c = (lane >> 2) & 3, i = lane & 3;
  const long long item = blockIdx.x * 8LL + (threadIdx.x >> 5);
  const int g = static_cast<int>(item % G);
  const long long first = item / G * kDequantRows + (lane >> 4);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t w[4], sc[4], zp[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long r = first + 8 * h + 2 * j;
      if (r < nrows) {
        const int o = row0 + static_cast<int>(r), ro = o % kTileRows;
        const uint8_t* blk = stream + tile_group_offset(o, g, G);
        w[j] = *reinterpret_cast<const uint32_t*>(blk + c * kChunkBytes + weight_slot(ro, c) * 16 + i * 4);
        sc[j] = reinterpret_cast<const uint16_t*>(blk + kTgScaleOff)[ro];
        zp[j] = blk[kTgZpOff + ro];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long r = first + 8 * h + 2 * j;
      if (r < nrows) {
        const uint32_t spair = sc[j] | (sc[j] << 16), zpair = __byte_perm(zp[j], 0x43434343u, 0x4040);
        uint32_t v[4];
#pragma unroll
        for (int p = 0; p < 4; ++p)
          v[p] = mul_bf16x2(sub_bf16x2(((w[j] >> (4 * p)) & 0x000F000Fu) | 0x43004300u, zpair), spair);
        reinterpret_cast<uint4*>(dst + r * K + static_cast<size_t>(g) * kGroup)[lane & 15] = make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
  }
}

// A wait that nothing satisfies: the same bounded mbarrier wait the kernels use, on a barrier nobody
// arrives at. It gives up after `polls` tests, reports through the status word and the kernel returns.
__global__ void k_wait_timeout_selftest(int* status, uint32_t polls) {
  __shared__ uint64_t bar;
  const uint32_t bar_a = smem_u32(&bar);
  if (threadIdx.x == 0) {
    mbar_init(bar_a, 1);
    fence_mbar_init();
    if (!mbar_wait_bounded(bar_a, 0, polls)) atomicExch(status, W4A16_ETIMEOUT);
  }
}

}  // namespace

// The capture that the stream's calls go to, or 0: they are executed. (An error says that the legacy stream cannot be used while
// another one is captured; the launch that follows reports it and the note comes back.)
static unsigned long long capture_of(cudaStream_t st) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(st, &status, &id) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return status == cudaStreamCaptureStatusNone ? 0 : id;
}

void note_weight_write(cudaStream_t st) {
  std::lock_guard<std::mutex> lk(g_ww_mu);
  for (WeightWrite& w : g_ww)
    if (w.stream == st) {
      w.followed_in = 0;
      return;
    }
  g_ww.push_back({st, 0});
  g_ww_count.store(static_cast<int>(g_ww.size()), std::memory_order_release);
}
bool take_weight_write(cudaStream_t st) {
  if (g_ww_count.load(std::memory_order_relaxed) == 0) return false;
  std::lock_guard<std::mutex> lk(g_ww_mu);
  for (size_t i = 0; i < g_ww.size(); ++i)
    if (g_ww[i].stream == st) {
      if (const unsigned long long capture = capture_of(st)) {
        const bool first = g_ww[i].followed_in != capture;
        g_ww[i].followed_in = capture;
        return first;
      }
      g_ww.erase(g_ww.begin() + static_cast<long>(i));
      g_ww_count.store(static_cast<int>(g_ww.size()), std::memory_order_release);
      return true;
    }
  return false;
}

int check_weights(const w4a16_weights_t* w) {
  W4_REQUIRE(w != nullptr, "weights: null struct");
  W4_REQUIRE(w->qweight && w->scale && w->zp, "weights: null buffer");
  W4_REQUIRE(w->group_size == kGroup, "weights: group_size %d unsupported (only 128)", w->group_size);
  W4_REQUIRE(w->out_f > 0 && w->out_f % kRowGranule == 0, "weights: out_f %d not a positive multiple of 16",
             w->out_f);
  W4_REQUIRE(w->in_f > 0 && w->in_f % kGroup == 0, "weights: in_f %d not a positive multiple of 128",
             w->in_f);
  W4_REQUIRE(w->num_groups == w->in_f / kGroup, "weights: num_groups %d != in_f/128", w->num_groups);
  W4_REQUIRE((reinterpret_cast<uintptr_t>(w->qweight) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(w->scale) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(w->zp) & 15) == 0,
             "weights: buffers must be 16-byte aligned");
  return W4A16_OK;
}

}  // namespace w4a16

using namespace w4a16;

extern "C" {

const char* w4a16_last_error(void) { return g_err; }

int w4a16_device_status(void) {
  int v = 0;
  W4_CUDA(cudaDeviceSynchronize());
  W4_CUDA(cudaMemcpyFromSymbol(&v, g_status_word, sizeof(int)));
  if (v != 0) set_error("device status %d: a bounded device-side wait expired", v);
  return v;
}

int w4a16_device_status_clear(void) {
  const int zero = 0;
  W4_CUDA(cudaDeviceSynchronize());
  W4_CUDA(cudaMemcpyToSymbol(g_status_word, &zero, sizeof(int)));
  return W4A16_OK;
}

int w4a16_selftest_wait_timeout(int polls, void* stream) {
  W4_REQUIRE(polls >= 1 && polls <= 4096, "selftest_wait_timeout: polls = %d outside [1,4096]", polls);
  const DeviceInfo* di = device_info();
  if (!di) return W4A16_ECUDA;
  k_wait_timeout_selftest<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(di->status, static_cast<uint32_t>(polls));
  W4_CUDA(cudaGetLastError());
  return W4A16_OK;
}

int w4a16_weights_alloc(w4a16_weights_t* w, int out_f, int in_f, int group_size, void* stream) {
  W4_REQUIRE(w != nullptr, "weights_alloc: null struct");
  W4_REQUIRE(group_size == kGroup, "weights_alloc: group_size %d unsupported (only 128)", group_size);
  W4_REQUIRE(out_f > 0 && out_f % kRowGranule == 0, "weights_alloc: out_f %d not a positive multiple of 16",
             out_f);
  W4_REQUIRE(in_f > 0 && in_f % kGroup == 0, "weights_alloc: in_f %d not a positive multiple of 128", in_f);
  memset(w, 0, sizeof *w);
  const int G = in_f / group_size;
  // The whole weight stream (int4 blocks with their scales and zero points interleaved per
  // 128-row x 128-k block) lives behind `qweight`; for out_f a multiple of 128 its size is exactly
  // the reference's total_bytes() = int4 + bf16 scales + one-byte zero points. `scale` and `zp` stay valid,
  // independently freeable allocations because the reference's callers cudaFree all three
  // pointers one by one (src/model/model.cu:111,204), but nothing is read through them.
  const size_t qb = stream_bytes(out_f, G);  // out_f rounded up to whole 128-row tiles
  const size_t sb = 256;
  const size_t zb = 256;
  void *q = nullptr, *s = nullptr, *z = nullptr;
  cudaError_t e = cudaMalloc(&q, qb);
  if (e == cudaSuccess) e = cudaMalloc(&s, sb);
  if (e == cudaSuccess) e = cudaMalloc(&z, zb);
  if (e != cudaSuccess) {
    cudaFree(q);
    cudaFree(s);
    cudaFree(z);
    return fail(W4A16_ECUDA, "weights_alloc(%d x %d): %s", out_f, in_f, cudaGetErrorString(e));
  }
  if (out_f % kTileRows != 0) {
    // rows of the last tile past out_f: zero scales, so they contribute nothing and are never stored.
    // On the caller's stream, so that it is ordered before the repack that follows on that stream.
    e = cudaMemsetAsync(q, 0, qb, static_cast<cudaStream_t>(stream));
    note_weight_write(static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) {
      cudaFree(q);
      cudaFree(s);
      cudaFree(z);
      return fail(W4A16_ECUDA, "weights_alloc: %s", cudaGetErrorString(e));
    }
  }
  w->qweight = static_cast<uint32_t*>(q);
  w->scale = static_cast<uint16_t*>(s);
  w->zp = static_cast<uint8_t*>(z);
  w->out_f = out_f;
  w->in_f = in_f;
  w->group_size = group_size;
  w->num_groups = G;
  return W4A16_OK;
}

static int repack_rows(const w4a16_weights_t* w, int dst_row_offset, const uint32_t* packed, const uint16_t* scale,
                       const uint32_t* zp, int out_f, int inter, void* stream) {
  if (int rc = check_weights(w)) return rc;
  W4_REQUIRE(packed && scale && zp, "repack_into: null source tensor");
  W4_REQUIRE(out_f > 0 && out_f % kRowGranule == 0, "repack_into: out_f %d not a positive multiple of 16",
             out_f);
  W4_REQUIRE(dst_row_offset >= 0 && dst_row_offset % kRowGranule == 0,
             "repack_into: row offset %d not a multiple of 16", dst_row_offset);
  W4_REQUIRE(dst_row_offset + out_f <= w->out_f, "repack_into: rows [%d,%d) exceed out_f %d",
             dst_row_offset, dst_row_offset + out_f, w->out_f);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* stream_base = reinterpret_cast<uint8_t*>(w->qweight);
  const long long blocks = static_cast<long long>((out_f + kTileRows - 1) / kTileRows) * ((w->num_groups + kRepackGroups - 1) / kRepackGroups);
  W4_REQUIRE(blocks <= INT_MAX, "repack_into: %d x %d is too large", out_f, w->in_f);
  k_repack<<<static_cast<unsigned>(blocks), kRepackThreads, 0, st>>>(stream_base, packed, scale, zp, out_f, w->num_groups,
                                                                     dst_row_offset, inter);
  W4_CUDA(cudaGetLastError());
  note_weight_write(st);
  return W4A16_OK;
}

int w4a16_repack_into(const w4a16_weights_t* w, int dst_row_offset, const uint32_t* packed,
                      const uint16_t* scale, const uint32_t* zp, int out_f, void* stream) {
  return repack_rows(w, dst_row_offset, packed, scale, zp, out_f, 0, stream);
}

int w4a16_repack_into_swiglu(const w4a16_weights_t* w, int dst_row_offset, const uint32_t* packed,
                             const uint16_t* scale, const uint32_t* zp, int out_f, int inter, void* stream) {
  W4_REQUIRE(w != nullptr && inter > 0 && 2 * inter == w->out_f,
             "repack_into_swiglu: inter = %d must be half of the container's rows", inter);
  return repack_rows(w, dst_row_offset, packed, scale, zp, out_f, inter, stream);
}

int w4a16_weights_free(w4a16_weights_t* w) {
  W4_REQUIRE(w != nullptr, "weights_free: null struct");
  cudaFree(w->qweight);
  cudaFree(w->scale);
  cudaFree(w->zp);
  memset(w, 0, sizeof *w);
  return W4A16_OK;
}

int w4a16_dequant_rows(uint16_t* dst, const w4a16_weights_t* w, int row0, int nrows, void* stream) {
  if (int rc = check_weights(w)) return rc;
  W4_REQUIRE(dst != nullptr && (reinterpret_cast<uintptr_t>(dst) & 15) == 0,
             "dequant_rows: dst null or not 16-byte aligned");
  W4_REQUIRE(row0 >= 0 && nrows >= 0 && row0 + nrows <= w->out_f, "dequant_rows: rows [%d,%d) outside [0,%d)",
             row0, row0 + nrows, w->out_f);
  if (nrows == 0) return W4A16_OK;
  const long long warps = static_cast<long long>((nrows + kDequantRows - 1) / kDequantRows) * w->num_groups;
  W4_REQUIRE((warps + 7) / 8 <= INT_MAX, "dequant_rows: %d x %d is too large", nrows, w->in_f);
  k_dequant_rows<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      dst, reinterpret_cast<const uint8_t*>(w->qweight), row0, nrows, w->in_f, w->num_groups);
  W4_CUDA(cudaGetLastError());
  return W4A16_OK;
}

}  // extern "C"
