// dst[N,M] = src[M,N]^T for 1-byte and 4-byte elements, M and N multiples of 128 (HBM-bound: every
// byte is read once and written once, both sides in full 128-byte lines).
//
// Replaces the reference's transpose_matrix__aligned_128<T> (src/base/base.cu:9-155), which the FP8
// path uses to turn checkpoint-layout B[K,N] into the K-contiguous B_transposed[N,K] the GEMM reads
// (examples/005.fp8.mm.cu:2657-2660).  The reference transposes 128x128 (1-byte) / 64x64 (4-byte)
// tiles inside one warp's registers; here a CTA stages a tile in shared memory:
//   * 4-byte: 64x64-word tiles, 1-byte: 128x128-byte tiles; a thread transposes 4x4 blocks in registers
//     (bytes by permutes), stored under an XOR swizzle that keeps both the transposed writes and the row
//     reads free of bank conflicts; global memory sees 16-byte accesses only;
//   * small 4-byte matrices: 32x32-word tiles, padded rows (33 words).
#include "host_common.h"
#include "sm100.cuh"

namespace llmmm {

// 64x64 words per CTA.  A thread transposes a 4x4-word block in registers, so that global and shared memory are only
// touched with 16-byte accesses.  Output row c of the tile lies in T[c] with its 16-byte chunks XOR-swizzled by c / 4: the
// eight lanes of a shared-memory phase write (eight column blocks, one row block) and read (eight chunks of one row)
// eight different bank groups.  HBM-bound: 6430 GB/s at 19456x2560, 62 us, where the kernel below takes 77 to 87 us
// (tiles of 128x64, 64x128 and 32x128 words: 62 to 65 us).
__global__ void __launch_bounds__(256) transpose_b32_kernel(uint32_t* __restrict__ dst, const uint32_t* __restrict__ src, int M, int N)
{
  __shared__ uint4 T[64][16];
  pdl_wait();  // (no pdl_launch_dependents() in the kernels of this file: they write weights, see sm100.cuh)
  const int tx = threadIdx.x % 16;  // 4-column block of the input tile
  const int ry = threadIdx.x / 16;  // 4-row block
  const int m0 = blockIdx.y * 64;
  const int n0 = blockIdx.x * 64;
  uint4     v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = __ldcs(reinterpret_cast<const uint4*>(src + (size_t)(m0 + 4 * ry + i) * N + n0) + tx);
  }
  T[4 * tx + 0][ry ^ tx] = make_uint4(v[0].x, v[1].x, v[2].x, v[3].x);
  T[4 * tx + 1][ry ^ tx] = make_uint4(v[0].y, v[1].y, v[2].y, v[3].y);
  T[4 * tx + 2][ry ^ tx] = make_uint4(v[0].z, v[1].z, v[2].z, v[3].z);
  T[4 * tx + 3][ry ^ tx] = make_uint4(v[0].w, v[1].w, v[2].w, v[3].w);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = ry + 16 * j;  // output row inside the tile = input column; this thread's chunk of it: tx
    __stcs(reinterpret_cast<uint4*>(dst + (size_t)(n0 + c) * M + m0) + tx, T[c][tx ^ (c >> 2)]);
  }
}

// 32x32 words per CTA, one word per access: few words per thread and eight warps per tile, for matrices that do not fill
// the GPU several times over.
__global__ void __launch_bounds__(256) transpose_b32_small_kernel(uint32_t* __restrict__ dst, const uint32_t* __restrict__ src, int M, int N)
{
  __shared__ uint32_t tile[32][33];
  pdl_wait();
  const int tx = threadIdx.x & 31;
  const int ty = threadIdx.x >> 5;
  const int m0 = blockIdx.y * 32;
  const int n0 = blockIdx.x * 32;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int r = ty + 8 * j;
    tile[r][tx] = __ldcs(src + (size_t)(m0 + r) * N + n0 + tx);
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int r = ty + 8 * j;  // output row inside the tile = input column
    __stcs(dst + (size_t)(n0 + r) * M + m0 + tx, tile[tx][r]);
  }
}

// Four rows of four bytes (one word each) to four columns: word q of the result holds byte q of r0..r3.
__device__ __forceinline__ uint4 transpose_4x4_bytes(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3)
{
  const uint32_t a0 = __byte_perm(r0, r1, 0x5140);  // r0.b0 r1.b0 r0.b1 r1.b1
  const uint32_t a1 = __byte_perm(r2, r3, 0x5140);
  const uint32_t a2 = __byte_perm(r0, r1, 0x7362);  // r0.b2 r1.b2 r0.b3 r1.b3
  const uint32_t a3 = __byte_perm(r2, r3, 0x7362);
  return make_uint4(__byte_perm(a0, a1, 0x5410), __byte_perm(a0, a1, 0x7632), __byte_perm(a2, a3, 0x5410), __byte_perm(a2, a3, 0x7632));
}

// 128x128 bytes per CTA.  A thread reads 4 rows x 16 bytes and writes 16 words; word w of output row r (input rows
// 4w..4w+3) lies at T[r][w ^ 4 (r / 16)]: the 32 lanes of a write (eight 16-byte column blocks x four row blocks) touch 32
// banks, and 16-byte chunks stay whole, so that rows leave with 16-byte accesses.
__global__ void __launch_bounds__(256) transpose_b8_kernel(uint8_t* __restrict__ dst, const uint8_t* __restrict__ src, int M, int N)
{
  __shared__ uint4 T[128 * 8];
  pdl_wait();
  const int tx = threadIdx.x & 7;   // 16-byte column block of the input tile
  const int ry = threadIdx.x >> 3;  // 4-row block
  const int m0 = blockIdx.y * 128;
  const int n0 = blockIdx.x * 128;
  uint4     v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = __ldcs(reinterpret_cast<const uint4*>(src + (size_t)(m0 + 4 * ry + i) * N + n0) + tx);
  }
  uint32_t*   t  = reinterpret_cast<uint32_t*>(T) + 16 * tx * 32 + (ry ^ (4 * tx));
  const uint4 t0 = transpose_4x4_bytes(v[0].x, v[1].x, v[2].x, v[3].x);
  const uint4 t1 = transpose_4x4_bytes(v[0].y, v[1].y, v[2].y, v[3].y);
  const uint4 t2 = transpose_4x4_bytes(v[0].z, v[1].z, v[2].z, v[3].z);
  const uint4 t3 = transpose_4x4_bytes(v[0].w, v[1].w, v[2].w, v[3].w);
  const uint32_t w[16] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w, t2.x, t2.y, t2.z, t2.w, t3.x, t3.y, t3.z, t3.w};
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    t[i * 32] = w[i];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int k = threadIdx.x & 7, r = (threadIdx.x >> 3) + 32 * j;  // chunk, output row
    __stcs(reinterpret_cast<uint4*>(dst + (size_t)(n0 + r) * M + m0) + k, T[r * 8 + (k ^ (r >> 4))]);
  }
}

}  // namespace llmmm

extern "C" int llmmm_transpose_aligned_128(void* dst, const void* src, int M, int N, int elem_bytes, llmmm_stream_t stream)
{
  using namespace llmmm;
  if (dst == nullptr || src == nullptr) {
    return set_error(LLMMM_ERR_SHAPE, "null pointer argument");
  }
  if (M < 128 || N < 128 || (M % 128) != 0 || (N % 128) != 0) {
    return set_error(LLMMM_ERR_SHAPE, "M or N can't be divided 128. (got %d %d)", M, N);
  }
  if (elem_bytes != 1 && elem_bytes != 4) {
    return set_error(LLMMM_ERR_UNSUPPORTED, "T is not supported. (element size %d; 1 and 4 bytes are)", elem_bytes);
  }
  if (((uintptr_t)dst | (uintptr_t)src) & 15) {
    return set_error(LLMMM_ERR_SHAPE, "dst and src must be 16-byte aligned");
  }
  const DeviceInfo* device = device_info();
  if (device == nullptr) {
    return LLMMM_ERR_UNSUPPORTED;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (elem_bytes == 4) {
    // Up to about five 64x64-word tiles per SM the small kernel is the faster one (1024x1024: 2.04 against 2.91 us, 2048x1024
    // 3.60 / 4.24, 2560x1024 4.33 / 4.61; 1280x2560 4.89 / 4.83, 2048x2048 5.94 / 5.43).  Its tiles with 16-byte accesses by
    // 64 threads: 2.65 us at 1024x1024, 4.24 at 2048x1024.
    uint32_t*       d = static_cast<uint32_t*>(dst);
    const uint32_t* w = static_cast<const uint32_t*>(src);
    if ((long long)(N / 64) * (M / 64) >= 5 * device->sm_count) {
      LLMMM_CUDA_TRY(launch_pdl(transpose_b32_kernel, dim3(N / 64, M / 64), dim3(256), 0, s, 1, d, w, M, N));
    }
    else {
      LLMMM_CUDA_TRY(launch_pdl(transpose_b32_small_kernel, dim3(N / 32, M / 32), dim3(256), 0, s, 1, d, w, M, N));
    }
  }
  else {
    LLMMM_CUDA_TRY(launch_pdl(transpose_b8_kernel, dim3(N / 128, M / 128), dim3(256), 0, s, 1, static_cast<uint8_t*>(dst),
                              static_cast<const uint8_t*>(src), M, N));
  }
  g_launches.fetch_add(1);
  return LLMMM_OK;
}
