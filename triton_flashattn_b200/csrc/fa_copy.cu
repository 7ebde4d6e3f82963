// Copies between rows of any pitch and address: a bias or mask into the 16-byte aligned rows that the tile kernels read, and
// a bias gradient out of such rows into a dense tensor.
//
// Both sides cannot be aligned at once (a row of 777 elements starts anywhere), so a thread writes 16 aligned bytes and
// puts them together from five aligned words of the source, which its neighbours find in the L1 cache.  What bounds it is
// the memory: read once, written once.  Elementwise copy -> here, us: byte mask of 4 x 1000 x 777 from one row each 9.0 -> 4.9;
// 128 x 1023 x 1023, 16 bit, either way 300 -> 99 (5.4 TB/s), bytes 290 -> 52; 32 x 1001 x 1001, 32 bit 88 -> 50.
#include "fa_common.cuh"
#include "fa_host.cuh"

namespace fa {
namespace {

// 16 bytes from `src` on, of which the first `bytes` exist (the rest reads as zero).  Only aligned words that hold one of
// them are touched.
__device__ __forceinline__ uint4 gather16(const uint8_t* src, int bytes) {
  const uint32_t off = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src)) & 15u;
  if (off == 0 && bytes >= 16) return *reinterpret_cast<const uint4*>(src);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(src) & ~static_cast<uintptr_t>(3));
  const int end = bytes + static_cast<int>(off & 3u);  // bytes from *w on
  uint32_t x[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) x[i] = i * 4 < end && i * 4 < 16 + static_cast<int>(off & 3u) ? w[i] : 0u;
  uint32_t y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    y[i] = __funnelshift_r(x[i], x[i + 1], (off & 3u) * 8);
    const int left = bytes - 4 * i;
    if (left < 4) y[i] = left <= 0 ? 0u : y[i] & ((1u << (8 * left)) - 1u);
  }
  return make_uint4(y[0], y[1], y[2], y[3]);
}

struct RowsParams {
  const uint8_t* src;
  uint8_t* dst;
  int64_t s_sB, s_sH, s_sM, d_sB, d_sH, d_sM;  // bytes
  int H, M, row_bytes, chunks;  // (row_bytes + 16 fits, see row_fits_copy)
};
// Into rows whose starts are multiples of 16 bytes; the last unit of a row is filled up with zeros.
__global__ void __launch_bounds__(256) pad_rows_kernel(const RowsParams p) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  const int m = i / p.chunks, c = i - m * p.chunks;
  if (m >= p.M) return;
  const int b = blockIdx.y / p.H, h = blockIdx.y - b * p.H;
  const uint4 v = gather16(p.src + b * p.s_sB + h * p.s_sH + m * p.s_sM + c * 16, p.row_bytes - c * 16);
  *reinterpret_cast<uint4*>(p.dst + b * p.d_sB + h * p.d_sH + m * p.d_sM + c * 16) = v;
}

struct PackParams {
  const uint8_t* src;
  uint8_t* dst;
  int64_t pitch;  // bytes
  int64_t rows;
  int row_bytes;
};
// Rows of one pitch into a dense tensor at a 16-byte aligned address.
template <typename I>
__global__ void __launch_bounds__(256) pack_rows_kernel(const PackParams p) {
  const I at = (static_cast<I>(blockIdx.x) * 256 + threadIdx.x) * 16;  // byte of the dense tensor
  const I total = static_cast<I>(p.rows) * p.row_bytes;
  if (at >= total) return;
  I row = at / static_cast<I>(p.row_bytes);
  int col = static_cast<int>(at - row * p.row_bytes);
  const uint8_t* src = p.src + static_cast<int64_t>(row) * p.pitch;
  if (col + 16 <= p.row_bytes) {
    *reinterpret_cast<uint4*>(p.dst + at) = gather16(src + col, 16);
    return;
  }
  // across the end of a row (elements are two or four bytes), or of the tensor
  const int count = static_cast<int>(total - at < 16 ? total - at : 16);
  for (int k = 0; k < count; k += 2) {
    *reinterpret_cast<uint16_t*>(p.dst + at + k) = *reinterpret_cast<const uint16_t*>(src + col);
    col += 2;
    if (col >= p.row_bytes) {
      col = 0;
      src += p.pitch;
    }
  }
}

}  // namespace

int launch_pad_rows(void* dst, const int64_t dst_stride[3], const void* src, const int64_t src_stride[3], int eb, int B, int H, int M,
                    int N, cudaStream_t stream) {
  RowsParams p;
  p.src = static_cast<const uint8_t*>(src);
  p.dst = static_cast<uint8_t*>(dst);
  p.s_sB = src_stride[0] * eb, p.s_sH = src_stride[1] * eb, p.s_sM = src_stride[2] * eb;
  p.d_sB = dst_stride[0] * eb, p.d_sH = dst_stride[1] * eb, p.d_sM = dst_stride[2] * eb;
  if (reinterpret_cast<uintptr_t>(dst) % 16 || p.d_sB % 16 || p.d_sH % 16 || p.d_sM % 16) return FA_ERR_ALIGN;
  const int64_t row = static_cast<int64_t>(N) * eb, chunks = (row + 15) / 16;
  if (static_cast<int64_t>(B) * H > 65535 || chunks * M > (1ll << 30)) return FA_ERR_TOO_LARGE;
  p.H = H, p.M = M, p.row_bytes = static_cast<int>(row), p.chunks = static_cast<int>(chunks);
  return launch_ordered(pad_rows_kernel, dim3(static_cast<unsigned>((chunks * M + 255) / 256), B * H), 256, stream, p);
}

int launch_pack_rows(void* dst, const void* src, int64_t pitch, int eb, int64_t rows, int N, cudaStream_t stream) {
  PackParams p = {static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), pitch * eb, rows, N * eb};
  if (reinterpret_cast<uintptr_t>(dst) % 16 || eb % 2) return FA_ERR_ALIGN;
  const int64_t total = rows * N * eb, blocks = (total + 4095) / 4096;
  if (blocks > (1ll << 30)) return FA_ERR_TOO_LARGE;
  const dim3 grid(static_cast<unsigned>(blocks));
  return total < (1ll << 30) ? launch_ordered(pack_rows_kernel<uint32_t>, grid, 256, stream, p)
                             : launch_ordered(pack_rows_kernel<uint64_t>, grid, 256, stream, p);
}

}  // namespace fa
