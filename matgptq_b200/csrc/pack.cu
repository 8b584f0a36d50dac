// Load-time kernels: MSB slicing, weight packing and scale reordering, each with
// a host (CPU) twin that uses the same layout functions.
//
// Replaces matryoshka_slice (src/quant_utils_matgpqt.py:9-17), the single-threaded
// CPU packers swizzle_weights / split_up_n_bits / swizzle_matgptq
// (csrc/utils.cpp:22-217) behind pack_matgptq_qweights (csrc/bindings.cpp:43-84)
// and reorder_matgptq_scales (csrc/bindings.cpp:86-142).  The reference copies the
// codes to the host, packs on one thread and copies back; here slicing and
// packing are one pass over the codes on the GPU.
#include <cuda_runtime.h>

#include <cstring>

#include "kernels.h"
#include "layout.cuh"

namespace mg {

// ---------------------------------------------------------------------------
// slicing
// ---------------------------------------------------------------------------
__global__ void slice_kernel(const uint8_t *__restrict__ in, uint8_t *__restrict__ out, long long numel,
                             int master_bitwidth, int bitwidth) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long nvec = numel / 16;
  const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (aligned) {
    for (long long v = tid; v < nvec; v += stride) {
      uint4 q = reinterpret_cast<const uint4 *>(in)[v];
      uint32_t *words = reinterpret_cast<uint32_t *>(&q);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t o = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) o |= matryoshka_slice((words[i] >> (8 * e)) & 0xFFu, master_bitwidth, bitwidth) << (8 * e);
        words[i] = o;
      }
      reinterpret_cast<uint4 *>(out)[v] = q;
    }
    for (long long i = nvec * 16 + tid; i < numel; i += stride) out[i] = static_cast<uint8_t>(matryoshka_slice(in[i], master_bitwidth, bitwidth));
  } else {
    for (long long i = tid; i < numel; i += stride) out[i] = static_cast<uint8_t>(matryoshka_slice(in[i], master_bitwidth, bitwidth));
  }
}

int slice_launch(const uint8_t *in, uint8_t *out, long long numel, int master_bitwidth, int bitwidth,
                 cudaStream_t stream) {
  if (numel == 0) return MG_OK;
  const int threads = 256;
  long long blocks = (numel / 16 + threads - 1) / threads;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 16) blocks = 148 * 16;
  slice_kernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(in, out, numel, master_bitwidth, bitwidth);
  return cudaGetLastError() == cudaSuccess ? MG_OK : MG_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// packing: one thread builds the 2*b words that one lane will later decode (pack_lane on the host)
// ---------------------------------------------------------------------------
template <int B>
static void pack_lane(const uint8_t *codes, int K, int tile, int kb, int lane, int slice_from_master,
                     uint32_t (&w)[2 * B]) {
  for (int j = 0; j < 2 * B; ++j) w[j] = 0u;
  const int g = lane >> 2, t = lane & 3;
  for (int i = 0; i < 8; ++i) {
    for (int rr = 0; rr < 2; ++rr) {
      const int row = tile * 16 + g + 8 * rr;
      const int col = kb * 128 + 32 * (i >> 1) + 8 * t + 4 * (i & 1);
      const uint8_t *src = codes + static_cast<size_t>(row) * K + col;
      for (int e = 0; e < 4; ++e) {
        uint32_t c = src[e];
        if (slice_from_master > 0) c = matryoshka_slice(c, slice_from_master, B);
        c &= (1u << B) - 1u;
        place_code<B>(w, 4 * i + 2 * (e >> 1) + rr, e & 1, c);
      }
    }
  }
}

// Four codes at once: mask to B bits, or slice from the master (matryoshka_slice() on every byte of the word).  The
// rounded value is at most 2^B, which fits the byte for B < 8, so no carry crosses a byte.
template <int B> __device__ __forceinline__ uint32_t slice4(uint32_t x, int slice_from_master) {
  constexpr uint32_t kOnes = 0x01010101u, kMask = ((1u << B) - 1u) * kOnes;
  if (slice_from_master == 0) return x & kMask;
  if constexpr (B == 8) {
    return x;
  } else {
    uint32_t v = (x >> (8 - B)) & kMask;
    if (slice_from_master != B) {
      v += (x >> (7 - B)) & kOnes;  // the rounding bit
      v -= (v >> B) & kOnes;        // saturate: 2^B becomes 2^B - 1
    }
    return v;
  }
}

// One warp packs one block of 16 x 128 codes, as it will later be decoded: a lane reads 8 consecutive codes of rows g
// and g+8 in each of four 32-wide chunks (8-byte loads that fill whole 32-byte sectors), slices four bytes per
// instruction, spreads two codes over the halves of a word with one PRMT, and writes its words as 16-byte vectors.
// Bound by HBM (one byte in, B/8 out per code).  The byte-wise form it replaces needed 64 one-byte loads and 64
// scalar slices a lane: 14336 x 4096 from 8 to 3 bits: 61.4 -> 18.4 us on B200 (80.7 MB, 4.4 TB/s; a copy of as many
// bytes at the measured peak takes 12.5 us).
template <int B>
__global__ void __launch_bounds__(256) pack_kernel(const uint8_t *__restrict__ codes, uint32_t *__restrict__ packed, int tiles,
                                                   int kblocks, int K, int slice_from_master) {
  const long long gid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long nblocks = static_cast<long long>(tiles) * kblocks;
  const long long blk = gid >> 5;
  const int lane = static_cast<int>(gid & 31);
  if (blk >= nblocks) return;
  const int tile = static_cast<int>(blk / kblocks), kb = static_cast<int>(blk - static_cast<long long>(tile) * kblocks);
  const int g = lane >> 2, t = lane & 3;
  const uint8_t *src = codes + (static_cast<size_t>(tile) * 16 + g) * K + kb * 128 + 8 * t;
  uint32_t c[2][8];  // [row g, g+8][k-step]: four consecutive codes
  if ((reinterpret_cast<uintptr_t>(codes) & 7u) == 0) {
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const uint2 q = *reinterpret_cast<const uint2 *>(src + static_cast<size_t>(8 * rr) * K + 32 * jj);
        c[rr][2 * jj] = q.x;
        c[rr][2 * jj + 1] = q.y;
      }
  } else {  // a caller's buffer may start anywhere
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const uint8_t *p = src + static_cast<size_t>(8 * rr) * K + 32 * (i >> 1) + 4 * (i & 1);
        c[rr][i] = p[0] | (static_cast<uint32_t>(p[1]) << 8) | (static_cast<uint32_t>(p[2]) << 16) | (static_cast<uint32_t>(p[3]) << 24);
      }
  }
  uint32_t w[2 * B];
#pragma unroll
  for (int j = 0; j < 2 * B; ++j) w[j] = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const uint32_t v = slice4<B>(c[rr][i], slice_from_master);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t pair = __byte_perm(v, 0u, e ? 0x4342 : 0x4140);  // codes 2e and 2e+1 in the low and high half
        Piece pc[3];
        const int n = code_pieces<B>(4 * i + 2 * e + rr, 0, pc);
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (k < n) w[pc[k].word] |= ((pair >> pc[k].cshift) & (((1u << pc[k].nbits) - 1u) * 0x00010001u)) << pc[k].off;
      }
    }
  uint32_t *dst = packed + blk * BlockTraits<B>::WORDS;
  if ((reinterpret_cast<uintptr_t>(packed) & 15u) != 0) {
#pragma unroll
    for (int j = 0; j < 2 * B; ++j) dst[word_slot<B>(lane, j)] = w[j];
    return;
  }
#pragma unroll
  for (int v = 0; v < BlockTraits<B>::NV; ++v)
    *reinterpret_cast<uint4 *>(dst + v * 128 + lane * 4) = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
  if constexpr (BlockTraits<B>::TAIL == 2)
    *reinterpret_cast<uint2 *>(dst + BlockTraits<B>::NV * 128 + lane * 2) =
        make_uint2(w[4 * BlockTraits<B>::NV], w[4 * BlockTraits<B>::NV + 1]);
}

template <int B>
static int pack_launch_b(const uint8_t *codes, uint32_t *packed, int N, int K, int slice_from_master,
                         cudaStream_t stream) {
  const int tiles = N / 16, kblocks = K / 128;
  const long long threads_total = static_cast<long long>(tiles) * kblocks * 32;
  if (threads_total == 0) return MG_OK;
  const int threads = 256;
  const long long blocks = (threads_total + threads - 1) / threads;
  pack_kernel<B><<<static_cast<unsigned>(blocks), threads, 0, stream>>>(codes, packed, tiles, kblocks, K, slice_from_master);
  return cudaGetLastError() == cudaSuccess ? MG_OK : MG_ERR_CUDA;
}

int pack_launch(const uint8_t *codes, uint32_t *packed, int N, int K, int bitwidth, int slice_from_master,
                cudaStream_t stream) {
  switch (bitwidth) {
    case 2: return pack_launch_b<2>(codes, packed, N, K, slice_from_master, stream);
    case 3: return pack_launch_b<3>(codes, packed, N, K, slice_from_master, stream);
    case 4: return pack_launch_b<4>(codes, packed, N, K, slice_from_master, stream);
    case 6: return pack_launch_b<6>(codes, packed, N, K, slice_from_master, stream);
    case 8: return pack_launch_b<8>(codes, packed, N, K, slice_from_master, stream);
    default: return MG_ERR_BAD_ARG;
  }
}

template <int B> static void pack_host_b(const uint8_t *codes, uint32_t *packed, int N, int K, int slice_from_master) {
  const int tiles = N / 16, kblocks = K / 128;
  for (int tile = 0; tile < tiles; ++tile)
    for (int kb = 0; kb < kblocks; ++kb) {
      uint32_t *dst = packed + (static_cast<size_t>(tile) * kblocks + kb) * BlockTraits<B>::WORDS;
      for (int lane = 0; lane < 32; ++lane) {
        uint32_t w[2 * B];
        pack_lane<B>(codes, K, tile, kb, lane, slice_from_master, w);
        for (int j = 0; j < 2 * B; ++j) dst[word_slot<B>(lane, j)] = w[j];
      }
    }
}

int pack_host(const uint8_t *codes, uint32_t *packed, int N, int K, int bitwidth, int slice_from_master) {
  switch (bitwidth) {
    case 2: pack_host_b<2>(codes, packed, N, K, slice_from_master); return MG_OK;
    case 3: pack_host_b<3>(codes, packed, N, K, slice_from_master); return MG_OK;
    case 4: pack_host_b<4>(codes, packed, N, K, slice_from_master); return MG_OK;
    case 6: pack_host_b<6>(codes, packed, N, K, slice_from_master); return MG_OK;
    case 8: pack_host_b<8>(codes, packed, N, K, slice_from_master); return MG_OK;
    default: return MG_ERR_BAD_ARG;
  }
}

template <int B> static void unpack_host_b(const uint32_t *packed, uint8_t *codes, int N, int K) {
  const int tiles = N / 16, kblocks = K / 128;
  for (int tile = 0; tile < tiles; ++tile)
    for (int kb = 0; kb < kblocks; ++kb) {
      const uint32_t *src = packed + (static_cast<size_t>(tile) * kblocks + kb) * BlockTraits<B>::WORDS;
      for (int lane = 0; lane < 32; ++lane) {
        uint32_t w[2 * B];
        for (int j = 0; j < 2 * B; ++j) w[j] = src[word_slot<B>(lane, j)];
        for (int P = 0; P < kPairs; ++P)
          for (int h = 0; h < 2; ++h) {
            int row, col;
            pair_coord(lane, P, h, row, col);
            codes[static_cast<size_t>(tile * 16 + row) * K + kb * 128 + col] = static_cast<uint8_t>(extract_code<B>(w, P, h));
          }
      }
    }
}

int unpack_host(const uint32_t *packed, uint8_t *codes, int N, int K, int bitwidth) {
  switch (bitwidth) {
    case 2: unpack_host_b<2>(packed, codes, N, K); return MG_OK;
    case 3: unpack_host_b<3>(packed, codes, N, K); return MG_OK;
    case 4: unpack_host_b<4>(packed, codes, N, K); return MG_OK;
    case 6: unpack_host_b<6>(packed, codes, N, K); return MG_OK;
    case 8: unpack_host_b<8>(packed, codes, N, K); return MG_OK;
    default: return MG_ERR_BAD_ARG;
  }
}

// ---------------------------------------------------------------------------
// scales: [N, G] -> [N/16, G, 16] so that the 16 scales a warp needs for one
// block are one 32-byte sector (same order as csrc/bindings.cpp:113-119)
// ---------------------------------------------------------------------------
__global__ void reorder_scales_kernel(const uint16_t *__restrict__ in, uint16_t *__restrict__ out, int N, int G) {
  const long long total = static_cast<long long>(N) * G;
  for (long long o = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; o < total;
       o += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(o & 15);
    const long long tg = o >> 4;
    const int grp = static_cast<int>(tg % G);
    const long long tile = tg / G;
    out[o] = in[(tile * 16 + r) * G + grp];
  }
}

int reorder_scales_launch(const uint16_t *in, uint16_t *out, int N, int K, int group_size, cudaStream_t stream) {
  const int G = group_size == -1 ? 1 : K / group_size;
  const long long total = static_cast<long long>(N) * G;
  if (total == 0) return MG_OK;
  if (G == 1) {
    return cudaMemcpyAsync(out, in, total * 2, cudaMemcpyDeviceToDevice, stream) == cudaSuccess ? MG_OK : MG_ERR_CUDA;
  }
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  reorder_scales_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(in, out, N, G);
  return cudaGetLastError() == cudaSuccess ? MG_OK : MG_ERR_CUDA;
}

int reorder_scales_host(const uint16_t *in, uint16_t *out, int N, int K, int group_size) {
  const int G = group_size == -1 ? 1 : K / group_size;
  for (long long tile = 0; tile < N / 16; ++tile)
    for (int grp = 0; grp < G; ++grp)
      for (int r = 0; r < 16; ++r) out[(tile * G + grp) * 16 + r] = in[(tile * 16 + r) * G + grp];
  return MG_OK;
}

}  // namespace mg
