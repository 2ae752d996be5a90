// GPTQ / AWQ -> Marlin tile layout repacking.
//
// GPTQ and 8-bit AWQ sources in checkpoint row order, for 16-bit activations, take RepackWarpKernel: a warp turns
// 64 columns by 16 k at a time in registers.  4-bit AWQ sources, 8-bit-activation layouts and activation-order
// checkpoints (each output word then gathers from arbitrary rows) take RepackKernel: one thread block owns a strip
// of TK quantised rows (16, or 32 for the 8-bit-activation layouts) by up to 256 columns.  It first expands that
// strip from the source packing into an unpacked byte tile in shared memory with coalesced word loads, then every
// thread assembles four consecutive output words from the tile and writes them with one 16-byte
// store.  The strip maps to one contiguous range of the output, so global traffic is one
// coalesced read and one coalesced write of the weights.
#include "common.cuh"

namespace iob {
namespace {

constexpr int kTileN = 256;
constexpr int kThreads = 256;

enum class Source { kGptq, kGptqPerm, kAwq };

// Which (k, n) of a 1024-element chunk sits in bit-field `field` of chunk word `inner`.
// 16-bit activations: chunk = 16 k x 64 n; 8-bit activations: chunk = 32 k x 32 n.
template <int kBits, bool kA8>
__device__ __forceinline__ void ChunkSource(int inner, int field, int& k, int& n) {
  if constexpr (!kA8 && kBits == 4) {
    const int lane = inner >> 2, sub = inner & 3;
    k = 2 * (lane & 3) + (field >> 2) + 8 * (field & 1);
    n = (lane >> 2) + 8 * ((field >> 1) & 1) + 16 * sub;
  } else if constexpr (!kA8 && kBits == 8) {
    const int lane = inner >> 3, sub = (inner >> 1) & 3, half = inner & 1;
    k = 2 * (lane & 3) + (field >> 1) + 8 * (field & 1);
    n = (lane >> 2) + 8 * half + 16 * sub;
  } else if constexpr (kA8 && kBits == 4) {
    const int lane = inner >> 2, sub = (inner >> 1) & 1, half = inner & 1;
    k = 4 * (lane & 3) + (field >> 1) + 16 * (field & 1);
    n = (lane >> 2) + 8 * half + 16 * sub;
  } else {
    const int lane = inner >> 3, sub = (inner >> 2) & 1, q = inner & 3;
    k = 4 * (lane & 3) + field + 16 * (q & 1);
    n = (lane >> 2) + 8 * (q >> 1) + 16 * sub;
  }
}

template <int kBits, bool kA8, Source kSource>
__global__ void __launch_bounds__(kThreads)
RepackKernel(const uint32_t* __restrict__ in, const int32_t* __restrict__ perm,
             uint32_t* __restrict__ out, int size_k, int size_n) {
  constexpr int kPf = 32 / kBits;
  constexpr int kTileK = kA8 ? 32 : 16;
  constexpr int kChunkN = kA8 ? 32 : 64;
  constexpr int kWordsPerChunk = 1024 / kPf;
  constexpr uint32_t kMask = (1u << kBits) - 1u;
  constexpr int kPitch = kTileN + 4;
  __shared__ __align__(16) uint8_t tile[kTileK][kPitch];

  const int n0 = blockIdx.x * kTileN;
  const int k0 = blockIdx.y * kTileK;
  const int tn = min(kTileN, size_n - n0);

  if constexpr (kSource == Source::kGptq) {
    constexpr int kRows = kTileK / kPf;
    for (int idx = threadIdx.x; idx < kRows * tn; idx += kThreads) {
      const int r = idx / tn, c = idx - r * tn;
      const uint32_t word = in[static_cast<int64_t>(k0 / kPf + r) * size_n + n0 + c];
#pragma unroll
      for (int i = 0; i < kPf; ++i) {
        tile[r * kPf + i][c] = static_cast<uint8_t>((word >> (kBits * i)) & kMask);
      }
    }
  } else if constexpr (kSource == Source::kGptqPerm) {
    for (int idx = threadIdx.x; idx < kTileK * tn; idx += kThreads) {
      const int k = idx / tn, c = idx - k * tn;
      const int src = perm[k0 + k];
      const uint32_t word = in[static_cast<int64_t>(src / kPf) * size_n + n0 + c];
      tile[k][c] = static_cast<uint8_t>((word >> (kBits * (src % kPf))) & kMask);
    }
  } else {
    // AWQ: logical column j of a word lives in field kOrder[j].
    constexpr int kOrder4[8] = {0, 4, 1, 5, 2, 6, 3, 7};
    constexpr int kOrder8[4] = {0, 2, 1, 3};
    const int words = tn / kPf;
    const int row_words = size_n / kPf;
    for (int idx = threadIdx.x; idx < kTileK * words; idx += kThreads) {
      const int k = idx / words, cw = idx - k * words;
      const uint32_t word = in[static_cast<int64_t>(k0 + k) * row_words + n0 / kPf + cw];
#pragma unroll
      for (int j = 0; j < kPf; ++j) {
        const int field = kBits == 4 ? kOrder4[j] : kOrder8[j & 3];
        tile[k][cw * kPf + j] = static_cast<uint8_t>((word >> (kBits * field)) & kMask);
      }
    }
  }
  __syncthreads();

  int64_t out_start;
  if constexpr (kA8) {
    out_start = (static_cast<int64_t>(k0 / 32) * (size_n / 32) + n0 / 32) * kWordsPerChunk;
  } else {
    out_start = static_cast<int64_t>(k0 / 16) * (static_cast<int64_t>(size_n) * 16 / kPf) +
                static_cast<int64_t>(n0) * 16 / kPf;
  }
  const int total_words = kTileK * tn / kPf;
  for (int w4 = threadIdx.x * 4; w4 < total_words; w4 += kThreads * 4) {
    uint32_t words[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int wi = w4 + u;
      const int chunk = wi / kWordsPerChunk;
      const int inner = wi - chunk * kWordsPerChunk;
      uint32_t word = 0;
#pragma unroll
      for (int field = 0; field < kPf; ++field) {
        int k, n;
        ChunkSource<kBits, kA8>(inner, field, k, n);
        word |= static_cast<uint32_t>(tile[k][chunk * kChunkN + n]) << (kBits * field);
      }
      words[u] = word;
    }
    *reinterpret_cast<uint4*>(out + out_start + w4) = make_uint4(words[0], words[1], words[2], words[3]);
  }
}

// ---- one warp per 64-column chunk, no shared memory -----------------------------------------------
//
// Lane 4 g + c of a chunk owns the output words of columns 16 t + g and 16 t + g + 8 (t = 0..3) for rows
// 2c, 2c + 1, 2c + 8, 2c + 9: contiguous, and stored by 16-byte writes that cover 512 (1024) contiguous
// bytes per warp.  The words it needs come straight from global memory in whole 32-byte sectors; bytes and
// nibbles are moved a word at a time, where the staged form above handles every element by itself in
// shared memory.  Several k-tiles per warp keep more loads in flight (8-bit AWQ: one tile of 32 words).
//
// 4096 x 28672, cold, staged form -> this one: GPTQ 4-bit 50.2 -> 21.8 us (5.4 TB/s read plus written), GPTQ 8-bit
// 80.6 -> 46.8, AWQ 8-bit 77.1 -> 64.2; 4096 x 4096 9.2 -> 5.4, 14.6 -> 9.5, 14.1 -> 11.9.  Not for 4-bit AWQ, whose
// words hold eight columns of a row: eight lanes then load the same words for one nibble of each, 55.9 us staged
// and 57.9 this way (2.6 and 3.5 at 1024 x 1024).
template <int kBits, Source kSource>
constexpr int kTilesPerWarp = kBits == 4 ? 4 : kSource == Source::kGptq ? 2 : 1;

// x = four bytes (one per source) -> low nibbles in bits 0..15, high nibbles in bits 16..31.
__device__ __forceinline__ uint32_t SplitNibbles(uint32_t x) {
  const uint32_t lo = x & 0x0F0F0F0Fu, hi = (x >> 4) & 0x0F0F0F0Fu;
  return __byte_perm(lo | (lo >> 4), hi | (hi >> 4), 0x6420u);
}

template <int kBits, Source kSource>
struct WarpTile;

// A source word holds rows 8r .. 8r + 7 of one column.  Lane (g, c) loads the four words of columns
// 16 c + g and + 8; the output words of its own (g, c) take byte c of the four words of each t, so the four
// lanes of a g exchange a 4 x 4 table of words.
template <>
struct WarpTile<4, Source::kGptq> {
  uint32_t w[4];
  __device__ __forceinline__ void Load(const uint32_t* in, int kt, int size_n, int n0, int lane) {
    const uint32_t* src = in + static_cast<int64_t>(2 * kt) * size_n + n0 + 16 * (lane & 3) + (lane >> 2);
    w[0] = __ldg(src);
    w[1] = __ldg(src + size_n);
    w[2] = __ldg(src + 8);
    w[3] = __ldg(src + size_n + 8);
  }
  __device__ __forceinline__ void Store(uint32_t* out, int lane) const {
    // byte b of the four words side by side, for b = 0..3
    const uint32_t p0 = __byte_perm(w[0], w[1], 0x5140u), p1 = __byte_perm(w[2], w[3], 0x5140u);
    const uint32_t p2 = __byte_perm(w[0], w[1], 0x7362u), p3 = __byte_perm(w[2], w[3], 0x7362u);
    uint32_t m[4] = {SplitNibbles(__byte_perm(p0, p1, 0x5410u)), SplitNibbles(__byte_perm(p0, p1, 0x7632u)),
                     SplitNibbles(__byte_perm(p2, p3, 0x5410u)), SplitNibbles(__byte_perm(p2, p3, 0x7632u))};
    // lane t of the quad holds column m[c] of t; transpose, so that lane c holds its words of t = 0..3
    const bool odd = lane & 1, upper = lane & 2;
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, odd ? m[i] : m[i + 1], 1);
      if (odd) {
        m[i] = got;
      } else {
        m[i + 1] = got;
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, upper ? m[i] : m[i + 2], 2);
      if (upper) {
        m[i] = got;
      } else {
        m[i + 2] = got;
      }
    }
    reinterpret_cast<uint4*>(out)[lane] = make_uint4(m[0], m[1], m[2], m[3]);
  }
};

// A source word holds rows 4r .. 4r + 3 of one column: an output word is two bytes of each of two words.
template <>
struct WarpTile<8, Source::kGptq> {
  uint32_t w[16];
  __device__ __forceinline__ void Load(const uint32_t* in, int kt, int size_n, int n0, int lane) {
    const uint32_t* src = in + static_cast<int64_t>(4 * kt + ((lane & 3) >> 1)) * size_n + n0 + (lane >> 2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      w[2 * j] = __ldg(src + 8 * j);
      w[2 * j + 1] = __ldg(src + 2 * static_cast<int64_t>(size_n) + 8 * j);
    }
  }
  __device__ __forceinline__ void Store(uint32_t* out, int lane) const {
    const uint32_t select = (lane & 1) ? 0x7362u : 0x5140u;
    uint32_t m[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) m[j] = __byte_perm(w[2 * j], w[2 * j + 1], select);
    reinterpret_cast<uint4*>(out)[2 * lane] = make_uint4(m[0], m[1], m[2], m[3]);
    reinterpret_cast<uint4*>(out)[2 * lane + 1] = make_uint4(m[4], m[5], m[6], m[7]);
  }
};

// A source word holds four columns of one row, column j in byte {0, 2, 1, 3}[j].
template <>
struct WarpTile<8, Source::kAwq> {
  uint32_t w[32];
  __device__ __forceinline__ void Load(const uint32_t* in, int kt, int size_n, int n0, int lane) {
    const int64_t pitch = size_n / 4;
    const uint32_t* src = in + (static_cast<int64_t>(kt) * 16 + 2 * (lane & 3)) * pitch + n0 / 4 + (lane >> 4);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int j = 0; j < 8; ++j) w[8 * r + j] = __ldg(src + ((r & 1) + 8 * (r >> 1)) * pitch + 2 * j);
    }
  }
  __device__ __forceinline__ void Store(uint32_t* out, int lane) const {
    const int j4 = (lane >> 2) & 3, byte = ((j4 & 1) << 1) | (j4 >> 1);
    const uint32_t select = static_cast<uint32_t>(byte) | (static_cast<uint32_t>(byte + 4) << 4);
    uint32_t m[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      m[j] = __byte_perm(__byte_perm(w[j], w[16 + j], select), __byte_perm(w[8 + j], w[24 + j], select), 0x5410u);
    }
    reinterpret_cast<uint4*>(out)[2 * lane] = make_uint4(m[0], m[1], m[2], m[3]);
    reinterpret_cast<uint4*>(out)[2 * lane + 1] = make_uint4(m[4], m[5], m[6], m[7]);
  }
};

template <int kBits, Source kSource>
__global__ void __launch_bounds__(kThreads) RepackWarpKernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                            int size_k, int size_n) {
  constexpr int kU = kTilesPerWarp<kBits, kSource>;
  const int lane = threadIdx.x & 31, chunks = size_n / 64, tiles = size_k / 16;
  const long long unit = static_cast<long long>(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5);
  const int kt0 = static_cast<int>(unit / chunks) * kU, chunk = static_cast<int>(unit % chunks);
  WarpTile<kBits, kSource> tile[kU];
#pragma unroll
  for (int u = 0; u < kU; ++u) {
    if (kt0 + u < tiles) tile[u].Load(in, kt0 + u, size_n, chunk * 64, lane);
  }
  constexpr int kWords = 1024 * kBits / 32;  // output words of a tile
#pragma unroll
  for (int u = 0; u < kU; ++u) {
    if (kt0 + u < tiles) tile[u].Store(out + (static_cast<int64_t>(kt0 + u) * chunks + chunk) * kWords, lane);
  }
}

template <int kBits, Source kSource>
int LaunchWarps(const int32_t* in, int32_t* out, int64_t size_k, int64_t size_n, cudaStream_t stream) {
  constexpr int kU = kTilesPerWarp<kBits, kSource>;
  const int64_t units = (size_n / 64) * ((size_k / 16 + kU - 1) / kU);
  const int64_t blocks = (units + kThreads / 32 - 1) / (kThreads / 32);
  RepackWarpKernel<kBits, kSource><<<static_cast<unsigned>(blocks), kThreads, 0, stream>>>(
      reinterpret_cast<const uint32_t*>(in), reinterpret_cast<uint32_t*>(out), static_cast<int>(size_k),
      static_cast<int>(size_n));
  return CheckLaunch("marlin repack launch");
}

template <int kBits, bool kA8, Source kSource>
int Launch(const int32_t* in, const int32_t* perm, int32_t* out, int64_t size_k, int64_t size_n,
           cudaStream_t stream) {
  constexpr int kTileK = kA8 ? 32 : 16;
  const dim3 grid(static_cast<unsigned>((size_n + kTileN - 1) / kTileN),
                  static_cast<unsigned>(size_k / kTileK));
  RepackKernel<kBits, kA8, kSource><<<grid, kThreads, 0, stream>>>(
      reinterpret_cast<const uint32_t*>(in), perm, reinterpret_cast<uint32_t*>(out),
      static_cast<int>(size_k), static_cast<int>(size_n));
  return CheckLaunch("marlin repack launch");
}

int CheckCommon(const void* in, const void* out, int64_t size_k, int64_t size_n, int num_bits,
                int is_a_8bit) {
  IOB_REQUIRE(in != nullptr && out != nullptr, "marlin repack: null weight pointer");
  IOB_REQUIRE(num_bits == 4 || num_bits == 8, "marlin repack: `num_bits` must be 4 or 8");
  IOB_REQUIRE(size_k > 0 && size_n > 0 && size_k % 16 == 0 && size_n % 64 == 0,
              "marlin repack: needs positive `size_k` divisible by 16 and `size_n` divisible by 64");
  IOB_REQUIRE(!is_a_8bit || size_k % 32 == 0,
              "marlin repack: `size_k` must be divisible by 32 for 8-bit-activation layouts");
  IOB_REQUIRE(size_k <= INT32_MAX && size_n <= INT32_MAX && size_k / 16 <= 65535,
              "marlin repack: dimensions exceed kernel limits");
  IOB_REQUIRE(reinterpret_cast<uintptr_t>(out) % 16 == 0 && reinterpret_cast<uintptr_t>(in) % 4 == 0,
              "marlin repack: output must be 16-byte aligned");
  return IOB_OK;
}

}  // namespace
}  // namespace iob

extern "C" int infiniops_b200_gptq_marlin_repack(const int32_t* b_q_weight, const int32_t* perm,
                                                 int64_t size_k, int64_t size_n, int num_bits,
                                                 int is_a_8bit, int32_t* out, void* stream) {
  using namespace iob;
  if (const int rc = CheckCommon(b_q_weight, out, size_k, size_n, num_bits, is_a_8bit)) return rc;
  IOB_REQUIRE(!(is_a_8bit && perm != nullptr),
              "gptq_marlin_repack: `perm` is not supported for 8-bit-activation layouts");
  auto s = static_cast<cudaStream_t>(stream);
  if (perm != nullptr) {
    return num_bits == 4 ? Launch<4, false, Source::kGptqPerm>(b_q_weight, perm, out, size_k, size_n, s)
                         : Launch<8, false, Source::kGptqPerm>(b_q_weight, perm, out, size_k, size_n, s);
  }
  if (num_bits == 4) {
    if (is_a_8bit) return Launch<4, true, Source::kGptq>(b_q_weight, nullptr, out, size_k, size_n, s);
    // Small matrices leave the warp form too few warps: 2.6 us staged and 2.8 us this way at 1024 x 1024, 2.7 and 2.9 at
    // 1536 x 1024, but 3.3 and 3.0 at 1024 x 3072.
    return size_k * size_n < (2 << 20) ? Launch<4, false, Source::kGptq>(b_q_weight, nullptr, out, size_k, size_n, s)
                                       : LaunchWarps<4, Source::kGptq>(b_q_weight, out, size_k, size_n, s);
  }
  return is_a_8bit ? Launch<8, true, Source::kGptq>(b_q_weight, nullptr, out, size_k, size_n, s)
                   : LaunchWarps<8, Source::kGptq>(b_q_weight, out, size_k, size_n, s);
}

extern "C" int infiniops_b200_awq_marlin_repack(const int32_t* b_q_weight, int64_t size_k,
                                                int64_t size_n, int num_bits, int is_a_8bit,
                                                int32_t* out, void* stream) {
  using namespace iob;
  if (const int rc = CheckCommon(b_q_weight, out, size_k, size_n, num_bits, is_a_8bit)) return rc;
  auto s = static_cast<cudaStream_t>(stream);
  if (num_bits == 4) {
    return is_a_8bit ? Launch<4, true, Source::kAwq>(b_q_weight, nullptr, out, size_k, size_n, s)
                     : Launch<4, false, Source::kAwq>(b_q_weight, nullptr, out, size_k, size_n, s);
  }
  return is_a_8bit ? Launch<8, true, Source::kAwq>(b_q_weight, nullptr, out, size_k, size_n, s)
                   : LaunchWarps<8, Source::kAwq>(b_q_weight, out, size_k, size_n, s);
}
