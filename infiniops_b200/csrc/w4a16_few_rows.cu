// W4A16 / W8A16 GEMM for at most 16 activation rows per weight matrix: decode-sized dense linears and
// routed GEMMs with 8- or 16-row routing blocks.
//
// What bounds it: one pass over the packed weights.  The tensor-memory kernel of w4a16_gemm.cu spends a
// 128 x 16 x 16 instruction slot whatever the number of tokens and needs 10 to 15 us of set-up, ring fill and
// split-K hand-over per launch; with so few tokens the register-operand MMA (m16n8k16) has the rate, and a
// Marlin word *is* its A fragment -- columns g, g + 8 and k pairs {2c, 2c+1}, {2c+8, 2c+9} of lane 4g + c --
// with the weights as the 16 rows and the tokens as the 8 columns.  So a word comes by a 16-byte
// asynchronous copy (coalesced, 512 bytes per warp) into a slot that only its own lane reads back -- no
// barrier, and no registers held while it is under way --, is expanded to exact 16-bit integers q - zero and
// multiplied at once.
//
// Split: a warp owns 64 columns and every kWarps-th 128-k chunk of its block's share of K; kWarps warps are a
// block, up to eight blocks that share a column tile are a cluster.  Partial sums meet in shared memory and
// over the cluster's distributed shared memory in a fixed order: no scratch, no counters, the same bits on
// every run.  Each warp keeps 4 KB of weights in flight ahead of their use (8 KB of 8-bit weights at up to 8 rows),
// refilled slab by slab.
// Activations of a chunk (live rows only) and its scales and zero points come the same way into a warp's own
// double buffer, so no block-wide barrier stands in the main loop.
//
// Scales are applied per group in fp32 to the products of the exact integers.
//
// Two token tiles of 4-bit weights sit at the cap of 128 registers (two blocks an SM) and spill 16 to 24 bytes, as do two
// tiles of 8-bit weights with zero points in bfloat16.
//
// Measured, cold L2, against the tensor-memory kernel: the four linears of a 4096 / 14336 layer as four launches,
// 74.9 -> 67.5 us at 1 row (uint4), 73.6 -> 61.8 at 16 rows (uint4b8, float16), 121.6 -> 66.6 at 7 rows (8-bit,
// 3.4 TB/s).  Not for a batch of linears in one launch: the persistent blocks of the tensor-memory kernel pay their
// set-up once for all of them (sixteen linears of 1..64 rows: 191 us, with the small ones here 200).
// Error against 64-bit arithmetic: the rounding of the result (0.00165 in the 2-norm for bfloat16), where the other
// kernel also rounds the scaled weights of 8-bit types and groups of 64 (0.0023).
#include "w4a16_few_rows.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace iob {
namespace {

constexpr int kWarps = 8;
constexpr int kResident = 2;            // blocks per SM: 16 warps with 128 registers
constexpr int kThreads = kWarps * 32;
constexpr int kCols = 64;               // columns per block (and per warp)
constexpr int kChunk = 128;             // k per step of a warp
constexpr int kSteps = kChunk / 16;
constexpr int kPitch = kChunk * 2 + 16; // bytes of a staged activation row: an odd number of 16-byte units
// scales and zero points of up to two groups: 64 x 2 bytes and 32 (4-bit) or 64 (8-bit) bytes each
constexpr int kScaleBytes = 128, kZeroBytes = 64, kGroupBytes = 2 * (kScaleBytes + kZeroBytes);
constexpr int kRedPitch = kCols + 4;
constexpr int kMaxSplit = 8;            // portable cluster size

__device__ __forceinline__ uint32_t Smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint4 LdShared16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void CopyAsync16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void CopyCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All but the `kPending` youngest groups of this lane's copies have landed.
template <int kPending>
__device__ __forceinline__ void CopyWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}
__device__ __forceinline__ void LdMatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// d = a b (+ d unless `kFirst`)
template <typename T, bool kFirst>
__device__ __forceinline__ void Mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  const float c0 = kFirst ? 0.0f : d[0], c1 = kFirst ? 0.0f : d[1], c2 = kFirst ? 0.0f : d[2], c3 = kFirst ? 0.0f : d[3];
  if constexpr (std::is_same_v<T, __half>) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
  }
}

// Position of logical column n inside a row of scales.  Provider layout: a row is cut into blocks
// of 64 columns stored as [n % 8][n / 8] (so that the four columns c, c + 8, c + 16, c + 24 an MMA
// thread owns are adjacent); with a single group, blocks of 32 stored as [(n % 8) / 2][n / 8][n % 2].
__device__ __forceinline__ int ScaleColumnOf(int layout, int groups, int n) {
  if (layout == 0) return n;
  if (groups > 1) return (n & ~63) + ((n & 7) << 3) + ((n & 63) >> 3);
  return (n & ~31) + (((n & 7) >> 1) << 3) + (((n & 31) >> 3) << 1) + (n & 1);
}
// Provider layout of the zero points: word (n / 64) * 8 + n % 8 of a row holds the eight columns
// n % 8 + 8 j of the block, column j in nibble j / 2 + 4 (j % 2).
__device__ __forceinline__ int ZeroNibble(int j) { return (j >> 1) + 4 * (j & 1); }

// ---- packed words -> exact 16-bit values ------------------------------------------------------------
template <typename T>
__device__ __forceinline__ uint32_t Sub2(uint32_t a, uint32_t b) {
  using H2 = std::conditional_t<std::is_same_v<T, __half>, __half2, __nv_bfloat162>;
  const H2 r = __hsub2(*reinterpret_cast<const H2*>(&a), *reinterpret_cast<const H2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
template <typename T>
__device__ __forceinline__ uint32_t Mul2(uint32_t a, uint32_t b) {
  using H2 = std::conditional_t<std::is_same_v<T, __half>, __half2, __nv_bfloat162>;
  const H2 r = __hmul2(*reinterpret_cast<const H2*>(&a), *reinterpret_cast<const H2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// What `Expand` takes off a column's biased words: 4-bit, 16-bit pairs of 1024 + zero (float16) or
// 128 + zero (bfloat16); 8-bit, pairs of 1024 + zero (float16) or the float32 2^23 + zero (bfloat16).
template <typename T, FewRowsWeights kW>
__device__ __forceinline__ uint32_t CentreOf(uint32_t zero) {
  if constexpr (kW == FewRowsWeights::kInt8 && !std::is_same_v<T, __half>) return 0x4B000000u | zero;
  return (zero | (std::is_same_v<T, __half> ? 0x6400u : 0x4300u)) * 0x10001u;
}
template <typename T>
__device__ __forceinline__ uint32_t Nibbles(uint32_t word, uint32_t centre) {
  constexpr uint32_t kMagic = std::is_same_v<T, __half> ? 0x64006400u : 0x43004300u;
  uint32_t biased;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(biased) : "r"(word), "r"(0x000F000Fu), "r"(kMagic));
  return Sub2<T>(biased, centre);
}
// float16, nibbles at bits 4..7 of each half in place: 1024 + 16 q, brought to q - zero by one exact fused
// multiply-add, (1024 + 16 q) / 16 - (64 + zero).  Saves the shift; takes a second constant per column, so only
// where that is an immediate or the registers are there.
__device__ __forceinline__ uint32_t HighNibbles(uint32_t word, uint32_t minus_64_zero) {
  uint32_t biased;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(biased) : "r"(word), "r"(0x00F000F0u), "r"(0x64006400u));
  const uint32_t sixteenth = 0x2C002C00u;
  const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&biased), *reinterpret_cast<const __half2*>(&sixteenth),
                            *reinterpret_cast<const __half2*>(&minus_64_zero));
  return *reinterpret_cast<const uint32_t*>(&r);
}
template <typename T, int kNt, FewRowsWeights kW, bool kZeros>
constexpr bool kHighNibbles = std::is_same_v<T, __half> && kW == FewRowsWeights::kInt4 && (kNt == 1 || !kZeros);
// Bytes 0 and 2 (`kOdd` = 0: k = 2c, 2c + 1) or 1 and 3 (`kOdd` = 1: k = 2c + 8, 2c + 9) of a word.
template <typename T, FewRowsWeights kW, int kOdd>
__device__ __forceinline__ uint32_t Bytes(uint32_t word, uint32_t centre) {
  if constexpr (kW == FewRowsWeights::kFloat8) {
    // exponent and mantissa to where T keeps them, the difference of the exponent biases multiplied back in: exact
    const uint32_t v = __byte_perm(word, 0u, kOdd ? 0x3414u : 0x2404u);
    if constexpr (std::is_same_v<T, __half>) return Mul2<T>((v & 0x80008000u) | ((v >> 1) & 0x3F803F80u), 0x5C005C00u);
    return Mul2<T>((v & 0x80008000u) | ((v >> 4) & 0x07F007F0u), 0x7B807B80u);
  } else if constexpr (std::is_same_v<T, __half>) {
    return Sub2<T>(__byte_perm(word, 0x64646464u, kOdd ? 0x4341u : 0x4240u), centre);
  } else {
    // through float32 (2^23 + q); |q - zero| <= 255 has eight significant bits, so the upper half is all of it
    const float c = __uint_as_float(centre);
    const float lo = __uint_as_float(__byte_perm(word, 0x4B000000u, kOdd ? 0x7541u : 0x7540u)) - c;
    const float hi = __uint_as_float(__byte_perm(word, 0x4B000000u, kOdd ? 0x7543u : 0x7542u)) - c;
    return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632u);
  }
}
template <FewRowsWeights kW>
struct Words {  // a lane's words of one 16-k slab: 64 columns by 16 k per warp
  static constexpr int kVecs = kW == FewRowsWeights::kInt4 ? 1 : 2;
  uint4 v[kVecs];
};
// MMA A fragment of columns 16 t .. 16 t + 15.
template <typename T, FewRowsWeights kW, bool kHigh>
__device__ __forceinline__ void Expand(uint32_t (&a)[4], const Words<kW>& w, int t, uint32_t centre_lo, uint32_t centre_hi,
                                       uint32_t high_lo, uint32_t high_hi) {
  if constexpr (kW == FewRowsWeights::kInt4) {
    const uint32_t word = t == 0 ? w.v[0].x : t == 1 ? w.v[0].y : t == 2 ? w.v[0].z : w.v[0].w;
    a[0] = Nibbles<T>(word, centre_lo);
    const uint32_t word8 = word >> 8;
    a[1] = Nibbles<T>(word8, centre_hi);
    if constexpr (kHigh) {
      a[2] = HighNibbles(word, high_lo);
      a[3] = HighNibbles(word8, high_hi);
    } else {
      a[2] = Nibbles<T>(word >> 4, centre_lo);
      a[3] = Nibbles<T>(word >> 12, centre_hi);
    }
  } else {
    const uint4& v = w.v[t >> 1];
    const uint32_t lo = (t & 1) ? v.z : v.x, hi = (t & 1) ? v.w : v.y;
    a[0] = Bytes<T, kW, 0>(lo, centre_lo);
    a[1] = Bytes<T, kW, 0>(hi, centre_hi);
    a[2] = Bytes<T, kW, 1>(lo, centre_lo);
    a[3] = Bytes<T, kW, 1>(hi, centre_hi);
  }
}

// 16-k slabs of weights under way per warp.
template <int kNt, FewRowsWeights kW>
constexpr int kRingSlabs = kNt == 2 && kW != FewRowsWeights::kInt4 ? 4 : 8;
template <FewRowsWeights kW>
constexpr int kSlabBytes = kW == FewRowsWeights::kInt4 ? 512 : 1024;  // 64 columns x 16 k

// One unit: 64 columns of one problem (or routing block), K shared by `split` blocks of a cluster.
// kNt: token tiles of 8.
template <typename T, int kNt, FewRowsWeights kW, bool kZeros, bool kMoe>
__device__ __forceinline__ void FewRowsTile(const FewRowsParams& p, int tile, int block, uint32_t split, uint32_t rank) {
  constexpr int kRows = 8 * kNt;
  constexpr int kSlab = kSlabBytes<kW>, kRing = kRingSlabs<kNt, kW>;
  constexpr bool kHigh = kHighNibbles<T, kNt, kW, kZeros>;
  constexpr int kActBytes = kRows * kPitch + kGroupBytes;  // a chunk's activations, scales and zero points
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int row_in[kRows], row_out[kRows];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const int n0 = tile * kCols;
  const int chunks = p.k / kChunk;
  const int first = static_cast<int>(static_cast<long long>(chunks) * rank / split) + warp;
  const int last = static_cast<int>(static_cast<long long>(chunks) * (rank + 1) / split);

  asm volatile("griddepcontrol.launch_dependents;");
  int expert = 0;
  if constexpr (kMoe) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (block * p.block_size >= *p.num_post_pad) return;  // all blocks of a split tile
    expert = p.expert_ids[block];
    if (expert < 0) return;
  }

  // ---- weights under way ------------------------------------------------------------------------
  const int words_per_row = p.n * (kW == FewRowsWeights::kInt4 ? 2 : 4);
  const uint32_t* wq = p.wq + static_cast<size_t>(expert) * (p.k / 16) * words_per_row +
                       n0 * (kW == FewRowsWeights::kInt4 ? 2 : 4) + lane * (kW == FewRowsWeights::kInt4 ? 4 : 8);
  const uint32_t slots = Smem(smem) + 2 * kWarps * kActBytes + warp * kRing * kSlab + lane * (kSlab / 32);
  const size_t row_bytes = static_cast<size_t>(words_per_row) * 4;
  const unsigned char* next = reinterpret_cast<const unsigned char*>(wq) + static_cast<size_t>(first) * kSteps * row_bytes;
  auto load = [&](int slot) {  // the warp's next slab
    CopyAsync16(slots + slot * kSlab, next);
    if constexpr (Words<kW>::kVecs == 2) CopyAsync16(slots + slot * kSlab + 16, next + 16);
    next += row_bytes;
  };
  // Rows of the activations and of the result.  (Activation rows that are not live are never staged: whatever the
  // buffers hold there reaches only its own columns of the products, which are not stored.)
  auto set_rows = [&]() {
    if constexpr (kMoe) {
      if (tid < kRows) {
        const int at = block * p.block_size + tid;
        const int id = tid < p.block_size ? p.sorted_ids[at] : p.out_rows;
        const bool live = id < p.out_rows;
        row_in[tid] = live ? (p.a_sorted ? at : id / p.top_k) : -1;
        // (sorted output: a block's padding rows are written too, as products of zeros)
        row_out[tid] = p.out_sorted ? (tid < p.block_size ? at : -1) : live ? id : -1;
      }
    } else if (tid < kRows) {
      row_in[tid] = row_out[tid] = tid < p.m ? tid : -1;
    }
    __syncthreads();
  };
  if constexpr (!kMoe) {
    // Nothing that a predecessor in the stream could have written is read before the wait: not the activations, and
    // not the weights, after a repack or an update.  (Weight copies ahead of it would give 0.2 to 1.7 us a launch:
    // 4096 x 28672, 1 row, back to back 20.3 us against 21.2 with 4-bit weights, 26.8 against 28.5 with 8-bit ones.
    // Pulling the slabs into L2 instead gives nothing: 21.2 to 21.5 us and 28.9 to 29.3.)
    set_rows();
    asm volatile("griddepcontrol.wait;" ::: "memory");
  }
  if (first < last) {
#pragma unroll
    for (int s = 0; s < kRing; ++s) load(s);
  }
  const size_t skip_bytes = (kWarps - 1) * kSteps * row_bytes;  // from a chunk's end to the warp's next chunk
  if constexpr (kRing == kSteps) next += skip_bytes;
  CopyCommit();

  // ---- activations -------------------------------------------------------------------------------
  if constexpr (kMoe) set_rows();
  // a lane copies one 16-byte column piece of every second row
  const uint32_t act0 = Smem(smem) + warp * 2 * kActBytes;
  const unsigned char* a = static_cast<const unsigned char*>(p.a) + (lane & 15) * 16;
  const size_t a_row = static_cast<size_t>(p.k) * 2;
  int from[kRows / 2];
  bool second = false;  // any of rows 8..15 live: else their products are not formed
#pragma unroll
  for (int i = 0; i < kRows / 2; ++i) from[i] = row_in[2 * i + (lane >> 4)];
  if constexpr (kNt == 2) {
#pragma unroll
    for (int i = 4; i < 8; ++i) second = second || from[i] >= 0;
    second = __any_sync(0xFFFFFFFFu, second);
  }
  auto stage = [&](int chunk, int buf) {
    const uint32_t dst = act0 + buf * kActBytes + (lane >> 4) * kPitch + (lane & 15) * 16;
    const unsigned char* column = a + static_cast<size_t>(chunk) * (kChunk * 2);
#pragma unroll
    for (int i = 0; i < kRows / 2; ++i) {
      if (from[i] >= 0) CopyAsync16(dst + 2 * i * kPitch, column + from[i] * a_row);
    }
    // lanes 0..7 / 8..15: scales of the chunk's first / second group, 16..19 / 20..23: their zero points
    const int which = lane < 16 ? lane >> 3 : (lane >> 2) & 1;
    if (lane < 24 && (which == 0 || p.group_size == 64)) {
      const size_t row = static_cast<size_t>(expert) * p.groups + (chunk * kChunk + which * 64) / p.group_size;
      const uint32_t at = act0 + buf * kActBytes + kRows * kPitch + which * (kScaleBytes + kZeroBytes);
      if (lane < 16) {
        CopyAsync16(at + (lane & 7) * 16, static_cast<const T*>(p.scales) + row * p.n + n0 + (lane & 7) * 8);
      } else if constexpr (kZeros) {
        constexpr int kPieces = kW == FewRowsWeights::kInt4 ? 2 : 4;
        if ((lane & 3) < kPieces) {
          CopyAsync16(at + kScaleBytes + (lane & 3) * 16,
                      reinterpret_cast<const uint8_t*>(p.zeros) + (row * p.n + n0) / 64 * (kPieces * 16) + (lane & 3) * 16);
        }
      }
    }
    CopyCommit();
  };
  if (first < last) stage(first, 0);

  // ---- main loop ---------------------------------------------------------------------------------
  float total[4][kNt][4] = {};
  int buf = 0;
  for (int chunk = first; chunk < last; chunk += kWarps, buf ^= 1) {
    const bool more = chunk + kWarps < last;
    if (more) {
      stage(chunk + kWarps, buf ^ 1);
    } else {
      CopyCommit();  // the same number of groups in every chunk
    }
    const int halves = p.group_size == 64 ? 2 : 1;
    float scale[8];
    uint32_t centre[8], high[8];
    float acc[4][kNt][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 0) {
        // this chunk's activations and first slab have landed (the first chunk's came after its slabs)
        if (chunk == first) {
          CopyWait<1>();
        } else {
          CopyWait<kRing>();
        }
        __syncwarp();
      }
      if (h == 0 || halves == 2) {
        // constants of this group: columns g + 8 j
        const unsigned char* rows = smem + (warp * 2 + buf) * kActBytes + kRows * kPitch + h * (kScaleBytes + kZeroBytes);
        const T* srow = reinterpret_cast<const T*>(rows);
        if (p.layout == 0) {
#pragma unroll
          for (int j = 0; j < 8; ++j) scale[j] = ToFloat<T>(srow[g + 8 * j]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) scale[j] = ToFloat<T>(srow[ScaleColumnOf(1, p.groups, g + 8 * j)]);
        }
        if constexpr (!kZeros) {
#pragma unroll
          for (int j = 0; j < 8; ++j) centre[j] = CentreOf<T, kW>(kW == FewRowsWeights::kInt4 ? 8 : 128);
        } else if constexpr (kW == FewRowsWeights::kInt4) {
          const uint32_t* zrow = reinterpret_cast<const uint32_t*>(rows + kScaleBytes);
          if (p.layout == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) centre[j] = CentreOf<T, kW>((zrow[j] >> (4 * g)) & 0xF);
          } else {
            const uint32_t z = zrow[g];
#pragma unroll
            for (int j = 0; j < 8; ++j) centre[j] = CentreOf<T, kW>((z >> (4 * ZeroNibble(j))) & 0xF);
          }
        } else {
          const uint8_t* zrow = rows + kScaleBytes + g;
#pragma unroll
          for (int j = 0; j < 8; ++j) centre[j] = CentreOf<T, kW>(zrow[8 * j]);
        }
        if constexpr (kHigh) {
#pragma unroll
          for (int j = 0; j < 8; ++j) high[j] = kZeros ? Sub2<T>(0x63806380u, centre[j]) : 0xD480D480u;  // -(64 + zero)
        }
      }
#pragma unroll
      for (int pair = 0; pair < 2; ++pair) {
        uint32_t b[kNt][4];
#pragma unroll
        for (int i = 0; i < kNt; ++i) {
          LdMatrix4(b[i], act0 + buf * kActBytes + (8 * i + (lane & 7)) * kPitch + (4 * h + 2 * pair) * 32 + (lane >> 3) * 16);
        }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int step = 4 * h + 2 * pair + s;
          // groups younger than this slab's: the copies of the slabs after it and, if it was issued a
          // chunk ago, the next activations
          if (step >= kRing) {
            CopyWait<kRing - 1>();
          } else if (step > 0) {
            CopyWait<kRing>();
          }
          Words<kW> words;
          words.v[0] = LdShared16(slots + (step % kRing) * kSlab);
          if constexpr (Words<kW>::kVecs == 2) words.v[1] = LdShared16(slots + (step % kRing) * kSlab + 16);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            uint32_t frag[4];
            Expand<T, kW, kHigh>(frag, words, t, centre[2 * t], centre[2 * t + 1], high[2 * t], high[2 * t + 1]);
            // the first slab of a group starts its sums
            auto multiply = [&](auto is_first) {
              Mma<T, decltype(is_first)::value>(acc[t][0], frag, b[0][2 * s], b[0][2 * s + 1]);
              if constexpr (kNt == 2) {
                if (second) Mma<T, decltype(is_first)::value>(acc[t][1], frag, b[1][2 * s], b[1][2 * s + 1]);
              }
            };
            if (step == 0 || (step == 4 && halves == 2)) {
              multiply(std::true_type{});
            } else {
              multiply(std::false_type{});
            }
          }
          // refill the slot just read (the products above have used its words)
          if (step + kRing < kSteps || more) load(step % kRing);
          if (step == kSteps - 1 - kRing % kSteps) next += skip_bytes;  // that was a chunk's last slab
          CopyCommit();
        }
      }
      if (h == 1 || halves == 2) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
          for (int i = 0; i < kNt; ++i) {
            if (i == 1 && !second) continue;
#pragma unroll
            for (int e = 0; e < 4; ++e) total[t][i][e] = fmaf(scale[2 * t + (e >> 1)], acc[t][i][e], total[t][i][e]);
          }
        }
      }
    }
    __syncwarp();  // every lane has read this buffer before it is staged again
  }

  // ---- sums over the warps, then over the cluster ------------------------------------------------
  __syncthreads();
  float* red = reinterpret_cast<float*>(smem);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
#pragma unroll
    for (int i = 0; i < kNt; ++i) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        red[(warp * kRows + 8 * i + 2 * c + (e & 1)) * kRedPitch + 16 * t + g + 8 * (e >> 1)] = total[t][i][e];
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < kRows * kCols; i += kThreads) {
    const int at = (i / kCols) * kRedPitch + i % kCols;
    float v = red[at];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) v += red[w * kRows * kRedPitch + at];
    red[at] = v;
  }
  if (split > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  // Two columns of one row, summed over the cluster, with bias and routing weight.
  const T* bias = p.bias != nullptr ? static_cast<const T*>(p.bias) + static_cast<size_t>(expert) * p.n + n0 : nullptr;
  auto sum = [&](int r, int col, float weight, float (&v)[2]) {
    v[0] = v[1] = 0.0f;
    if (row_in[r] >= 0) {  // (a padding row of sorted output has no products)
      if (split == 1) {
        v[0] = red[r * kRedPitch + col];
        v[1] = red[r * kRedPitch + col + 1];
      } else {
        const uint32_t at = Smem(red + r * kRedPitch + col);
        for (uint32_t s = 0; s < split; ++s) {
          uint32_t remote;
          float x, y;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(s));
          asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(remote) : "memory");
          v[0] += x;
          v[1] += y;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (bias != nullptr) v[e] += ToFloat<T>(bias[col + e]);
      if (kMoe && p.mul_weights) v[e] *= weight;
    }
  };
  T* out = static_cast<T*>(p.out);
  for (int i = (rank * kThreads + tid) * 2; i < kRows * kCols; i += static_cast<int>(split) * kThreads * 2) {
    const int r = i / kCols, col = i % kCols;
    const int to = row_out[r];
    if (to < 0) continue;
    float weight = 1.0f;
    if constexpr (kMoe) {
      if (p.mul_weights) weight = p.topk_weights[to];  // (not with sorted output)
    }
    float v[2];
    T pair[2];
    T* dst = out + static_cast<size_t>(to) * p.out_ld + p.out_col0 + n0 + col;
    if (kMoe && p.fuse_silu) {
      // gate columns 32 b + 0..15 with their up columns 32 b + 16..31, both rounded first as stored products are
      if (col & 16) continue;
      float up[2];
      sum(r, col, weight, v);
      sum(r, col + 16, weight, up);
#pragma unroll
      for (int e = 0; e < 2; ++e) pair[e] = SiluMulRounded<T>(ToFloat<T>(FromFloat<T>(v[e])), ToFloat<T>(FromFloat<T>(up[e])));
      dst = out + static_cast<size_t>(to) * p.out_ld + n0 / 2 + (col >> 5) * 16 + (col & 15);
    } else {
      sum(r, col, weight, v);
#pragma unroll
      for (int e = 0; e < 2; ++e) pair[e] = FromFloat<T>(v[e]);
    }
    *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(pair);
  }
  __syncwarp();
  if (split > 1) {  // no block leaves while another still reads its sums
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// Which unit a block works on.  Blocks come in clusters of `size`; the first `whole` units (a multiple of it)
// are taken by one block each, every later one by a whole cluster that splits K.
struct Place {
  int unit;
  uint32_t split, rank;
};
__device__ __forceinline__ Place PlaceOf(int whole) {
  uint32_t size, rank;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(size));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  if (static_cast<int>(blockIdx.x) < whole) return Place{static_cast<int>(blockIdx.x), 1u, 0u};
  return Place{whole + static_cast<int>((blockIdx.x - whole) / size), size, rank};
}

template <typename T, int kNt, FewRowsWeights kW, bool kZeros, bool kMoe>
__global__ void __launch_bounds__(kThreads, kResident) FewRowsKernel(const FewRowsParams p, int whole) {
  const Place at = PlaceOf(whole);
  const int tile = kMoe ? at.unit / p.blocks : at.unit;
  FewRowsTile<T, kNt, kW, kZeros, kMoe>(p, tile, kMoe ? at.unit - tile * p.blocks : 0, at.split, at.rank);
}

// How many units are taken whole and by how many blocks each of the others is shared.  A block takes chunks /
// (kWarps * split) steps and about one and a half steps' time of set-up and summing (one more with a cluster's
// exchange).  The whole units fill the SMs' slots a number of times; the rest, which would leave most
// slots empty for a unit's full time, is split.  Clusters leave about a tenth of the slots unused.
// (A model, not measurements of its parts.  What it plans took 1.5 % longer than the best of all plans on the
// average of 13 shapes from 1024 x 1536 to 4096 x 28672, 1 and 16 rows, 4 and 8 bits; 20 % at worst, 2048 x 5632.)
//
// `live`: units that will have work.  A routed launch has room for the worst routing, and blocks past the sort's
// count return at once; where such are expected, the units with work lie scattered among them, so all units are
// treated alike: taken whole, or all split.  (Planned as if all had work, 16 x 7168 x 1024 with 4 rows per expert
// took 40.0 us, its last 8 of 304 units split over clusters of 8, and takes 24.8 this way; 16 x 14336 x 3648 with 1
// row per expert 116 -> 87, 64 x 14336 x 7168 536 -> 507.)
struct Plan {
  int whole, split;
};
Plan PlanFor(int64_t units, double live, int chunks) {
  const int slots = kResident * NumSms();
  const bool padded = live < static_cast<double>(units) * 0.9;
  auto time = [&](double blocks, double slots_used, int share) {
    const int per_block = (chunks + share - 1) / share, steps = (per_block + kWarps - 1) / kWarps;
    return blocks <= 0 ? 0.0 : std::ceil(blocks / slots_used) * (steps + (share > 1 ? 2.5 : 1.5));
  };
  Plan best{static_cast<int>(units), 1};
  double best_cost = time(padded ? live : static_cast<double>(units), slots, 1);
  const int most = std::min(kMaxSplit, chunks);
  for (int split = 2; split <= most; split *= 2) {
    for (int64_t rounds = 0; rounds * slots <= units; ++rounds) {
      if (padded && rounds > 0) break;
      if (units / slots > 8) rounds = std::max(rounds, units / slots - 1);  // many rounds: only how they end matters
      const int64_t whole = rounds * slots / split * split;
      const double rest = padded ? live : static_cast<double>(units - whole);
      const double cost = time(static_cast<double>(whole), slots, 1) + time(rest * split, 0.9 * slots, split);
      if (cost < best_cost - 1e-9) {
        best_cost = cost;
        best = Plan{static_cast<int>(whole), split};
      }
    }
  }
  return best;
}
// Routing blocks that hold rows, of `p.blocks`, for even routing: each token goes to `top_k` of the experts, so an
// expert's rows are binomial (past two blocks of them: their share of blocks and half a block more).
double LiveBlocks(const FewRowsParams& p) {
  const double q = std::min(1.0, static_cast<double>(p.top_k) / p.experts), share = q * p.m;
  double per_expert = 0.0;
  if (q >= 1.0 || share > 2.0 * p.block_size) {
    per_expert = q >= 1.0 ? std::ceil(share / p.block_size) : share / p.block_size + 0.5;
  } else {
    double term = std::pow(1.0 - q, p.m);
    for (int n = 1; n <= std::min(p.m, 4 * p.block_size); ++n) {
      term *= (p.m - n + 1.0) / n * q / (1.0 - q);
      per_expert += term * ((n + p.block_size - 1) / p.block_size);
    }
  }
  return std::min(static_cast<double>(p.blocks), p.experts * per_expert);
}

template <int kNt, FewRowsWeights kW, typename Kernel, typename Params>
int LaunchClusters(Kernel kernel, const Params& params, int64_t units, const Plan& plan, bool* configured, cudaStream_t stream) {
  constexpr int kStage = 2 * kWarps * (8 * kNt * kPitch + kGroupBytes) + kWarps * kRingSlabs<kNt, kW> * kSlabBytes<kW>;
  constexpr int kSums = kWarps * 8 * kNt * kRedPitch * 4;
  constexpr int smem = kStage > kSums ? kStage : kSums;
  int device = 0;
  cudaGetDevice(&device);
  if (device < 0 || device >= 64 || !configured[device]) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return Fail(IOB_CUDA_ERROR, "W4A16 GEMM (few rows): %s", cudaGetErrorString(err));
    if (device >= 0 && device < 64) configured[device] = true;
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(plan.whole + (units - plan.whole) * plan.split));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = plan.split;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  config.attrs = attr;
  config.numAttrs = 2;
  const cudaError_t err = cudaLaunchKernelEx(&config, kernel, params, plan.whole);
  if (err != cudaSuccess) return Fail(IOB_CUDA_ERROR, "W4A16 GEMM (few rows) launch: %s", cudaGetErrorString(err));
  return CheckLaunch("W4A16 GEMM (few rows) launch");
}

template <typename T, int kNt, FewRowsWeights kW, bool kZeros, bool kMoe>
int Launch(const FewRowsParams& p, cudaStream_t stream) {
  static thread_local bool configured[64] = {};
  const int tiles = p.n / kCols;
  const int64_t units = static_cast<int64_t>(tiles) * (kMoe ? p.blocks : 1);
  const Plan plan = PlanFor(units, kMoe ? tiles * LiveBlocks(p) : static_cast<double>(units), p.k / kChunk);
  return LaunchClusters<kNt, kW>(FewRowsKernel<T, kNt, kW, kZeros, kMoe>, p, units, plan, configured, stream);
}

template <typename T, int kNt, bool kMoe>
int DispatchWeights(FewRowsWeights weights, const FewRowsParams& p, cudaStream_t stream) {
  switch (weights) {
    case FewRowsWeights::kInt4:
      return p.zeros != nullptr ? Launch<T, kNt, FewRowsWeights::kInt4, true, kMoe>(p, stream)
                                : Launch<T, kNt, FewRowsWeights::kInt4, false, kMoe>(p, stream);
    case FewRowsWeights::kInt8:
      return p.zeros != nullptr ? Launch<T, kNt, FewRowsWeights::kInt8, true, kMoe>(p, stream)
                                : Launch<T, kNt, FewRowsWeights::kInt8, false, kMoe>(p, stream);
    default: return Launch<T, kNt, FewRowsWeights::kFloat8, false, kMoe>(p, stream);
  }
}
template <typename T>
int DispatchRows(FewRowsWeights weights, const FewRowsParams& p, cudaStream_t stream) {
  const bool moe = p.expert_ids != nullptr;
  if ((moe ? p.block_size : p.m) <= 8) {
    return moe ? DispatchWeights<T, 1, true>(weights, p, stream) : DispatchWeights<T, 1, false>(weights, p, stream);
  }
  return moe ? DispatchWeights<T, 2, true>(weights, p, stream) : DispatchWeights<T, 2, false>(weights, p, stream);
}

}  // namespace

int FewRowsGemm(int a_dtype, FewRowsWeights weights, const FewRowsParams& p, cudaStream_t stream) {
  return a_dtype == IOB_BF16 ? DispatchRows<__nv_bfloat16>(weights, p, stream) : DispatchRows<__half>(weights, p, stream);
}

}  // namespace iob
