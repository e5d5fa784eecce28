// Flash-style attention for sm_100a on tcgen05 / TMEM: the local queries of one
// strip against the full key/value sequence, which lives as up to 8 per-peer
// slots [B, L_slot, 2C] (K in columns [0,C), V in [C,2C), head h at columns
// h*64..h*64+63).  The slots are read IN PLACE through one TMA descriptor per
// slot: the own strip's fresh K/V and the peers' stale K/V are never
// concatenated.  attention_short_kernel serves one slot of few keys (cross-attention).
//
// Work unit of attention_kernel<kGroups, kTileKV> = up to kGroups query tiles of 128 rows of one (image, head):
// three with key tiles of 64 tokens, or two with 128.  A CTA walks several units (or, with a K/V split, a cluster
// of 2 or 4 CTAs shares one unit).  Warps:
//   4 per group softmax: thread r of a group owns query row r of its tile (= TMEM lane r).  Per K/V tile
//               it reads its row of S once, releases S at once so the next Q K^T can start, takes the row
//               maximum, forms P = exp2(S*scale - m) in fp32 (14 of 16 on the special-function unit, 2 on
//               the FMA pipe), sums the row in fp32 registers, packs P to fp16 and stores it to TENSOR
//               MEMORY (tcgen05.st), from where the P V product reads it as its A operand: P never touches
//               shared memory.  The running maximum m is only raised when the tile maximum exceeds it by
//               more than 8 (a factor of 256, harmless in fp16/fp32) and, while fewer than 128 keys have
//               been seen, by any amount: the largest probability of the first 128 keys is then exactly 1,
//               not rounded to fp16 (error against 64 bits 1 to 3 % smaller at 77 to 231 keys of normal
//               scores, 4 to 13 % where the scores are three times as peaked; 2 x 10 x 4096 x 4096
//               138.2 -> 138.1 us).  Only then O is rescaled in tensor memory (tcgen05.ld / multiply /
//               tcgen05.st) and the row sum in its register.  The result is exact: O and the row sum always
//               refer to the same m.
//               These warps raise their register budget (setmaxnreg) at the expense of the others.
//   1 TMA producer: the Q tiles of a unit (double buffered across units), then a ring of {K tile, V tile}
//               shared by the query tiles
//   kGroups tcgen05.mma issuers, one per query tile; the first owns tensor memory
//
// While one group runs its softmax the tensor core works for the others; the K/V tiles of
// all units of a CTA form one stream, so the first Q K^T of the next unit and the read-out of
// the finished unit's output overlap the unit boundary.
//
// Roofline: tensor cores; algorithmic FLOPs = 4 * L_q * L_kv * 64 per (image, head).  With head dimension 64
// the exponentials are the narrowest resource: 14 of 16 scores at 16 per clock and SM, 1315 TFLOP/s at 1.9 GHz.
// A softmax warp's own dependences (read S, maximum, exponentials, publish P) bound the kernel: 64 % of that unit,
// 54 % of the issue slots and 36 % of the tensor pipe are busy at 2 x 20 x 4096 x 4096, so three warps per scheduler
// work side by side where the work fills them.  Measured (two groups of 128-token tiles -> three of 64):
// 2 x 10 x 4096 x 4096 152 -> 138 us (622 TFLOP/s), 2 x 20 x 4096 x 4096 246 -> 231 (744), 2 x 20 x 1024 x 1024 31.8 -> 25.5,
// 1024 queries against 4 x 1024 keys 56.9 -> 46.5; at 2 x 10 x 16384 x 16384 the two are the faster (1850 -> 1789).  Exponentials on the FMA pipe: none 144.0 us on the first
// shape, 4 of 16 137.8.

#include "bxl_common.cuh"
#include "bxl_host.h"
#include "../../include/basedxl_b200.h"

namespace bxl {

constexpr int kPolyOf16 = 2;        // score pairs of every 16 whose exponentials run on the FMA pipe
constexpr int kHeadDim = 64;
constexpr int kTileQ = 128;
constexpr int kQBytes = kTileQ * kHeadDim * 2;   // one Q tile
constexpr int kMaxSlots = 8;

// kGroups softmax warpgroups (query tiles in flight), key tiles of kTileKV tokens: <3, 64> or <2, 128>.
template <int kGroups, int kTileKV>
struct AttnShape {
  static constexpr int kWarpLoad = 4 * kGroups;   // producer warp; then one MMA issuer warp per group
  static constexpr int kWarpMma = kWarpLoad + 1;
  static constexpr int kThreads = (4 * kGroups + 4) * 32;
  // registers per thread after the split: 12 x 32 x 144 + 4 x 32 x 80 = 512 x 128; 8 x 32 x 208 + 4 x 32 x 88 = 384 x 168
  static constexpr int kSoftmaxRegs = kGroups == 3 ? 144 : 208;
  static constexpr int kOtherRegs = kGroups == 3 ? 80 : 88;
  static_assert(4 * kGroups * kSoftmaxRegs + 4 * kOtherRegs == (kGroups == 3 ? 16 * 128 : 12 * 168), "the registers of the launch");
  static constexpr int kKvStages = kTileKV == 64 ? 6 : 4;
  static constexpr int kKvBytes = kTileKV * kHeadDim * 2;   // one K or V tile
  // tensor memory columns: S_g, O_g (fp32), P_g (two fp16 per column, the A operand of the P V product)
  static constexpr int kTmemO = kGroups * kTileKV, kTmemP = kTmemO + kGroups * kHeadDim;
  static_assert(kTmemP + kGroups * kTileKV / 2 <= 512, "tensor memory");
  // shared memory: 2 buffers x kGroups Q tiles, the ring of K tiles and that of V tiles, barriers
  static constexpr int kQ = 0;
  static constexpr int kK = 2 * kGroups * kQBytes;
  static constexpr int kV = kK + kKvStages * kKvBytes;
  static constexpr int kBar = kV + kKvStages * kKvBytes;
  static constexpr int kTotal = kBar + 1024 + 1024;
  static_assert(kTotal <= 227 * 1024, "shared memory");
  // the merge of a K/V split receives 66 values of a half of the rows, or three times those of a quarter, in the ring
  static_assert(3 * 66 * (kGroups * kTileQ / 4) * 4 <= 2 * kKvStages * kKvBytes, "merge buffer");
};

struct alignas(64) AttnParams {
  CUtensorMap q_map;               // [C_q cols, L_q, B]
  CUtensorMap kv_map[kMaxSlots];   // [2C cols, L_slot, B] per slot
  int n_slots;
  int L_q, L_slot;
  int heads, B;
  int v_col0;                      // column of V for head 0 (= C)
  __half* out;                     // [B, L_q, ld_out]
  long long out_img_stride, ld_out;
  float scale_log2e;               // softmax scale * log2(e)
  int kv_split;                    // K/V range split over a cluster of 1, 2 or 4 CTAs
  int groups;                      // query tiles per unit (1..kGroups of the kernel)
  int* dev_status;
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two fp32 values in one 64-bit register pair: one instruction for both (half the issue slots of the
// softmax's multiply-adds and sums; the rounding is that of the scalar forms).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpair2(f32x2 r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// 2^x on the FMA pipe, for part of the scores: the special-function unit (16 results per clock and SM) is the
// softmax's narrowest unit.  x = n + f with n the nearest integer (the sum with 1.5 * 2^23 + 127 leaves n + 127 in
// the low mantissa bits), 2^f by a degree-5 polynomial fitted to |f| <= 0.5 for the smallest relative error
// (2.1e-7 in fp32 arithmetic, the error bound of the special-function unit), times 2^n built from those bits.
// x <= 8, unless the caller's scale is negative: the result is then wrong from 128 on, where fp16 has long overflowed in
// the other scores; below -120 it is as good as zero; NaN stays NaN.
__device__ __forceinline__ f32x2 poly_exp2(f32x2 x) {
  float x0, x1;
  unpair2(x, x0, x1);
  x = pair2(max_nan(x0, -120.f), max_nan(x1, -120.f));
  const float magic = 12582912.f + 127.f;
  const f32x2 t = add2(x, pair2(magic, magic));
  const f32x2 n = add2(t, pair2(-magic, -magic));
  const f32x2 f = fma2(n, pair2(-1.f, -1.f), x);
  f32x2 p = fma2(f, pair2(1.3276472454890609e-3f, 1.3276472454890609e-3f), pair2(9.675540961325169e-3f, 9.675540961325169e-3f));
  p = fma2(p, f, pair2(5.550713092088699e-2f, 5.550713092088699e-2f));
  p = fma2(p, f, pair2(2.4022120237350464e-1f, 2.4022120237350464e-1f));
  p = fma2(p, f, pair2(6.931469440460205e-1f, 6.931469440460205e-1f));
  p = fma2(p, f, pair2(1.f, 1.f));
  float t0, t1;
  unpair2(t, t0, t1);
  return mul2(p, pair2(__uint_as_float(__float_as_uint(t0) << 23), __uint_as_float(__float_as_uint(t1) << 23)));
}
// P = 2^(s * scale - m) of two neighbouring scores: added to the row sum in fp32, packed to fp16.
template <bool kPoly>
__device__ __forceinline__ uint32_t exp_pair(uint32_t s0, uint32_t s1, f32x2 scale, f32x2 minus_m, f32x2& sum) {
  const f32x2 x = fma2(pair2(__uint_as_float(s0), __uint_as_float(s1)), scale, minus_m);
  float e0, e1;
  f32x2 e;
  if (kPoly) {
    e = poly_exp2(x);
    unpair2(e, e0, e1);
  } else {
    float x0, x1;
    unpair2(x, x0, x1);
    e0 = fast_exp2(x0), e1 = fast_exp2(x1);
    e = pair2(e0, e1);
  }
  sum = add2(sum, e);
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(e1), "f"(e0));
  return r;
}
__device__ __forceinline__ uint32_t pack_f16x2(float a, float b) {
  uint32_t packed;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(b), "f"(a));
  return packed;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Ragged last tile of a slot, one 32-column chunk with nv valid columns (warp-uniform): row
// maximum, and P = exp2(s*sc - m) packed into pk[off .. off+15] with its sum.  Chunks without
// a valid column cost nothing.
__device__ __forceinline__ float ragged_chunk_max(const uint32_t (&v)[32], int nv) {
  float m = -INFINITY;
  if (nv >= 32) {
    float m2 = -INFINITY;
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      m = max3(m, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      m2 = max3(m2, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
    }
    m = fmaxf(m, m2);
  } else if (nv > 0) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < nv) m = fmaxf(m, __uint_as_float(v[i]));
  }
  return m;
}
template <int kWords>
__device__ __forceinline__ float ragged_chunk_p(const uint32_t (&v)[32], uint32_t (&pk)[kWords], int off, int nv, float sc, float m) {
  float s0 = 0.f, s1 = 0.f;
  if (nv >= 32) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float a = fast_exp2(fmaf(__uint_as_float(v[2 * i]), sc, -m)), b = fast_exp2(fmaf(__uint_as_float(v[2 * i + 1]), sc, -m));
      s0 += a, s1 += b;
      pk[off + i] = pack_f16x2(a, b);
    }
  } else if (nv > 0) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float a = (2 * i < nv) ? fast_exp2(fmaf(__uint_as_float(v[2 * i]), sc, -m)) : 0.f;
      const float b = (2 * i + 1 < nv) ? fast_exp2(fmaf(__uint_as_float(v[2 * i + 1]), sc, -m)) : 0.f;
      s0 += a, s1 += b;
      pk[off + i] = pack_f16x2(a, b);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) pk[off + i] = 0u;
  }
  return s0 + s1;
}

// One query row of a finished unit: read O (64 fp32 columns of this thread's TMEM lane),
// normalise by the row sum and store 64 halves.
__device__ __forceinline__ void attn_store_row_inline(uint32_t o_addr, __half* dst, float inv_l) {
  uint32_t o0[32], o1[32];
  tmem_ld_32x32(o_addr, o0);
  tmem_ld_32x32(o_addr + 32, o1);
  tmem_ld_wait();
  if (dst == nullptr) return;
  // 128 bytes of this thread's output row: four whole 32-byte sectors when the row is aligned
  uint32_t w[32];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    w[j] = pack_f16x2(__uint_as_float(o0[2 * j]) * inv_l, __uint_as_float(o0[2 * j + 1]) * inv_l);
    w[16 + j] = pack_f16x2(__uint_as_float(o1[2 * j]) * inv_l, __uint_as_float(o1[2 * j + 1]) * inv_l);
  }
  if ((reinterpret_cast<uintptr_t>(dst) & 31u) == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      st_global_v8(dst + q * 16, w[8 * q], w[8 * q + 1], w[8 * q + 2], w[8 * q + 3], w[8 * q + 4], w[8 * q + 5], w[8 * q + 6],
                   w[8 * q + 7]);
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) *reinterpret_cast<uint4*>(dst + q * 8) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  }
}

// Out of line for attention_kernel, which calls it inside its K/V loop, where the registers are needed for the
// row of S.  A copy for each kernel: a function that kernels of different register counts share is compiled for
// one of them.
template <int kGroups, int kTileKV>
__device__ __noinline__ void attn_store_row(uint32_t o_addr, __half* dst, float inv_l) {
  attn_store_row_inline(o_addr, dst, inv_l);
}

template <int kGroups, int kTileKV>
__global__ void __launch_bounds__(AttnShape<kGroups, kTileKV>::kThreads, 1) attention_kernel(const __grid_constant__ AttnParams p) {
  using Shape = AttnShape<kGroups, kTileKV>;
  constexpr int kWarpLoad = Shape::kWarpLoad, kWarpMma = Shape::kWarpMma, kKvStages = Shape::kKvStages, kKvBytes = Shape::kKvBytes;
  constexpr int kTmemO = Shape::kTmemO, kTmemP = Shape::kTmemP;
  constexpr int kChunks = kTileKV / 32;   // a row of S in registers: chunks of 32 columns
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + Shape::kBar;
  // barriers: q_full[2], q_empty[2], kv_full[stages], kv_empty[stages], then per group s_full, o_full, p_full, s_free
  auto q_full = [&](int b) { return bar_base + 8u * b; };
  auto q_empty = [&](int b) { return bar_base + 8u * (2 + b); };
  auto kv_full = [&](int s) { return bar_base + 8u * (4 + s); };
  auto kv_empty = [&](int s) { return bar_base + 8u * (4 + kKvStages + s); };
  constexpr int kGroupBar = 4 + 2 * kKvStages;
  auto s_full = [&](int g) { return bar_base + 8u * (kGroupBar + g); };
  auto o_full = [&](int g) { return bar_base + 8u * (kGroupBar + kGroups + g); };
  auto p_full = [&](int g) { return bar_base + 8u * (kGroupBar + 2 * kGroups + g); };
  auto s_free = [&](int g) { return bar_base + 8u * (kGroupBar + 3 * kGroups + g); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + Shape::kBar + 512);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + Shape::kBar + 520);

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  constexpr uint32_t kTmemCols = 512;

  // Work units: up to `groups` query tiles of one (image, head).
  //   kv_split == 1: the CTA walks units blockIdx.x, blockIdx.x + gridDim.x, ...; barriers, the
  //     K/V ring and tensor memory live across units, Q is double buffered, so the loads and the
  //     first Q K^T of the next unit overlap the tail of the current one.
  //   kv_split == S > 1: the S CTAs of a cluster serve ONE unit, each over 1/S of the K/V tiles;
  //     their partial (max, sum, output) triples are merged through distributed shared memory at
  //     the end (every CTA merges 1/S of the rows).
  const int S = p.kv_split;
  const uint32_t crank = (S > 1) ? cluster_ctarank() : 0u;
  const int unit_rows = p.groups * kTileQ;
  const int q_units = (p.L_q + unit_rows - 1) / unit_rows;
  const int units_total = q_units * p.heads * p.B;
  const int first_unit = (S > 1) ? static_cast<int>(blockIdx.x) / S : static_cast<int>(blockIdx.x);
  const int unit_step = (S > 1) ? units_total : static_cast<int>(gridDim.x);
  auto unit_q_row0 = [&](int w) { return (w % q_units) * unit_rows; };
  auto unit_head = [&](int w) { return (w / q_units) % p.heads; };
  auto unit_img = [&](int w) { return w / (q_units * p.heads); };
  // the last unit of a head may have fewer tiles
  auto unit_groups = [&](int w) { return min(p.groups, (p.L_q - unit_q_row0(w) + kTileQ - 1) / kTileQ); };
  const int tiles_per_slot = (p.L_slot + kTileKV - 1) / kTileKV;
  const int total_tiles = p.n_slots * tiles_per_slot;
  const int tile0 = static_cast<int>((static_cast<long long>(crank) * total_tiles) / S);   // first K/V tile of this CTA
  const int n_tiles = static_cast<int>((static_cast<long long>(crank + 1) * total_tiles) / S) - tile0;
  // kv_split > 1 only: per-thread result of the K/V loop (softmax threads), kept for the merge
  uint32_t fin_o[kHeadDim];
  float fin_l = 0.f, fin_m = -INFINITY;
  bool fin_valid = false;

  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(q_full(b), 1);
      mbar_init(q_empty(b), kGroups);   // one arrival per issuer warp
    }
    for (int s = 0; s < kKvStages; ++s) {
      mbar_init(kv_full(s), 1);
      mbar_init(kv_empty(s), kGroups);
    }
    for (int g = 0; g < kGroups; ++g) {
      mbar_init(s_full(g), 1);
      mbar_init(o_full(g), 1);
      mbar_init(p_full(g), 128);
      mbar_init(s_free(g), 128);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kWarpMma) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // the softmax warps hold a row of S (kTileKV values) and of P: give them the registers the
  // producer / MMA warpgroup does not need
  pdl_wait();  // the set-up above overlaps the previous kernel's tail; global data from here on

  if (warp >= kWarpLoad) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Shape::kOtherRegs));
  if (warp == kWarpLoad) {
    // ======================= TMA producer =======================
    // all 32 lanes run the loop (addresses stay warp-uniform); the elected lane issues
    const bool leader = elect_one();
    if (leader) tma_prefetch_desc(&p.q_map);
    __syncwarp();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int ul = 0;  // units started by this CTA
    for (int w = first_unit; w < units_total && ok; w += unit_step, ++ul) {
      const int qb = ul & 1;
      const int ng = unit_groups(w);
      const int head = unit_head(w), img = unit_img(w), q_row0 = unit_q_row0(w);
      // the Q buffer was last used by unit ul - 2: all its Q K^T products must have completed
      if (ul >= 2 && !mbar_wait_warp(q_empty(qb), ((ul >> 1) - 1) & 1u, abort_flag, p.dev_status, 401)) break;
      if (leader) {
        mbar_arrive_expect_tx(q_full(qb), static_cast<uint32_t>(kQBytes) * ng);
        for (int g = 0; g < ng; ++g)
          tma_load_3d(smem_base + Shape::kQ + (qb * kGroups + g) * kQBytes, &p.q_map, q_full(qb), head * kHeadDim,
                      q_row0 + g * kTileQ, img);
      }
      __syncwarp();
      int slot = tile0 / tiles_per_slot, ts = tile0 % tiles_per_slot;
      for (int j = 0; j < n_tiles; ++j) {
        const int t0 = ts * kTileKV;
        if (!mbar_wait_warp(kv_empty(stage), phase ^ 1u, abort_flag, p.dev_status, 400)) {
          ok = false;
          break;
        }
        if (leader) {
          mbar_arrive_expect_tx(kv_full(stage), 2 * kKvBytes);
          tma_load_3d(smem_base + Shape::kK + stage * kKvBytes, &p.kv_map[slot], kv_full(stage), head * kHeadDim, t0, img);
          tma_load_3d(smem_base + Shape::kV + stage * kKvBytes, &p.kv_map[slot], kv_full(stage),
                      p.v_col0 + head * kHeadDim, t0, img);
        }
        __syncwarp();
        if (++ts == tiles_per_slot) ts = 0, ++slot;
        if (++stage == kKvStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp < kWarpMma + kGroups) {
    // ======================= MMA issuers =======================
    // One warp per query tile: its waits come true in a fixed order (S copied out, then P published), and
    // a late group holds up nobody.  All 32 lanes run the loop and the waits; the elected lane issues
    // every tcgen05.mma and tcgen05.commit, so descriptors are formed from warp-uniform values.  The K/V
    // tiles of all units of this CTA form one stream: while the softmax of tile t runs, Q K^T of tile
    // t + 1 is issued, also across a unit boundary.
    const int g = warp - kWarpMma;
    const bool leader = elect_one();
    const uint32_t idesc_s = make_idesc_f16(kTileQ, kTileKV, 0, 0);   // S = Q K^T, both K-major
    const uint32_t idesc_o = make_idesc_f16(kTileQ, kHeadDim, 0, 1);  // O = P V, V MN-major
    int n_s = 0;     // Q K^T products issued (= phases of s_full started)
    int n_pv = 0;    // P V products issued
    int st = 0;      // ring stage and phase of the stream's current tile
    uint32_t ph = 0;
    bool s_issued = false;   // Q K^T of the current tile is already under way
    bool ok = true;
    // S_g = Q_g K^T for the tile in ring stage `stage`; S_g must have been read by the softmax group if it
    // was ever written
    auto issue_s = [&](int qb, int stage, uint32_t phase) -> bool {
      if (!mbar_wait_warp(kv_full(stage), phase, abort_flag, p.dev_status, 501)) return false;
      if (n_s > 0 && !mbar_wait_warp(s_free(g), (n_s - 1) & 1u, abort_flag, p.dev_status, 503)) return false;
      tc_fence_after_sync();
      const uint64_t qdesc = make_smem_desc_sw128(smem_base + Shape::kQ + (qb * kGroups + g) * kQBytes, 16, 1024);
      const uint64_t kdesc = make_smem_desc_sw128(smem_base + Shape::kK + stage * kKvBytes, 16, 1024);
      if (leader) {
#pragma unroll
        for (int k = 0; k < kHeadDim / 16; ++k) umma_f16(tmem_base + g * kTileKV, qdesc + 2u * k, kdesc + 2u * k, idesc_s, k != 0);
        umma_commit(s_full(g));
      }
      __syncwarp();
      ++n_s;
      return true;
    };
    int ul = 0;
    for (int w = first_unit; w < units_total && ok; w += unit_step, ++ul) {
      const int qb = ul & 1;
      const bool active = g < unit_groups(w);
      const int w_next = w + unit_step;
      const bool next_active = w_next < units_total && g < unit_groups(w_next);
      if (!s_issued && !mbar_wait_warp(q_full(qb), (ul >> 1) & 1u, abort_flag, p.dev_status, 500)) {
        ok = false;
        break;
      }
      if (!active && leader) mbar_arrive(q_empty(qb));
      int ts = tile0 % tiles_per_slot;
      for (int j = 0; j < n_tiles; ++j) {
        int st_next = st + 1;
        uint32_t ph_next = ph;
        if (st_next == kKvStages) st_next = 0, ph_next ^= 1u;
        if (!active) {
          // the ring stage is released by all issuers, in step with its phases
          if (!mbar_wait_warp(kv_full(st), ph, abort_flag, p.dev_status, 504)) {
            ok = false;
            break;
          }
          if (leader) mbar_arrive(kv_empty(st));
          __syncwarp();
        } else {
          if (!s_issued && !issue_s(qb, st, ph)) {
            ok = false;
            break;
          }
          s_issued = false;
          if (j + 1 < n_tiles) {
            if (!issue_s(qb, st_next, ph_next)) {
              ok = false;
              break;
            }
            s_issued = true;
          } else {
            // every Q K^T of this unit has been issued: its Q buffer is free once they complete
            if (leader) umma_commit(q_empty(qb));
            __syncwarp();
            if (next_active) {
              if (!mbar_wait_warp(q_full(qb ^ 1), ((ul + 1) >> 1) & 1u, abort_flag, p.dev_status, 500) || !issue_s(qb ^ 1, st_next, ph_next)) {
                ok = false;
                break;
              }
              s_issued = true;
            }
          }
          // P_g of this tile is in tensor memory; O_g carries the right scale
          if (!mbar_wait_warp(p_full(g), n_pv & 1u, abort_flag, p.dev_status, 502)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          // tokens of this tile that exist (the last tile of a slot may be ragged): P is zero beyond
          // them, so their 16-token steps of the P V product are skipped
          const int k_steps = (min(kTileKV, p.L_slot - ts * kTileKV) + 15) / 16;
          // V tile [64 tokens][64] as stored: MN-major B operand, 8-token groups 1 KB apart
          const uint64_t vdesc = make_smem_desc_sw128(smem_base + Shape::kV + st * kKvBytes, 16, 1024);
          if (leader) {
#pragma unroll
            for (int k = 0; k < kTileKV / 16; ++k) {
              // tokens 16k..16k+15: 8 packed columns of P, V rows advance by 16 x 128 B
              if (k < k_steps)
                umma_f16_ts(tmem_base + kTmemO + g * kHeadDim, tmem_base + kTmemP + g * (kTileKV / 2) + 8u * k, vdesc + 128u * k, idesc_o,
                            (j != 0) | k);
            }
            umma_commit(o_full(g));
            // K and V of this tile are no longer needed by this group once everything issued so far has completed
            umma_commit(kv_empty(st));
          }
          __syncwarp();
          ++n_pv;
        }
        if (++ts == tiles_per_slot) ts = 0;
        st = st_next, ph = ph_next;
      }
    }
  }
    // producer / MMA warpgroup: the barriers of the hand-over, nothing to merge
    tc_fence_before_sync();
    __syncthreads();
    if (S > 1) {
      cluster_sync_all();
      cluster_sync_all();
    }
  } else {
    // ======================= softmax / output (warps 0..11) =======================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Shape::kSoftmaxRegs));
    const int g = warp >> 2;               // query tile served by this warp
    const int quarter = warp & 3;          // TMEM lane quarter this warp may access
    const int row = quarter * 32 + lane;   // query row inside the tile == TMEM lane
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t s_addr = t_lane + g * kTileKV;
    const uint32_t o_addr = t_lane + kTmemO + g * kHeadDim;
    const uint32_t p_addr = t_lane + kTmemP + g * (kTileKV / 2);
    const float sc = p.scale_log2e;
    constexpr float kRaise = 8.f;  // raise m only when the tile maximum exceeds it by 2^8
    int cnt = 0;                   // K/V tiles this group has processed (all units)
    bool ok = true;
    // The output of a finished unit stays in O_g while the first tile of the next unit is being
    // exponentiated; it is read out and stored just before that tile's P is published (the P V
    // product that would overwrite O_g is only issued after that).
    int pend_w = -1;             // unit whose output is still in tensor memory
    float pend_l = 1.f, pend_m = 0.f;
    // wait for the last P V product of the pending unit (tile cnt - 1), then store / keep its rows
    auto emit_pending = [&]() -> bool {
      if (!mbar_wait(o_full(g), (cnt - 1) & 1u, abort_flag, p.dev_status, 602)) return false;
      __syncwarp();
      tc_fence_after_sync();
      const int q_row = unit_q_row0(pend_w) + g * kTileQ + row;
      __half* dst = (q_row < p.L_q) ? p.out + (long long)unit_img(pend_w) * p.out_img_stride + (long long)q_row * p.ld_out +
                                          unit_head(pend_w) * kHeadDim
                                    : nullptr;
      attn_store_row<kGroups, kTileKV>(o_addr, dst, 1.f / pend_l);
      pend_w = -1;
      return true;
    };
    for (int w = first_unit; w < units_total && ok; w += unit_step) {
      if (g >= unit_groups(w)) continue;
      float m_run = -INFINITY;   // running row maximum in the exp2 domain (score * scale * log2 e)
      float l_run = 0.f;         // running row sum of P, same reference as O
      int ts = tile0 % tiles_per_slot;
      for (int j = 0; j < n_tiles && ok; ++j, ++cnt) {
        const int valid = min(kTileKV, p.L_slot - ts * kTileKV);
        if (++ts == tiles_per_slot) ts = 0;
        if (!mbar_wait(s_full(g), cnt & 1u, abort_flag, p.dev_status, 600)) {
          ok = false;
          break;
        }
        __syncwarp();
        tc_fence_after_sync();
        // the whole row of S into registers, then hand the buffer back
        uint32_t v[kChunks][32];
#pragma unroll
        for (int c = 0; c < kChunks; ++c) tmem_ld_32x32(s_addr + 32 * c, v[c]);
        tmem_ld_wait();
        tc_fence_before_sync();
        mbar_arrive(s_free(g));
        // row maximum over the valid columns
        float m_tile;
        if (valid == kTileKV) {
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
#pragma unroll
            for (int c = 0; c < kChunks; ++c) {
              float& m0 = mx[c & 1];
              float& m1 = mx[2 + (c & 1)];
              m0 = max3(m0, __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
              m1 = max3(m1, __uint_as_float(v[c][i + 2]), __uint_as_float(v[c][i + 3]));
            }
          }
          m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        } else {
          m_tile = ragged_chunk_max(v[0], valid);
#pragma unroll
          for (int c = 1; c < kChunks; ++c) m_tile = fmaxf(m_tile, ragged_chunk_max(v[c], valid - 32 * c));
        }
        const float m_new = fmaxf(m_run, m_tile * sc);
        float alpha = 1.f;
        const bool raise = kTileKV < 128 && j == 1 ? m_new > m_run : m_new > m_run + kRaise;
        if (j == 0) {
          m_run = m_new;  // O and L start from zero: nothing to rescale
        } else if (raise) {
          alpha = fast_exp2(m_run - m_new);
          m_run = m_new;
        }
        const bool rescale = __any_sync(0xffffffffu, alpha != 1.f);
        // as long as every score is -inf: P = 2^(-inf - 0) = 0, and the first finite maximum is raised to
        const float m_ref = m_run == -INFINITY ? 0.f : m_run;
        // P = exp2(S*scale - m) in fp32, summed in fp32, packed to fp16 for the tensor core:
        // two per 32-bit word
        uint32_t pa[kTileKV / 2];
        float sum = 0.f;
        if (valid == kTileKV) {
          const f32x2 sc2 = pair2(sc, sc), nm2 = pair2(-m_ref, -m_ref);
          f32x2 q[2] = {pair2(0.f, 0.f), pair2(0.f, 0.f)};
          // spread evenly over the row, so that both units stay busy
          auto on_fma = [](int k) { return (k * kPolyOf16) / 16 != ((k + 1) * kPolyOf16) / 16; };
#pragma unroll
          for (int i = 0; i < 16; ++i) {
#pragma unroll
            for (int c = 0; c < kChunks; ++c)
              pa[16 * c + i] = on_fma(kChunks * i + c) ? exp_pair<true>(v[c][2 * i], v[c][2 * i + 1], sc2, nm2, q[c & 1])
                                                       : exp_pair<false>(v[c][2 * i], v[c][2 * i + 1], sc2, nm2, q[c & 1]);
          }
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            float u0, u1;
            unpair2(q[c], u0, u1);
            sum += u0 + u1;
          }
        } else {
          // ragged last tile of a slot: columns >= valid contribute nothing
#pragma unroll
          for (int c = 0; c < kChunks; ++c) sum += ragged_chunk_p(v[c], pa, 16 * c, valid - 32 * c, sc, m_ref);
        }
        l_run = fmaf(l_run, alpha, sum);
        // the previous P V product of this group must have finished: it read the P buffer, and O
        // is only touched between two products
        if (j == 0) {
          if (pend_w >= 0 && !emit_pending()) {
            ok = false;
            break;
          }
        } else {
          if (!mbar_wait(o_full(g), (cnt - 1) & 1u, abort_flag, p.dev_status, 601)) {
            ok = false;
            break;
          }
          __syncwarp();
          tc_fence_after_sync();
          if (rescale) {
            uint32_t o0[32], o1[32];
            tmem_ld_32x32(o_addr, o0);
            tmem_ld_32x32(o_addr + 32, o1);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              o0[i] = __float_as_uint(__uint_as_float(o0[i]) * alpha);
              o1[i] = __float_as_uint(__uint_as_float(o1[i]) * alpha);
            }
            tmem_st_32x32(o_addr, o0);
            tmem_st_32x32(o_addr + 32, o1);
          }
        }
        // publish P in tensor memory
#pragma unroll
        for (int c = 0; c < kChunks / 2; ++c) tmem_st_32x32(p_addr + 32 * c, *reinterpret_cast<const uint32_t(*)[32]>(&pa[32 * c]));
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(p_full(g));
      }
      if (!ok) break;
      // a row without a finite score has the sum 0 (0 / 0 = NaN), not what poly_exp2 makes of -inf
      pend_w = w, pend_l = m_run == -INFINITY ? 0.f * l_run : l_run, pend_m = m_run;
    }
    if (ok && pend_w >= 0) {
      if (S == 1) {
        emit_pending();
      } else if (mbar_wait(o_full(g), (cnt - 1) & 1u, abort_flag, p.dev_status, 602)) {
        // kv_split > 1: keep the partial result for the merge
        __syncwarp();
        tc_fence_after_sync();
        uint32_t o0[32], o1[32];
        tmem_ld_32x32(o_addr, o0);
        tmem_ld_32x32(o_addr + 32, o1);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) fin_o[i] = o0[i], fin_o[32 + i] = o1[i];
        fin_l = pend_l;
        fin_m = pend_m;
        fin_valid = true;
      }
    }
    // ---- kv_split > 1: merge the partial results of the cluster and write the output -------
    // (the producer / MMA warps take part in the same three barriers in their own branch)
    tc_fence_before_sync();
    __syncthreads();
    if (S > 1) {
      const int w = first_unit;
      const int n_groups = unit_groups(w);
      const bool softmax_thread = (warp >> 2) < n_groups;
      const int sg = warp >> 2, srow = (warp & 3) * 32 + lane;     // group and row of a softmax thread
      const int grow = sg * kTileQ + srow;                                 // row within the unit's queries
      // every CTA of the cluster has left its K/V loop: the K/V ring of each CTA is free and serves
      // as the receive buffer  [sender][66 values][rows owned] (fp32)
      cluster_sync_all();
      const int rows_owned = unit_rows / S;
      const uint32_t owner = softmax_thread ? static_cast<uint32_t>(grow / rows_owned) : 0u;
      const int lrow = grow % rows_owned;
      const uint32_t recv = smem_base + Shape::kK;
      if (softmax_thread && owner != crank && fin_valid) {
        const uint32_t slot = (crank < owner) ? crank : crank - 1;
        const uint32_t base = map_to_cta(recv + ((slot * 66u) * rows_owned + lrow) * 4u, owner);
        const uint32_t stride = rows_owned * 4u;
  #pragma unroll
        for (int i = 0; i < kHeadDim; ++i) st_cluster_f32(base + i * stride, __uint_as_float(fin_o[i]));
        st_cluster_f32(base + 64u * stride, fin_l);
        st_cluster_f32(base + 65u * stride, fin_m);
      }
      cluster_sync_all();  // all partials have landed
      if (softmax_thread && owner == crank && fin_valid) {
        const float* rbuf = reinterpret_cast<const float*>(smem_gen + Shape::kK);
        float m_all = fin_m;
        for (int s2 = 0; s2 < S - 1; ++s2) m_all = fmaxf(m_all, rbuf[(s2 * 66 + 65) * rows_owned + lrow]);
        const float own_scale = fast_exp2(fin_m - m_all);
        float l_all = fin_l * own_scale;
        float acc[kHeadDim];
  #pragma unroll
        for (int i = 0; i < kHeadDim; ++i) acc[i] = __uint_as_float(fin_o[i]) * own_scale;
        for (int s2 = 0; s2 < S - 1; ++s2) {
          const float* rb = rbuf + (s2 * 66) * rows_owned + lrow;
          const float sc2 = fast_exp2(rb[65 * rows_owned] - m_all);
          l_all = fmaf(rb[64 * rows_owned], sc2, l_all);
  #pragma unroll
          for (int i = 0; i < kHeadDim; ++i) acc[i] = fmaf(rb[i * rows_owned], sc2, acc[i]);
        }
        const int q_row = unit_q_row0(w) + grow;
        if (q_row < p.L_q) {
          const float inv_l = 1.f / l_all;
          __half* dst = p.out + (long long)unit_img(w) * p.out_img_stride + (long long)q_row * p.ld_out + unit_head(w) * kHeadDim;
  #pragma unroll
          for (int q = 0; q < 8; ++q) {
            uint4 u;
            u.x = pack_f16x2(acc[q * 8] * inv_l, acc[q * 8 + 1] * inv_l);
            u.y = pack_f16x2(acc[q * 8 + 2] * inv_l, acc[q * 8 + 3] * inv_l);
            u.z = pack_f16x2(acc[q * 8 + 4] * inv_l, acc[q * 8 + 5] * inv_l);
            u.w = pack_f16x2(acc[q * 8 + 6] * inv_l, acc[q * 8 + 7] * inv_l);
            *reinterpret_cast<uint4*>(dst + q * 8) = u;
          }
        }
      }
    }
  }
  // ---- teardown ---------------------------------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kWarpMma) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Few keys (one slot of at most 128 tokens: cross-attention with the text).  What bounds such a call is latency:
// load, Q K^T, softmax, P V and store of a query tile follow one another.  So a CTA serves ONE query tile of one
// (image, head), and four CTAs on an SM overlap instead of a pipeline inside one.  The scores of all keys are in
// tensor memory at one time: the exact row maximum is the reference of the exponentials, nothing is rescaled, and
// the keys are read in one pass (in 64-token tiles 77 keys took two).  Measured (attention_kernel -> this one):
// 2 x 10 heads, 77 keys: 1024 queries 7.3 -> 6.4 us, 4096 13.6 -> 10.8 (21 MB: 2.0 TB/s), 16384 30.5 -> 27.0;
// 64 queries of 5 heads 4.9 -> 3.4.  The same with 256 columns and two CTAs per SM was slower than
// attention_kernel at 154 keys (16.1 -> 16.8) and 231 (19.0 -> 20.2).
//   warps 0..3  softmax: thread r owns query row r (= TMEM lane r); the row is read twice, 32 columns at a time
//   warp 4      TMA, tcgen05.mma and tensor memory
// Tensor memory, 128 columns: S [0, keys), P (two fp16 per column) over the columns of S that have been read,
// O in [64, 128) over the rest of S, written once every thread has read its row.  Shared memory is asked for in
// the proportion that these columns are of the SM's 512: CTAs that fit beside one another (of this kernel, or of
// the launch after it, which may start early) then never wait for tensor memory.
constexpr int kShortThreads = 160;
constexpr int kShortKeys = 128;
struct ShortSmem {
  static constexpr int kQ = 0, kK = kQBytes, kV = kK + kShortKeys * kHeadDim * 2, kBar = kV + kShortKeys * kHeadDim * 2;
  static constexpr int kTotal = (228 * kShortKeys / 512 - 1) * 1024;   // and 1 KB that the system takes
  static_assert(kBar + 64 + 1024 <= kTotal, "shared memory");
};

__global__ void __launch_bounds__(kShortThreads, 512 / kShortKeys) attention_short_kernel(const __grid_constant__ AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t qk_full = smem_base + ShortSmem::kBar, v_full = qk_full + 8, s_full = qk_full + 16, p_full = qk_full + 24, o_full = qk_full + 32;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + ShortSmem::kBar + 48);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + ShortSmem::kBar + 56);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(qk_full, 1);
    mbar_init(v_full, 1);
    mbar_init(s_full, 1);
    mbar_init(p_full, 128);
    mbar_init(o_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kShortKeys);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();  // not before: the next launch's CTAs must not take tensor memory that this grid still waits for
  pdl_wait();  // the set-up above overlaps the previous kernel's tail; global data from here on

  const int q_tiles = (p.L_q + kTileQ - 1) / kTileQ;
  const int q_row0 = static_cast<int>(blockIdx.x % q_tiles) * kTileQ;
  const int head = static_cast<int>(blockIdx.x / q_tiles) % p.heads, img = static_cast<int>(blockIdx.x / q_tiles) / p.heads;
  const int keys = p.L_slot;
  const int keys16 = (keys + 15) & ~15;   // rows of the K and V boxes; those past the last key arrive as zeros
  if (warp == 4) {
    const bool leader = elect_one();
    if (leader) {
      mbar_arrive_expect_tx(qk_full, static_cast<uint32_t>(kQBytes + keys16 * kHeadDim * 2));
      tma_load_3d(smem_base + ShortSmem::kQ, &p.q_map, qk_full, head * kHeadDim, q_row0, img);
      tma_load_3d(smem_base + ShortSmem::kK, &p.kv_map[0], qk_full, head * kHeadDim, 0, img);
      mbar_arrive_expect_tx(v_full, static_cast<uint32_t>(keys16 * kHeadDim * 2));
      tma_load_3d(smem_base + ShortSmem::kV, &p.kv_map[0], v_full, p.v_col0 + head * kHeadDim, 0, img);
    }
    __syncwarp();
    if (mbar_wait_warp(qk_full, 0, abort_flag, p.dev_status, 700)) {
      tc_fence_after_sync();
      const uint64_t qdesc = make_smem_desc_sw128(smem_base + ShortSmem::kQ, 16, 1024), kdesc = make_smem_desc_sw128(smem_base + ShortSmem::kK, 16, 1024);
      const uint32_t idesc = make_idesc_f16(kTileQ, keys16, 0, 0);   // S = Q K^T, both K-major
      if (leader) {
#pragma unroll
        for (int k = 0; k < kHeadDim / 16; ++k) umma_f16(tmem_base, qdesc + 2u * k, kdesc + 2u * k, idesc, k != 0);
        umma_commit(s_full);
      }
      __syncwarp();
      if (mbar_wait_warp(v_full, 0, abort_flag, p.dev_status, 701) && mbar_wait_warp(p_full, 0, abort_flag, p.dev_status, 702)) {
        tc_fence_after_sync();
        const uint64_t vdesc = make_smem_desc_sw128(smem_base + ShortSmem::kV, 16, 1024);
        const uint32_t idesc_o = make_idesc_f16(kTileQ, kHeadDim, 0, 1);  // O = P V, V MN-major
        if (leader) {
          for (int k = 0; k < keys16 / 16; ++k)
            umma_f16_ts(tmem_base + kShortKeys / 2, tmem_base + 8u * k, vdesc + 128u * k, idesc_o, k != 0);
          umma_commit(o_full);
        }
        __syncwarp();
      }
    }
  } else {
    const int row = warp * 32 + lane;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
    const float sc = p.scale_log2e;
    if (mbar_wait(s_full, 0, abort_flag, p.dev_status, 710)) {
      __syncwarp();
      tc_fence_after_sync();
      float m = -INFINITY;
      uint32_t v[32];
      for (int c = 0; c < keys; c += 32) {
        tmem_ld_32x32(t_lane + c, v);
        tmem_ld_wait();
        m = fmaxf(m, ragged_chunk_max(v, keys - c));
      }
      m *= sc;
      float l = 0.f;
      for (int c = 0; c < keys; c += 32) {
        tmem_ld_32x32(t_lane + c, v);
        tmem_ld_wait();
        uint32_t pk[16];
        l += ragged_chunk_p(v, pk, 0, keys - c, sc, m);
        tmem_st_32x16(t_lane + c / 2, pk);   // over columns of S that this thread has read
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(p_full);
      if (mbar_wait(o_full, 0, abort_flag, p.dev_status, 711)) {
        __syncwarp();
        tc_fence_after_sync();
        __half* dst = q_row0 + row < p.L_q ? p.out + (long long)img * p.out_img_stride + (long long)(q_row0 + row) * p.ld_out + head * kHeadDim : nullptr;
        attn_store_row_inline(t_lane + kShortKeys / 2, dst, 1.f / l);
      }
    }
  }
  // ---- teardown ---------------------------------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 4) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kShortKeys);
  }
}

// Test hook: poly_exp2 by itself.
__global__ void poly_exp2_kernel(const float* x, float* y, long long n) {
  const long long i = 2 * (blockIdx.x * (long long)blockDim.x + threadIdx.x);
  if (i >= n) return;
  float a, b;
  unpair2(poly_exp2(pair2(x[i], i + 1 < n ? x[i + 1] : 0.f)), a, b);
  y[i] = a;
  if (i + 1 < n) y[i + 1] = b;
}

static int g_force_attn_split = 0, g_force_attn_groups = 0, g_force_attn_keys = 0;  // test hooks: 0 = choose

// Tokens per key tile, query tiles per unit and K/V split: least rounds x time of a round.  Three groups of 64-token tiles
// keep the softmax units busiest; where a round has work for fewer query tiles than that (strips: few queries
// against the keys of all strips), two of 128 tokens spend less on each key, as one wait and one publication of P
// serve twice the keys.  A unit of fewer query tiles takes not much less time, it only fills more CTAs.  Without a
// split a CTA walks several units; with one each cluster serves one unit and merges.  The times (us per key tile by
// query tiles in it, per unit, per call) are a least-squares fit over 51 shapes (1 to 20 x 2 heads, 64 to 16384
// queries, 1 to 8 slots, 144 to 16384 keys) x 15 combinations; the choice is 0.5 % slower than the best of the 15 on
// average, 6 % at most.  2 x 20 heads: 512 queries of 2 strips 21.6 -> 18.7 us, 1208 of 4 138 -> 115, 128 of 8
// 15.9 -> 11.7; 2 x 10 heads: 512 of 8 40.4 -> 33.5 (64-token tiles alone -> both).
struct AttnPlan {
  int keys, groups, split;
  double us;
};
struct AttnCosts {
  double tile[4];        // per key tile, by query tiles
  double unit[5];        // per unit, by split
};
static constexpr AttnCosts kCosts64{{0.0, 0.685, 1.099, 1.261}, {0.0, 3.01, 4.99, 0.0, 5.56}};
static constexpr AttnCosts kCosts128{{0.0, 1.104, 1.608, 0.0}, {0.0, 2.90, 5.30, 0.0, 5.92}};

template <int kGroups, int kTileKV>
static void plan_attention(const AttnCosts& costs, int heads_b, int q_tiles, int n_slots, int L_slot, AttnPlan& best) {
  static std::atomic<int> resident[64][5] = {};
  using Shape = AttnShape<kGroups, kTileKV>;
  if (g_force_attn_keys && g_force_attn_keys != kTileKV) return;
  const int total_tiles = n_slots * ((L_slot + kTileKV - 1) / kTileKV);
  int at_once[5] = {0, sm_count(), 0, 0, 0};
  for (int w = 2; w <= 4; w *= 2) at_once[w] = resident_clusters(attention_kernel<kGroups, kTileKV>, Shape::kThreads, Shape::kTotal, w, resident);
  for (int g = 1; g <= kGroups; ++g) {
    if (g_force_attn_groups ? g != g_force_attn_groups : g > q_tiles) continue;
    const int work = ((q_tiles + g - 1) / g) * heads_b;
    for (int s2 = 1; s2 <= 4 && s2 <= total_tiles; s2 *= 2) {
      if (g_force_attn_split && s2 != g_force_attn_split) continue;
      const int rounds = (work + at_once[s2] - 1) / at_once[s2];
      const double us = 1.5 + rounds * (((total_tiles + s2 - 1) / s2) * costs.tile[g < q_tiles ? g : q_tiles] + costs.unit[s2]);
      if (best.keys == 0 || us < best.us) best = AttnPlan{kTileKV, g, s2, us};
    }
  }
}

template <int kGroups, int kTileKV>
static int launch_attention(AttnParams& p, const AttnPlan& plan, int q_tiles, cudaStream_t stream) {
  using Shape = AttnShape<kGroups, kTileKV>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (int rc = check_cuda(cudaFuncSetAttribute(attention_kernel<kGroups, kTileKV>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::kTotal),
                            "cudaFuncSetAttribute(attention)"))
      return rc;
    configured[dev] = true;
  }
  p.kv_split = plan.split, p.groups = plan.groups;
  const int work = ((q_tiles + plan.groups - 1) / plan.groups) * p.heads * p.B;
  const int grid = (plan.split == 1) ? (work < sm_count() ? work : sm_count()) : work * plan.split;
  return launch_kernel("attention_kernel launch", attention_kernel<kGroups, kTileKV>, dim3(grid), dim3(Shape::kThreads), Shape::kTotal, stream,
                       plan.split, p);
}

static int launch_short(const AttnParams& p, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (int rc = check_cuda(cudaFuncSetAttribute(attention_short_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ShortSmem::kTotal),
                            "cudaFuncSetAttribute(attention_short)"))
      return rc;
    configured[dev] = true;
  }
  const int q_tiles = (p.L_q + kTileQ - 1) / kTileQ;
  return launch_kernel("attention_short_kernel launch", attention_short_kernel, dim3(q_tiles * p.heads * p.B), dim3(kShortThreads),
                       ShortSmem::kTotal, stream, 1, p);
}

}  // namespace bxl

using namespace bxl;

extern "C" int bxl_debug_force_attn_split(int split) {
  if (split != 0 && split != 1 && split != 2 && split != 4) return fail(kErrInvalidArg, "bxl_debug_force_attn_split: 0, 1, 2 or 4");
  g_force_attn_split = split;
  return kOk;
}

extern "C" int bxl_debug_force_attn_tiles(int groups, int keys) {
  if (groups < 0 || groups > 3 || (keys != 0 && keys != 64 && keys != 128) || (keys == 128 && groups > 2))
    return fail(kErrInvalidArg, "bxl_debug_force_attn_tiles: 0..3 query tiles (2 of 128 keys), 0, 64 or 128 keys");
  g_force_attn_groups = groups, g_force_attn_keys = keys;
  return kOk;
}

extern "C" int bxl_debug_exp2_f32(const float* x, float* y, long long n, void* stream) {
  if (!x || !y || n <= 0) return fail(kErrInvalidArg, "bxl_debug_exp2_f32: bad argument");
  poly_exp2_kernel<<<(unsigned)((n + 511) / 512), 256, 0, (cudaStream_t)stream>>>(x, y, n);
  return check_cuda(cudaGetLastError(), "poly_exp2_kernel launch");
}

extern "C" int bxl_attn_fwd_f16(const void* q, long long q_img_stride, long long ld_q, const void* const* kv_slots,
                                int n_slots, long long kv_img_stride, long long ld_kv, int v_col0, void* out,
                                long long out_img_stride, long long ld_out, int B, int heads, int L_q, int L_slot,
                                float scale, void* stream) {
  if (!q || !kv_slots || !out) return fail(kErrInvalidArg, "bxl_attn_fwd_f16: null pointer");
  if (n_slots < 1 || n_slots > kMaxSlots) return fail(kErrInvalidArg, "bxl_attn_fwd_f16: n_slots=%d (1..%d)", n_slots, kMaxSlots);
  if (B <= 0 || heads <= 0 || L_q <= 0 || L_slot <= 0) return fail(kErrInvalidArg, "bxl_attn_fwd_f16: non-positive extent");
  if (ld_q % 8 || ld_kv % 8 || ld_out % 8 || q_img_stride % 8 || kv_img_stride % 8 || out_img_stride % 8 || v_col0 % 8)
    return fail(kErrInvalidArg, "bxl_attn_fwd_f16: strides must be multiples of 8 elements");
  if (ld_q < heads * kHeadDim || ld_out < heads * kHeadDim || ld_kv < v_col0 + heads * kHeadDim || v_col0 < heads * kHeadDim)
    return fail(kErrInvalidArg, "bxl_attn_fwd_f16: row strides too small for %d heads of 64", heads);
  if ((reinterpret_cast<uintptr_t>(q) & 15u) || (reinterpret_cast<uintptr_t>(out) & 15u))
    return fail(kErrInvalidArg, "bxl_attn_fwd_f16: q/out must be 16-byte aligned");
  int* st = device_status_ptr();
  if (!st) return fail(kErrCuda, "bxl_attn_fwd_f16: no device status word");
  AttnParams p;
  memset(&p, 0, sizeof(p));
  {
    uint64_t dims[3] = {(uint64_t)(heads * kHeadDim), (uint64_t)L_q, (uint64_t)B};
    uint64_t str[2] = {(uint64_t)ld_q * 2, (uint64_t)q_img_stride * 2};
    uint32_t box[3] = {kHeadDim, kTileQ, 1};
    if (int rc = encode_tmap_f16(&p.q_map, q, 3, dims, str, box)) return rc;
  }
  // attention_short_kernel is the faster one at every measured size that it serves; a forced plan means the other
  const bool few_keys = n_slots == 1 && L_slot <= kShortKeys && !g_force_attn_split && !g_force_attn_groups && !g_force_attn_keys;
  const int q_tiles = (L_q + kTileQ - 1) / kTileQ;
  AttnPlan plan{0, 0, 0, 0.0};
  if (!few_keys) {
    plan_attention<3, 64>(kCosts64, heads * B, q_tiles, n_slots, L_slot, plan);
    plan_attention<2, 128>(kCosts128, heads * B, q_tiles, n_slots, L_slot, plan);
    if (plan.keys == 0 && !g_force_attn_groups && !g_force_attn_keys) plan = AttnPlan{64, q_tiles < 3 ? q_tiles : 3, 1, 0.0};   // more splits forced than key tiles
    if (plan.keys == 0) return fail(kErrInvalidArg, "bxl_attn_fwd_f16: the forced tiles and split do not fit %d slots of %d keys", n_slots, L_slot);
  }
  for (int s = 0; s < (few_keys ? 1 : kMaxSlots); ++s) {
    const void* base = kv_slots[s < n_slots ? s : 0];
    if (!base) return fail(kErrInvalidArg, "bxl_attn_fwd_f16: slot %d null", s);
    uint64_t dims[3] = {(uint64_t)(v_col0 + heads * kHeadDim), (uint64_t)L_slot, (uint64_t)B};
    uint64_t str[2] = {(uint64_t)ld_kv * 2, (uint64_t)kv_img_stride * 2};
    uint32_t box[3] = {kHeadDim, (uint32_t)(few_keys ? (L_slot + 15) / 16 * 16 : plan.keys), 1};
    if (int rc = encode_tmap_f16(&p.kv_map[s], base, 3, dims, str, box)) return rc;
  }
  p.n_slots = n_slots, p.L_q = L_q, p.L_slot = L_slot, p.heads = heads, p.B = B, p.v_col0 = v_col0;
  p.out = static_cast<__half*>(out);
  p.out_img_stride = out_img_stride, p.ld_out = ld_out;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.dev_status = st;
  if (few_keys) return launch_short(p, (cudaStream_t)stream);
  return plan.keys == 128 ? launch_attention<2, 128>(p, plan, q_tiles, (cudaStream_t)stream)
                          : launch_attention<3, 64>(p, plan, q_tiles, (cudaStream_t)stream);
}
