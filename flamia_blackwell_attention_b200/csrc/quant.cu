// Fused block-scaled quantiser (token-block MXFP8, optional NVFP4 S-operand copy, optional Hadamard rotation) and the
// fused backward prologue (D = rowsum(O * dequant(dO)), shifted log2 LSE, zeroed f16 dQ accumulator).
//
// Replaces the reference's quantize_fp8_blocks launch (flash_attn/cute/quant/fp8.py:2512, kernel_stream :1639; its input
// staging :262-300) and the fused NVFP4 copy (flash_attn/cute/quant/_fp8_nvfp4.py:121-158). Outputs are byte-identical to
// the reference's eager definitions (tests/cute/quant_reference.py:714-798, 270-369).
//
// Persistent CTAs walk the (128-token tile, head) pairs of the tensor, heads fastest, so the CTAs running at any moment read one
// contiguous stretch of the (b, s, h, d) input. Each CTA keeps STAGES tiles in flight: one thread
// issues the TMA loads of tile t + STAGES (plain cp.async.bulk.tensor, never multicast) as soon as every thread has read
// tile t out of its stage, so the memory system stays busy while the butterflies and conversions of the current tile run.
// Four lanes share a token row: lane q of the row holds the 16-byte chunks c = 4 j + q (8 elements each); element index
// i = 32 j + 8 q + e, so the Hadamard levels 1, 2, 4 and 32, 64 are in-thread and levels 8, 16 are two lane exchanges:
// the same order of operations as a one-thread-per-row butterfly, hence the same bits. The butterflies run as packed
// f32x2 instructions on register pairs (chunk j, chunk j + 2): one issue slot per two additions, same rounding.
// Bound: HBM (2 B read + 1 B written per element, plus the optional copies).
#include "doc_work.cuh"
#include "flamia_internal.h"

namespace fl {

static constexpr int QT = 128;        // tokens per tile
static constexpr int QSTAGES = 3;
// Threads (four lanes per token) and with them the steps of a tile: one of 512 threads, or in the prologue also two of 256. Its two
// input tiles and 127 registers a thread leave room for one block of 512 threads an SM, which waits for itself at every tile's
// barriers; two of 256 cover each other (prologue_steps() says when).
constexpr int q_threads(int steps) { return 512 / steps; }
constexpr int q_blocks(bool pro, int steps) { return pro && steps == 1 ? 1 : 2; }      // an SM

struct QuantParams {
  const float* lse;       // (b, h, s) or null
  uint8_t* codes;         // (b, s, h, d)
  uint8_t* codes_t;       // (b, h, d, s) or null
  uint8_t* e_tab;         // (b, h, s/32, d/32) or null
  float* fac;             // (b, h, s/32) or null
  uint8_t* sf_tok;        // (b, h, s/128, 512) or null
  uint8_t* sf_dim;        // (b, h, s/128, 512) or null
  float* token_factors;   // (b, h, s) or null
  uint8_t* x4;            // (b, s, h, d/2) or null
  uint8_t* sf4;           // (b, h, s/128, d/64, 512) or null
  float* d_out;           // (b, h, s) or null
  float* lse_log2;        // (b, h, s) or null
  uint16_t* zero_acc;     // f16 accumulator of b * h * s * d elements or null
  float* tile_stats;      // (b, h, s/128, 2): [amax of the values quantised, max row sum of squares] or null
  uint32_t* row_stat;     // (b, s) per-token maximum over the heads (float bits, zero on entry) or null
  int row_stat_kind;      // 1 = sum of squares, 2 = largest magnitude, 3 = 2-norm
  int o_packed;           // packed source: the forward output o has the packed rows of x (else the outputs' rows)
  int b, s, h;
  const int32_t* slot_src;   // packed source: first source row of each 128-row slot of the output (-1: an empty slot), or null
  const int32_t* slot_rows;  // packed source: valid rows of each slot (the rest of the slot reads as zero)
  int n_tiles;            // b * (s / 128) * h
  int skip_padding;       // host only: mostly_padding
  int token_local, d_per_factor;
  int in_f16;
  float lse_shift, d_multiplier;
  DevCtl ctl;
};

__device__ __forceinline__ float flush_sub(float v) { return fabsf(v) < 1.17549435e-38f ? v * 0.0f : v; }
// packed pairs: a + b, a - b, and a * b with subnormal inputs and results flushed to zero (the product and its flush in
// one instruction); each half rounds exactly as the scalar instruction does
__device__ __forceinline__ uint64_t mul2_ftz(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// UE8M0 round-up selector: smallest e with 448 * 2^e >= amax; byte 0 when fp32(amax * fp32(1/448)) is subnormal / zero
__device__ __forceinline__ uint32_t ue8m0_byte(float amax) {
  float r = __fmul_rn(amax, 1.0f / 448.0f);
  if (!(r >= 1.17549435e-38f)) return 0;
  uint32_t bits = __float_as_uint(amax);
  uint32_t E = bits >> 23, man = bits & 0x7FFFFF;
  return man <= 0x600000 ? E - 8 : E - 7;   // 448 = 1.75 * 2^8
}
__device__ __forceinline__ float pow2_from_field(int field) { return __uint_as_float((uint32_t)field << 23); }

// two E4M3 codes (low byte first) -> their exact values
__device__ __forceinline__ float2 e4m3x2_to_f32(uint16_t v) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(v));
  return __half22float2(*reinterpret_cast<const __half2*>(&h2));
}

// MODE bits: 1 = the E4M3 codes are of the rotated rows, 2 = also write the NVFP4 copy, 4 = rotate only the NVFP4 copy
// PK: packed source (slot tables); a template flag, so that the batched form pays nothing for it. 2: a warp whose rows lie past the slot's
// document writes zeros and does nothing else (mostly_padding says where).
template <int D, int MODE, bool PRO, int STEPS, int PK>
__global__ void __launch_bounds__(q_threads(STEPS), q_blocks(PRO, STEPS))
quant_blocks_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_o,
                    const QuantParams p) {
  constexpr bool ROT = (MODE & 1) != 0, NV4 = (MODE & 2) != 0, ROT4 = (MODE & 4) != 0;
  constexpr int NJ = D / 32;                     // 16-byte chunks per lane
  constexpr int NE = 8 * NJ;                     // elements per lane
  constexpr int QTHREADS = q_threads(STEPS), ROWS = QT / STEPS;     // tokens of a step
  constexpr int TILE_B = ROWS * D * 2;           // bytes of one 16-bit input tile (of a step)
  constexpr int STAGE_B = PRO ? 2 * TILE_B : TILE_B;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_codes = smem + QSTAGES * STAGE_B;   // channel-major copy only (present when codes_t is asked for)
  __shared__ __align__(8) uint64_t full[QSTAGES];
  // per-warp (8 rows) maximum and largest row sum of squares, by step: a tile's last step reads those of both, while a warp
  // that is ahead may write the next one's
  __shared__ float s_wmax[4][QTHREADS / 32], s_wsq[4][QTHREADS / 32];
  __shared__ __align__(16) uint32_t s_sign[4][4][4];   // [lane of the row][chunk][word]: sign bits of the rotation
  __shared__ int abort_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // lane -> (row of the warp's eight, lane of the row). The two rows of a quarter warp differ in bit 2, so that with
  // the 128-byte swizzle their 16-byte chunks fall into different bank groups (conflict-free 128-bit loads).
  const int q = lane & 3;
  const int rs = warp * 8 + ((lane >> 2) & 1) * 4 + (lane >> 3);     // token row of the step
  const int G = gridDim.x;
  const int ntile = p.s / QT;
  volatile int* abortp = &abort_s;

  auto issue = [&](int n) {                      // one thread: the loads of this block's step n
    const int L = blockIdx.x + n / STEPS * G, half = n % STEPS * ROWS, st = n % QSTAGES;
    if (L >= p.n_tiles) return;
    const int head = L % p.h, tile = (L / p.h) % ntile, bat = L / (p.h * ntile);
    uint8_t* dst = smem + st * STAGE_B;
    // packed source (documents stored back to back): the slot's rows start at an arbitrary row of the (1, total, h, d)
    // tensor; only the innermost TMA coordinate has an alignment rule. An empty slot loads nothing of x.
    int xrow = PK ? p.slot_src[tile] : tile * QT;
    if (!PK || xrow >= 0) xrow += half;
    mbar_arrive_expect_tx(&full[st], (xrow >= 0 ? TILE_B : 0) + ((PRO && (xrow >= 0 || !(PK && p.o_packed))) ? TILE_B : 0));
    if (xrow >= 0) {
      tma_load_4d(dst, &tm_x, &full[st], 0, head, xrow, bat);
      if (D == 128) tma_load_4d(dst + TILE_B / 2, &tm_x, &full[st], 64, head, xrow, bat);
    }
    if (PRO) {
      // (packed source: the forward output has the packed rows too; an empty slot's stage keeps what it held, and its
      // rows read as zero below)
      const int orow = (PK && p.o_packed) ? xrow : tile * QT + half;
      if (orow >= 0) {
        tma_load_4d(dst + TILE_B, &tm_o, &full[st], 0, head, orow, bat);
        if (D == 128) tma_load_4d(dst + TILE_B + TILE_B / 2, &tm_o, &full[st], 64, head, orow, bat);
      }
    }
  };
  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < QSTAGES; ++i) mbar_init(&full[i], 1);
    fence_barrier_init();
    tma_prefetch_desc(&tm_x);
    if (PRO) tma_prefetch_desc(&tm_o);
    grid_dependency();
    for (int n = 0; n < QSTAGES; ++n) issue(n);
  }
  if ((ROT || ROT4) && tid < 16) {               // sign words: bit 15 / 31 of word k = sign of element 2 k / 2 k + 1
    constexpr uint32_t NEG[4] = {0x10D2E03Eu, 0xE0D9F0E2u, 0x45809F07u, 0x75954FEDu};
    const int qq = tid >> 2, j = tid & 3;
    const uint32_t m = (NEG[j] >> (8 * qq)) & 0xFF;
#pragma unroll
    for (int k = 0; k < 4; ++k) s_sign[qq][j][k] = (((m >> (2 * k)) & 1) << 15) | (((m >> (2 * k + 1)) & 1) << 31);
  }
  __syncthreads();
  grid_dependency();

  // raw 16-byte chunk j of this thread's row (global chunk 4 j + q) from a staged tile
  bool row_live = true;                          // packed source: false for the rows of a slot past its document's end
  auto lds_chunk = [&](uint32_t tile_addr, int j) -> uint4 {
    const int g = 4 * j + q;
    const uint32_t box = (D == 128) ? (uint32_t)(g >> 3) * (TILE_B / 2) : 0u;
    return lds_u4(tile_addr + box + rs * 128 + (((g & 7) ^ (rs & 7)) << 4));
  };
  // the same for a chunk of x: rows that do not belong to the slot's document (or an empty slot, whose stage holds
  // whatever was there) read as zero
  auto lds_chunk_x = [&](uint32_t tile_addr, int j) -> uint4 {
    uint4 v = lds_chunk(tile_addr, j);
    if (PK && !row_live) v = make_uint4(0, 0, 0, 0);
    return v;
  };
  auto to_f32 = [&](const uint4& v, float* dst) {      // 8 elements of one chunk
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    if (p.in_f16) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
        dst[2 * k] = f.x;
        dst[2 * k + 1] = f.y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        dst[2 * k] = __uint_as_float(w[k] << 16);
        dst[2 * k + 1] = __uint_as_float(w[k] & 0xFFFF0000u);
      }
    }
  };
  // (y * signs) H_128 / sqrt(128): butterfly levels 1, 2, ..., 64 with (a, b) -> (a + b, a - b), then the scaling with
  // subnormal results flushed. Reads the staged tile, leaves the rotated row in y.
  auto load_rotated = [&](uint32_t tile_addr, float* y) {
    if constexpr (D == 128) {
      float t[32];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint4 v = lds_chunk_x(tile_addr, j);
        const uint4 sg = *reinterpret_cast<const uint4*>(&s_sign[q][j][0]);
        v.x ^= sg.x; v.y ^= sg.y; v.z ^= sg.z; v.w ^= sg.w;
        to_f32(v, t + 8 * j);
      }
      uint64_t Y[16];                              // Y[8 jp + e] = (element (jp, e), element (jp + 2, e))
#pragma unroll
      for (int k = 0; k < 16; ++k) Y[k] = pack2(t[k], t[k + 16]);
#pragma unroll
      for (int hs = 1; hs < 8; hs <<= 1) {         // element bits 0..2: inside one chunk
#pragma unroll
        for (int k = 0; k < 16; ++k)
          if ((k & hs) == 0) {
            const uint64_t a = Y[k], b2 = Y[k + hs];
            Y[k] = add2(a, b2);
            Y[k + hs] = sub2(a, b2);
          }
      }
#pragma unroll
      for (int lb = 1; lb < 4; lb <<= 1) {         // element bits 3, 4 = the lane of the row
        // low lane: y + other; high lane: other - y. Both are other + (+-1) y: one fma (the product is exact)
        const float sg = (q & lb) ? -1.0f : 1.0f;
        const uint64_t sg2 = pack2(sg, sg);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          float lo, hi;
          unpack2(Y[k], lo, hi);
          const uint64_t other = pack2(__shfl_xor_sync(0xFFFFFFFFu, lo, lb), __shfl_xor_sync(0xFFFFFFFFu, hi, lb));
          Y[k] = fma2(Y[k], sg2, other);
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {                // element bit 5 = chunk bit 0
        const uint64_t a = Y[k], b2 = Y[k + 8];
        Y[k] = add2(a, b2);
        Y[k + 8] = sub2(a, b2);
      }
      const uint64_t c2 = pack2(0.08838834764831845f, 0.08838834764831845f);
#pragma unroll
      for (int k = 0; k < 16; ++k) {               // element bit 6 = chunk bit 1: the two halves of a pair
        float lo, hi;
        unpack2(Y[k], lo, hi);
        const uint64_t s2 = mul2_ftz(pack2(__fadd_rn(lo, hi), __fsub_rn(lo, hi)), c2);   // scaled and flushed
        unpack2(s2, y[k], y[k + 16]);
      }
    }
  };
  auto load_plain = [&](uint32_t tile_addr, float* y) {
#pragma unroll
    for (int j = 0; j < NJ; ++j) to_f32(lds_chunk_x(tile_addr, j), y + 8 * j);
  };

  int it = 0;                                    // steps so far
  for (int L = blockIdx.x; L < p.n_tiles; it % STEPS == STEPS - 1 ? L += G : 0, ++it) {
    const int st = it % QSTAGES, par = it & 3, step = it % STEPS;
    const bool whole = step == STEPS - 1;          // with this step the tile's maxima are complete
    const int r = step * ROWS + rs;                // token row of the tile
    const int head = L % p.h, tile = (L / p.h) % ntile, bat = L / (p.h * ntile);
    const int t0 = tile * QT;
    const size_t row_off = (((size_t)bat * p.s + t0 + r) * p.h + head) * D;     // this row in a (b, s, h, D) tensor
    const size_t bh = (size_t)bat * p.h + head;
    const size_t ri = bh * p.s + t0 + r;
    const uint32_t tile_addr = smem_u32(smem + st * STAGE_B);
    // before the wait, which covers the loads (the LSE in the prologue alone: b2 s8192 h32 token scales 42.0 -> 41.0 us)
    const float lse_row = PRO && q == 0 && p.lse && p.lse_log2 ? p.lse[ri] : 0.f;
    const int live_rows = PK ? p.slot_rows[tile] : QT;
    bool ok = mbar_wait(&full[st], (it / QSTAGES) & 1, p.ctl, abortp, 50);
    if (PK) row_live = r < live_rows;
    const bool work = PK != 2 || step * ROWS + warp * 8 < live_rows;

    if (p.zero_acc) {   // this tile's share of the accumulator: 128 * D f16 = 32 D 16-byte chunks, contiguous
      uint4* z = reinterpret_cast<uint4*>(p.zero_acc + (bh * p.s + t0 + step * ROWS) * D);
      const uint4 zero = make_uint4(0, 0, 0, 0);
      for (int i = tid; i < ROWS * D / 8; i += QTHREADS) z[i] = zero;
    }

    // NVFP4 copy of y: per 16 along d (two neighbouring lanes): SF = E4M3_rn(amax * f32(1/6)); codes = E2M1_rn(ftz(y * m)),
    // m = 1 / SF | +inf (SF rounds to 0, amax > 0) | 0
    auto nvfp4_row = [&](const float* y) {
      uint32_t sfpack = 0;                         // this lane's scale bytes: chunk j in byte j
      uint8_t* x4row = p.x4 + row_off / 2;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        float am = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float a = fabsf(flush_sub(y[8 * j + e]));
          am = (a > am) ? a : am;                  // a NaN never wins
        }
        const float oth = __shfl_xor_sync(0xFFFFFFFFu, am, 1);
        am = (oth > am) ? oth : am;
        const float u = __fmul_rn(am, 1.0f / 6.0f);
        const uint32_t sfb = cvt_e4m3x2(u, 0.f) & 0xFF;
        const float sfv = e4m3x2_to_f32((uint16_t)sfb).x;
        const float m = sfv > 0.f ? __frcp_rn(sfv) : (u > 0.f ? __int_as_float(0x7F800000) : 0.f);
        uint32_t packed = 0;
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          const float a0 = flush_sub(__fmul_rn(flush_sub(y[8 * j + e]), m));
          const float a1 = flush_sub(__fmul_rn(flush_sub(y[8 * j + e + 1]), m));
          uint16_t c2;
          asm("{\n\t.reg .b8 t;\n\tcvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\n\tcvt.u16.u8 %0, t;\n\t}" : "=h"(c2) : "f"(a1), "f"(a0));
          packed |= (uint32_t)(c2 & 0xFF) << (e * 4);
        }
        *reinterpret_cast<uint32_t*>(x4row + (4 * j + q) * 4) = packed;
        sfpack |= sfb << (8 * j);
      }
      // group g = 2 j + (q >> 1): atom g / 4 = j / 2, byte g % 4 = 2 (j & 1) + (q >> 1); lane 0 of the row assembles
      const uint32_t hi = __shfl_down_sync(0xFFFFFFFFu, sfpack, 2);
      if (p.sf4 && q == 0) {
        uint8_t* atom = p.sf4 + ((bh * ntile + tile) * (D / 64)) * 512;
#pragma unroll
        for (int a = 0; a < D / 64; ++a) {
          const uint32_t lo0 = (sfpack >> (16 * a)) & 0xFF, lo1 = (sfpack >> (16 * a + 8)) & 0xFF;
          const uint32_t hi0 = (hi >> (16 * a)) & 0xFF, hi1 = (hi >> (16 * a + 8)) & 0xFF;
          *reinterpret_cast<uint32_t*>(atom + a * 512 + (r & 31) * 16 + (r >> 5) * 4) = lo0 | (hi0 << 8) | (lo1 << 16) | (hi1 << 24);
        }
      }
    };

    float x[NE];
    if (!work) {         // (the prologue alone: no rotation, no NVFP4 copy)
#pragma unroll
      for (int i = 0; i < NE; ++i) x[i] = 0.f;
    } else if (ROT4) {          // NVFP4 codes of the rotated row, E4M3 codes of the row as read
      load_rotated(tile_addr, x);
      nvfp4_row(x);
      load_plain(tile_addr, x);
    } else if (ROT) {
      load_rotated(tile_addr, x);
      if (NV4) nvfp4_row(x);
    } else {
      load_plain(tile_addr, x);
      if (NV4) nvfp4_row(x);
    }
    uint4 o_raw[NJ];     // prologue: the forward output's row, kept as read until the codes exist
    if (PRO) {
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        o_raw[j] = make_uint4(0, 0, 0, 0);
        if (work && !(PK && p.o_packed && !row_live)) o_raw[j] = lds_chunk(tile_addr + TILE_B, j);
      }
    }

    // ---- exponents: per token (4 lanes) and per 32-token block (4 warps)
    float amax = 0.f, sumsq = 0.f;
    if (!ROT || ROT4) {  // subnormal -> zero of the same sign (rotated rows were flushed by their scaling)
#pragma unroll
      for (int i = 0; i < NE; i += 2) {
        const uint64_t f2 = mul2_ftz(pack2(x[i], x[i + 1]), pack2(1.0f, 1.0f));
        unpack2(f2, x[i], x[i + 1]);
      }
    }
#pragma unroll
    for (int i = 0; i < NE; i += 2) amax = fmaxf(fmaxf(amax, fabsf(x[i])), fabsf(x[i + 1]));
    if (p.tile_stats || p.row_stat) {     // the row norm is only wanted with the statistics (K, V, dO)
      float sq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < NE; ++i) sq[i & 3] = fmaf(x[i], x[i], sq[i & 3]);
      sumsq = (sq[0] + sq[1]) + (sq[2] + sq[3]);
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));      // the token's maximum
    sumsq += __shfl_xor_sync(0xFFFFFFFFu, sumsq, 1);
    sumsq += __shfl_xor_sync(0xFFFFFFFFu, sumsq, 2);
    if (p.row_stat && q == 0 && (!PK || row_live)) {     // non-negative floats order as their bit patterns
      const float v = p.row_stat_kind == 2 ? amax : (p.row_stat_kind == 3 ? __fsqrt_rn(sumsq) : sumsq);
      atomicMax(p.row_stat + (size_t)bat * p.s + t0 + r, __float_as_uint(v));
    }
    float wmax = amax, wsq = sumsq;
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      wmax = fmaxf(wmax, __shfl_xor_sync(0xFFFFFFFFu, wmax, o));
      wsq = fmaxf(wsq, __shfl_xor_sync(0xFFFFFFFFu, wsq, o));
    }
    if (lane == 0) { s_wmax[par][warp] = wmax; s_wsq[par][warp] = wsq; }
    // every thread has read the stage: it can take tile it + STAGES. A wait that ran out leaves the loop here, all
    // threads together.
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    if (!ok) break;
    if (tid == 0) issue(it + QSTAGES);

    // the maximum of 32-token block b of the tile (of this step's or, in the last step, any)
    auto block_max = [&](int b) -> float {
      const float* wm = s_wmax[(it - step + b * 32 / ROWS) & 3] + b * 4 % (QTHREADS / 32);
      return fmaxf(fmaxf(wm[0], wm[1]), fmaxf(wm[2], wm[3]));
    };
    const int blk = r >> 5;                                         // this row's
    const float bmax = block_max(blk);
    const uint32_t bbyte = ue8m0_byte(bmax);
    const bool tl = p.token_local != 0;
    const uint32_t tbyte = tl ? ue8m0_byte(amax) : bbyte;
    const float inv = tbyte ? pow2_from_field(254 - (int)tbyte) : 0.f;
    const float scale = tbyte ? pow2_from_field((int)tbyte) : 0.f;

    uint32_t cw[2 * NJ];
    {
      const uint64_t inv2 = pack2(inv, inv);
#pragma unroll
      for (int i = 0; i < 2 * NJ; ++i) {
        float a0, a1, a2, a3;
        unpack2(mul2(pack2(x[4 * i], x[4 * i + 1]), inv2), a0, a1);
        unpack2(mul2(pack2(x[4 * i + 2], x[4 * i + 3]), inv2), a2, a3);
        cw[i] = cvt_e4m3x4(a0, a1, a2, a3);
      }
      uint8_t* crow = p.codes + row_off;
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        *reinterpret_cast<uint2*>(crow + (4 * j + q) * 8) = make_uint2(cw[2 * j], cw[2 * j + 1]);
    }

    // ---- prologue: D in the fixed tree order (column bits 1 (fma), 2, 3, 0, 6, 5, 4), shifted log2 LSE
    if (PRO && !work) {
      if (q == 0 && p.d_out) p.d_out[ri] = __fmul_rn(0.f, p.d_multiplier);
    } else if (PRO) {
      float o[NE];
#pragma unroll
      for (int j = 0; j < NJ; ++j) to_f32(o_raw[j], o + 8 * j);
      float v[4 * NJ];                               // columns with bit 1 clear: index (j, e bit 2, e bit 0)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        // the chunk's eight codes back as floats: the hardware conversion E4M3 -> f16 is exact (two codes per instruction)
        float c8[8];
#pragma unroll
        for (int hw = 0; hw < 4; ++hw) {
          const float2 f = e4m3x2_to_f32((uint16_t)(cw[2 * j + (hw >> 1)] >> (16 * (hw & 1))));
          c8[2 * hw] = f.x;
          c8[2 * hw + 1] = f.y;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int e = ((k >> 1) << 2) | (k & 1);   // 0, 1, 4, 5
          const float a0 = __fmul_rn(c8[e], scale);
          const float a2 = __fmul_rn(c8[e + 2], scale);
          v[4 * j + k] = __fmaf_rn(a0, o[8 * j + e], __fmul_rn(a2, o[8 * j + e + 2]));
        }
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {                 // bit 2
        v[4 * j + 0] = __fadd_rn(v[4 * j + 0], v[4 * j + 2]);
        v[4 * j + 1] = __fadd_rn(v[4 * j + 1], v[4 * j + 3]);
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {                 // bit 3 = lane bit 0
        v[4 * j + 0] = __fadd_rn(v[4 * j + 0], __shfl_xor_sync(0xFFFFFFFFu, v[4 * j + 0], 1));
        v[4 * j + 1] = __fadd_rn(v[4 * j + 1], __shfl_xor_sync(0xFFFFFFFFu, v[4 * j + 1], 1));
      }
      float w4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w4[j] = j < NJ ? __fadd_rn(v[4 * (j < NJ ? j : 0) + 0], v[4 * (j < NJ ? j : 0) + 1]) : 0.f;   // bit 0
      const float w2a = __fadd_rn(w4[0], w4[2]), w2b = __fadd_rn(w4[1], w4[3]);                  // bit 6
      float w1 = __fadd_rn(w2a, w2b);                                                            // bit 5
      w1 = __fadd_rn(w1, __shfl_xor_sync(0xFFFFFFFFu, w1, 2));                                   // bit 4 = lane bit 1
      w1 = __fmul_rn(w1, p.d_multiplier);
      if (q == 0 && p.d_out) p.d_out[ri] = p.d_per_factor ? __fmul_rn(w1, inv) : w1;     // (a power of two: exact)
    }
    if (p.lse && p.lse_log2 && q == 0) {
      const float l = PRO ? lse_row : p.lse[ri];
      p.lse_log2[ri] = __fsub_rn((l == -INFINITY) ? 0.f : __fmul_rn(l, 1.4426950408889634f), p.lse_shift);
    }

    // ---- side tables
    if ((tid & 127) == 0 && p.e_tab) {               // one thread per 32-token block (tid 128 k: row 32 k, lane 0 of it)
      uint8_t* e = p.e_tab + (bh * (p.s / 32) + tile * 4 + blk) * (D / 32);
#pragma unroll
      for (int g = 0; g < D / 32; ++g) e[g] = (uint8_t)bbyte;
    }
    // factors: in the prologue's one-step form by the thread that holds the block's exponent (d = 64: 13.6 -> 13.1 us at 8 x 1024 x 12
    // heads), else by the tile's first four threads
    constexpr bool OWN_FAC = PRO && STEPS == 1;
    uint32_t b0 = 0, b1 = 0, b2 = 0, b3 = 0;         // the tile's four exponents
    if (OWN_FAC || (whole && (tid < 4 || p.sf_dim))) {
      b0 = ue8m0_byte(block_max(0));
      b1 = ue8m0_byte(block_max(1));
      b2 = ue8m0_byte(block_max(2));
      b3 = ue8m0_byte(block_max(3));
    }
    if ((OWN_FAC ? (tid & 127) == 0 : whole && tid < 4) && p.fac) {
      const uint32_t tm = max(max(b0, b1), max(b2, b3)), own = OWN_FAC ? bbyte : tid == 0 ? b0 : tid == 1 ? b1 : tid == 2 ? b2 : b3;
      const uint32_t e0 = own ? own : tm;
      p.fac[bh * (p.s / 32) + tile * 4 + (OWN_FAC ? blk : tid)] = e0 ? pow2_from_field((int)e0) : 1.0f;
    }
    if (q == 0) {
      if (p.token_factors) p.token_factors[ri] = tbyte ? scale : 1.0f;
      if (p.sf_tok)
        *reinterpret_cast<uint32_t*>(p.sf_tok + (bh * ntile + tile) * 512 + (r & 31) * 16 + (r >> 5) * 4) = tbyte * 0x01010101u;
    }
    if (whole && p.sf_dim && tid < 128)
      *reinterpret_cast<uint32_t*>(p.sf_dim + (bh * ntile + tile) * 512 + tid * 4) = b0 | (b1 << 8) | (b2 << 16) | (b3 << 24);
    if (whole && p.tile_stats && tid == 0) {
      float a = 0.f, sq = 0.f;
#pragma unroll
      for (int w = 0; w < 16; ++w) {
        const int at = (it - step + w * 8 / ROWS) & 3, ws = w % (QTHREADS / 32);
        a = fmaxf(a, s_wmax[at][ws]);
        sq = fmaxf(sq, s_wsq[at][ws]);
      }
      p.tile_stats[(bh * ntile + tile) * 2] = a;
      p.tile_stats[(bh * ntile + tile) * 2 + 1] = sq;
    }

    // ---- channel-major copy (b, h, d, s): through shared memory, thread c gathers column c
    if (p.codes_t) {
      constexpr int CROWB = D + 16;
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        *reinterpret_cast<uint2*>(s_codes + r * CROWB + (4 * j + q) * 8) = make_uint2(cw[2 * j], cw[2 * j + 1]);
      if (!whole) continue;
      __syncthreads();
      for (int i = tid; i < D * 8; i += QTHREADS) {  // (channel, 16-token group)
        const int c = i >> 3, rg = (i & 7) * 16;
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          w[k] = (uint32_t)s_codes[(rg + 4 * k) * CROWB + c] | ((uint32_t)s_codes[(rg + 4 * k + 1) * CROWB + c] << 8) |
                 ((uint32_t)s_codes[(rg + 4 * k + 2) * CROWB + c] << 16) | ((uint32_t)s_codes[(rg + 4 * k + 3) * CROWB + c] << 24);
        *reinterpret_cast<uint4*>(p.codes_t + (bh * D + c) * (size_t)p.s + t0 + rg) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      __syncthreads();                               // the staging rows are rewritten by the next tile
    }
  }
  // a CTA that gave up must not exit while loads into its shared memory may still land
  if (abort_s) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    if (tid == 0) report_abort(p.ctl, abortp);
  }
}

// ------------------------------------------------------------------------------------------------ one thread per row
// The launches of the forward (codes, exponent / factor tables, NVFP4 copy, statistics; no prologue, no token-local exponents)
// run with ONE THREAD PER TOKEN ROW: CTA = 128 threads = one 128-token tile, warp = one 32-token block, so the block maximum
// is a warp reduction, the Hadamard butterflies need no shuffles, and one barrier per tile remains (it hands the input stage
// back to the loader and the codes to a TMA store). Every floating-point operation is the one the four-lanes-per-row kernel
// above performs on the same operands in the same order, so the two kernels' outputs are bit-identical
// (tests/test_gpu_quant.py compares them).
// One launch takes up to three operands (Q, K and V of a call): their tiles form one list, so that a short call pays one
// launch instead of three and a long one has one tail instead of three.
// What bounds it is latency, not traffic: a warp works through its rows alone (load, butterfly, maximum, codes), so the CTAs that
// share an SM have to cover each other. Three of them (d = 128: 168 registers a thread) instead of two need the codes to leave
// through the tile's own input buffer, whose rows every thread has read for itself; four at d = 64.
// One B200, before -> after: Q K V of b4 s4096 h16 d128 rotated 63.5 -> 56.5 us (traffic alone: 46), with NVFP4 copies 86 -> 82,
// 8 x 1000 x 12 heads at d = 64 18.3 -> 14.8.
static constexpr int QR_STAGES = 2;
constexpr int qr_ctas(int d) { return d == 128 ? 3 : 4; }
constexpr int qr_smem(int d) { return QR_STAGES * QT * d * 2 + (d == 128 ? 0 : 2 * QT * d) + 1024; }

struct QuantOperand {
  uint8_t* e_tab;         // outputs as in QuantParams; the codes leave through the operand's tensor map
  float* fac;
  uint8_t* x4;
  uint8_t* sf4;
  float* tile_stats;
  uint32_t* row_stat;
  int row_stat_kind;
  int s, h;
  int first;              // first tile of the operand in the launch's list
  int plain;              // no rotation and no NVFP4 copy for this operand (V), whatever the kernel's MODE
};
struct QuantRowsParams {
  QuantOperand op[3];
  int n_ops, n_tiles;
  const int32_t* slot_src;   // packed source, see QuantParams
  const int32_t* slot_rows;
  int skip_padding;          // host only: mostly_padding
  int in_f16;
  DocWork docs;              // packed source: the documents' work lists, made by block 0 while the others quantise (work null: none)
  DevCtl ctl;
};
struct QuantRowsMaps {
  CUtensorMap x[3], c[3];
};

// MODE and PK as in the four-lane kernel: bit 0 = the E4M3 codes are of the rotated row, bit 1 = also the NVFP4 copy, bit 2 =
// rotate only the NVFP4 copy.
template <int MODE, int D, int PK>
__global__ void __launch_bounds__(128, qr_ctas(D))
quant_rows_kernel(const __grid_constant__ QuantRowsMaps maps, const __grid_constant__ QuantRowsParams p) {
  static_assert(D == 128 || (D == 64 && MODE == 0), "head_dim 64 has no rotation and no NVFP4 copy");
  constexpr int QR_TILE_B = QT * D * 2;            // one 16-bit input tile (boxes of 64 columns: 128-byte rows)
  constexpr int QR_CODE_B = QT * D;                // its codes (rows of D bytes, the swizzle of that width)
  constexpr bool ROT = (MODE & 1) != 0, NV4 = (MODE & 2) != 0, ROT4 = (MODE & 4) != 0;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr bool OWN = D == 128;                   // the codes leave through the first box of the tile's own input buffer
  uint8_t* s_out = smem + (OWN ? 0 : QR_STAGES * QR_TILE_B);   // two code tiles (128 rows x D bytes)
  constexpr int OUT_STRIDE = OWN ? QR_TILE_B : QR_CODE_B;
  __shared__ __align__(8) uint64_t full[QR_STAGES];
  __shared__ float s_wmax[2][4], s_wsq[2][4];
  __shared__ __align__(16) uint4 s_zero[PK ? 8 : 1];           // what the rows past a slot's document read
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = tid;                               // token row of the tile
  if (PK && p.docs.work && blockIdx.x == 0) {
    static_assert(DOC_WORK_INTS * 4 <= QR_STAGES * QR_TILE_B);
    grid_dependency();
    doc_work<128>(p.docs, reinterpret_cast<int*>(smem), p.ctl.status);
    return;
  }
  const int G = gridDim.x - (PK && p.docs.work ? 1 : 0), cta = blockIdx.x - (PK && p.docs.work ? 1 : 0);
  volatile int* abortp = &abort_s;

  auto operand_of = [&](int L) { return (p.n_ops > 1 && L >= p.op[1].first) ? ((p.n_ops > 2 && L >= p.op[2].first) ? 2 : 1) : 0; };
  auto issue = [&](int L, int st) {
    const int o = operand_of(L);
    const int l = L - p.op[o].first, h = p.op[o].h, ntile = p.op[o].s / QT;
    const int head = l % h, tile = (l / h) % ntile, bat = l / (h * ntile);
    uint8_t* dst = smem + st * QR_TILE_B;
    // packed source (documents stored back to back): the slot's rows start at an arbitrary row of the (1, total, h, d)
    // tensor; only the innermost TMA coordinate has an alignment rule. An empty slot loads nothing.
    const int xrow = PK ? p.slot_src[tile] : tile * QT;
    mbar_arrive_expect_tx(&full[st], xrow >= 0 ? QR_TILE_B : 0);
    if (xrow >= 0) {
      tma_load_4d(dst, &maps.x[o], &full[st], 0, head, xrow, bat);
      if (D == 128) tma_load_4d(dst + QR_TILE_B / 2, &maps.x[o], &full[st], 64, head, xrow, bat);
    }
  };
  if (PK && tid < 8) s_zero[tid] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < QR_STAGES; ++i) mbar_init(&full[i], 1);
    fence_barrier_init();
    grid_dependency();
    for (int i = 0; i < QR_STAGES; ++i)
      if (cta + i * G < p.n_tiles) issue(cta + i * G, i);
  }
  __syncthreads();
  grid_dependency();

  int it = 0;
  for (int L = cta; L < p.n_tiles; L += G, ++it) {
    const int st = it % QR_STAGES, par = it & 1;
    const int oi = operand_of(L);
    const QuantOperand& op = p.op[oi];
    const int l = L - op.first, h = op.h, s = op.s, ntile = s / QT;
    const int head = l % h, tile = (l / h) % ntile, bat = l / (h * ntile);
    const int t0 = tile * QT;
    const size_t bh = (size_t)bat * h + head;
    const uint32_t tile_addr = smem_u32(smem + st * QR_TILE_B);
    const bool plain = MODE == 0 || op.plain;      // (CTA-uniform)
    const bool stats = op.tile_stats || op.row_stat;
    const int live_rows = PK ? p.slot_rows[tile] : QT;
    const bool live = r < live_rows;                    // packed source: rows past the slot's document read as zero
    const bool work = PK != 2 || warp * 32 < live_rows;
    bool ok = mbar_wait(&full[st], (it / QR_STAGES) & 1, p.ctl, abortp, 51);

    // the previous tile's buffer: filled again once its codes have left it (the store was issued a tile ago)
    if (OWN && tid == 0 && it > 0) {
      tma_store_wait_read<0>();
      if (L + (QR_STAGES - 1) * G < p.n_tiles) issue(L + (QR_STAGES - 1) * G, st ^ 1);
    }
    // ---- the row: D / 8 chunks of 8 elements (element 8 g + e in chunk g), rotation signs applied to the raw bits
    float x[D];
    // (one select of the row's address; of the loaded words it was 64: 16384 packed tokens h16/16 68 -> 66 us, lists included)
    const uint32_t row_at = PK && !live ? smem_u32(s_zero) : tile_addr + r * 128, box_at = PK && !live ? 0u : (uint32_t)(QR_TILE_B / 2);
    auto load_row = [&](bool signs) {
      constexpr uint32_t NEG[4] = {0x10D2E03Eu, 0xE0D9F0E2u, 0x45809F07u, 0x75954FEDu};
#pragma unroll
      for (int g = 0; g < D / 8; ++g) {
        const uint4 v = lds_u4(row_at + (g >> 3) * box_at + (((g & 7) ^ (r & 7)) << 4));
        uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (signs) {
            const int i0 = 8 * g + 2 * k, i1 = i0 + 1;
            const uint32_t m = (((NEG[i0 >> 5] >> (i0 & 31)) & 1u) << 15) | (((NEG[i1 >> 5] >> (i1 & 31)) & 1u) << 31);
            w[k] ^= m;
          }
          if (p.in_f16) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
            x[8 * g + 2 * k] = f.x;
            x[8 * g + 2 * k + 1] = f.y;
          } else {
            x[8 * g + 2 * k] = __uint_as_float(w[k] << 16);
            x[8 * g + 2 * k + 1] = __uint_as_float(w[k] & 0xFFFF0000u);
          }
        }
      }
    };
    // (y * signs) H_128 / sqrt(128): butterfly levels 1, 2, ..., 64 with (a, b) -> (a + b, a - b), the last one with the
    // scaling, subnormal results flushed
    auto rotate_row = [&]() {
      if constexpr (D == 128) {
      uint64_t Y[D / 2];
#pragma unroll
      for (int k = 0; k < D / 2; ++k) Y[k] = pack2(__fadd_rn(x[2 * k], x[2 * k + 1]), __fsub_rn(x[2 * k], x[2 * k + 1]));
#pragma unroll
      for (int hs = 1; hs < D / 4; hs <<= 1) {
#pragma unroll
        for (int k = 0; k < D / 2; ++k)
          if ((k & hs) == 0) {
            const uint64_t a = Y[k], b2 = Y[k + hs];
            Y[k] = add2(a, b2);
            Y[k + hs] = sub2(a, b2);
          }
      }
      const uint64_t c2 = pack2(0.08838834764831845f, 0.08838834764831845f);
#pragma unroll
      for (int k = 0; k < D / 4; ++k) {
        const uint64_t a = Y[k], b2 = Y[k + D / 4];
        unpack2(mul2_ftz(add2(a, b2), c2), x[2 * k], x[2 * k + 1]);
        unpack2(mul2_ftz(sub2(a, b2), c2), x[2 * k + D / 2], x[2 * k + D / 2 + 1]);
      }
      }
    };
    // NVFP4 copy of x: per 16 along d: SF = E4M3_rn(amax * f32(1/6)); codes = E2M1_rn(ftz(x * m)), m = 1 / SF | +inf (SF
    // rounds to 0, amax > 0) | 0. Scale bytes: group g of the row = byte g % 4 of the row's word in atom g / 4.
    auto nvfp4_row = [&]() {
      const size_t row_off = (((size_t)bat * s + t0 + r) * h + head) * D;
      uint8_t* x4row = op.x4 + row_off / 2;
      uint32_t sfw[2] = {0u, 0u};
#pragma unroll
      for (int g2 = 0; g2 < D / 32; ++g2) {           // two groups of 16 elements = one 16-byte store
        uint32_t pk[4];
#pragma unroll
        for (int gg = 0; gg < 2; ++gg) {
          const int g = 2 * g2 + gg;
          // the largest flushed magnitude = the flushed largest magnitude (flushing is monotone; a NaN never wins a max)
          float am = 0.f;
#pragma unroll
          for (int e = 0; e < 16; e += 2) am = fmax3_abs(am, x[16 * g + e], x[16 * g + e + 1]);
          am = flush_sub(am);
          const float u = __fmul_rn(am, 1.0f / 6.0f);
          const uint32_t sfb = cvt_e4m3x2(u, 0.f) & 0xFF;
          const float sfv = e4m3x2_to_f32((uint16_t)sfb).x;
          const float m = sfv > 0.f ? __frcp_rn(sfv) : (u > 0.f ? __int_as_float(0x7F800000) : 0.f);
          const uint64_t m2 = pack2(m, m);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {            // eight elements -> one word, low nibble first
            float a[8];
#pragma unroll
            for (int k = 0; k < 4; ++k)               // the product with subnormal inputs and results flushed, two at a time
              unpack2(mul2_ftz(pack2(x[16 * g + 8 * hh + 2 * k], x[16 * g + 8 * hh + 2 * k + 1]), m2), a[2 * k], a[2 * k + 1]);
            uint32_t w;
            asm("{\n\t.reg .b8 t0, t1, t2, t3;\n\t"
                "cvt.rn.satfinite.e2m1x2.f32 t0, %2, %1;\n\tcvt.rn.satfinite.e2m1x2.f32 t1, %4, %3;\n\t"
                "cvt.rn.satfinite.e2m1x2.f32 t2, %6, %5;\n\tcvt.rn.satfinite.e2m1x2.f32 t3, %8, %7;\n\t"
                "mov.b32 %0, {t0, t1, t2, t3};\n\t}"
                : "=r"(w)
                : "f"(a[0]), "f"(a[1]), "f"(a[2]), "f"(a[3]), "f"(a[4]), "f"(a[5]), "f"(a[6]), "f"(a[7]));
            pk[2 * gg + hh] = w;
          }
          sfw[g >> 2] |= sfb << (8 * (g & 3));
        }
        *reinterpret_cast<uint4*>(x4row + g2 * 16) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      }
      if (op.sf4) {
        uint8_t* atom = op.sf4 + ((bh * ntile + tile) * (D / 64)) * 512;
#pragma unroll
        for (int a = 0; a < D / 64; ++a) *reinterpret_cast<uint32_t*>(atom + a * 512 + (r & 31) * 16 + (r >> 5) * 4) = sfw[a];
      }
    };
    if (!work) {
      if (NV4 && !plain) {
        const uint4 zero = make_uint4(0, 0, 0, 0);
        uint4* x4row = reinterpret_cast<uint4*>(op.x4 + (((size_t)bat * s + t0 + r) * h + head) * (D / 2));
#pragma unroll
        for (int g2 = 0; g2 < D / 32; ++g2) x4row[g2] = zero;
        if (op.sf4)
#pragma unroll
          for (int a = 0; a < D / 64; ++a)
            *reinterpret_cast<uint32_t*>(op.sf4 + ((bh * ntile + tile) * (D / 64) + a) * 512 + (r & 31) * 16 + (r >> 5) * 4) = 0u;
      }
    } else if (ROT4 && !plain) {          // NVFP4 codes of the rotated row, E4M3 codes of the row as read
      load_row(true);
      rotate_row();
      nvfp4_row();
      load_row(false);
    } else if (ROT && !plain) {
      load_row(true);
      rotate_row();
      if (NV4) nvfp4_row();
    } else {
      load_row(false);
      if (NV4 && !plain) nvfp4_row();
    }
    if (work && (!ROT || ROT4 || plain)) {  // subnormal -> zero of the same sign (rotated rows were flushed by their scaling)
#pragma unroll
      for (int i = 0; i < D; i += 2) unpack2(mul2_ftz(pack2(x[i], x[i + 1]), pack2(1.0f, 1.0f)), x[i], x[i + 1]);
    }

    // ---- the row's maximum and (with the statistics) its sum of squares, in the four-lane kernel's summation order
    float amax = 0.f, sumsq = 0.f;
    if (work) {
      float aq[4] = {0.f, 0.f, 0.f, 0.f};          // per quarter q: elements 32 j + 8 q + e
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int j = 0; j < D / 32; ++j)
#pragma unroll
          for (int e = 0; e < 8; e += 2)
            aq[q] = fmax3_abs(aq[q], x[32 * j + 8 * q + e], x[32 * j + 8 * q + e + 1]);
      amax = fmaxf(fmaxf(aq[0], aq[1]), fmaxf(aq[2], aq[3]));
      if (stats) {
        float lq[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float sq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int j = 0; j < D / 32; ++j)
#pragma unroll
            for (int e = 0; e < 8; ++e) sq[e & 3] = fmaf(x[32 * j + 8 * q + e], x[32 * j + 8 * q + e], sq[e & 3]);
          lq[q] = (sq[0] + sq[1]) + (sq[2] + sq[3]);
        }
        sumsq = (lq[0] + lq[1]) + (lq[2] + lq[3]);
      }
    }
    if (op.row_stat && live) {
      const float v = op.row_stat_kind == 2 ? amax : (op.row_stat_kind == 3 ? __fsqrt_rn(sumsq) : sumsq);
      atomicMax(op.row_stat + (size_t)bat * s + t0 + r, __float_as_uint(v));
    }
    // the 32-token block = this warp (non-negative floats order as their bit patterns)
    uint32_t bm_bits, bs_bits;
    asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(bm_bits) : "r"(__float_as_uint(amax)));
    // (a row whose sum of squares is NaN does not take part, as with the NaN-ignoring maximum of the four-lane kernel)
    asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(bs_bits) : "r"(sumsq == sumsq ? __float_as_uint(sumsq) : 0u));
    const float bmax = __uint_as_float(bm_bits);
    if (lane == 0) { s_wmax[par][warp] = bmax; s_wsq[par][warp] = __uint_as_float(bs_bits); }
    const uint32_t bbyte = ue8m0_byte(bmax);
    const float inv = bbyte ? pow2_from_field(254 - (int)bbyte) : 0.f;

    // ---- codes -> this tile's staging buffer (rows of D bytes, the swizzle of that width)
    {
      const uint64_t inv2 = pack2(inv, inv);
      const uint32_t orow = smem_u32(s_out + par * OUT_STRIDE) + r * D;
      const int swz = D == 128 ? (r & 7) : ((r >> 1) & 3);
#pragma unroll
      for (int c = 0; c < D / 16; ++c) {            // 16 codes per 16-byte chunk
        uint32_t cw[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (!work) continue;
          float a0, a1, a2, a3;
          unpack2(mul2(pack2(x[16 * c + 4 * k], x[16 * c + 4 * k + 1]), inv2), a0, a1);
          unpack2(mul2(pack2(x[16 * c + 4 * k + 2], x[16 * c + 4 * k + 3]), inv2), a2, a3);
          cw[k] = cvt_e4m3x4(a0, a1, a2, a3);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(orow + ((c ^ swz) << 4)), "r"(cw[0]), "r"(cw[1]),
                     "r"(cw[2]), "r"(cw[3]) : "memory");
      }
    }
    fence_proxy_async();
    // the store of the previous tile has read its staging buffer (the other one): the next tile may write it
    if (!OWN && tid == 0) tma_store_wait_read<0>();
    // every thread has read the stage and written its codes; a wait that ran out leaves the loop here, all threads together
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    if (!ok) break;
    if (tid == 0) {
      if (!OWN && L + QR_STAGES * G < p.n_tiles) issue(L + QR_STAGES * G, st);
      tma_store_4d(&maps.c[oi], s_out + par * OUT_STRIDE, 0, head, t0, bat);
      tma_store_commit();
    }
    // ---- side tables
    const float* wm = s_wmax[par];
    if (lane == 0) {
      const uint32_t b0 = ue8m0_byte(wm[0]), b1 = ue8m0_byte(wm[1]), b2 = ue8m0_byte(wm[2]), b3 = ue8m0_byte(wm[3]);
      if (op.e_tab) {
        uint8_t* e = op.e_tab + (bh * (s / 32) + tile * 4 + warp) * (D / 32);
#pragma unroll
        for (int g = 0; g < D / 32; ++g) e[g] = (uint8_t)bbyte;
      }
      if (op.fac) {
        const uint32_t tm = max(max(b0, b1), max(b2, b3));
        const uint32_t e0 = bbyte ? bbyte : tm;
        op.fac[bh * (s / 32) + tile * 4 + warp] = e0 ? pow2_from_field((int)e0) : 1.0f;
      }
    }
    if (op.tile_stats && tid == 0) {
      op.tile_stats[(bh * ntile + tile) * 2] = fmaxf(fmaxf(wm[0], wm[1]), fmaxf(wm[2], wm[3]));
      op.tile_stats[(bh * ntile + tile) * 2 + 1] = fmaxf(fmaxf(s_wsq[par][0], s_wsq[par][1]), fmaxf(s_wsq[par][2], s_wsq[par][3]));
    }
  }
  // the staging buffers must outlive the stores that read them; a CTA that gave up must not exit while loads may still land
  if (tid == 0) tma_store_wait_read<0>();
  if (abort_s) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    if (tid == 0) report_abort(p.ctl, abortp);
  }
}

template <int MODE, int D>
static int launch_quant_rows(const QuantRowsMaps& maps, const QuantRowsParams& p, cudaStream_t st) {
  const int smem = qr_smem(D);
  const int grid = min(p.n_tiles + (p.docs.work ? 1 : 0), sm_count() * qr_ctas(D));
  auto launch = [&](auto kern) -> int {
    if (int rc = set_smem(kern, smem, "fl_quant_blocks: cudaFuncSetAttribute")) return rc;
    launch_after(kern, grid, 128, smem, st, maps, p);
    return FL_OK;
  };
  return !p.slot_src ? launch(quant_rows_kernel<MODE, D, 0>)
         : p.skip_padding && p.n_tiles > 3 * grid ? launch(quant_rows_kernel<MODE, D, 2>) : launch(quant_rows_kernel<MODE, D, 1>);
}

template <int D, int MODE, bool PRO, int STEPS, int PK>
static int launch_quant_pk(const CUtensorMap& mx, const CUtensorMap& mo, const QuantParams& p, bool want_t, cudaStream_t st) {
  const int smem = QSTAGES * (PRO ? 2 : 1) * (QT / STEPS * D * 2) + 1024 + (want_t ? QT * (D + 16) : 0);
  auto kern = quant_blocks_kernel<D, MODE, PRO, STEPS, PK>;
  if (int rc = set_smem(kern, smem, "fl_quant_blocks: cudaFuncSetAttribute")) return rc;
  const int per_sm = want_t ? 1 : q_blocks(PRO, STEPS);
  const int grid = min(p.n_tiles, sm_count() * per_sm);
  launch_after(kern, grid, q_threads(STEPS), smem, st, mx, mo, p);
  return FL_OK;
}

template <int D, int MODE, bool PRO, int STEPS = 1>
static int launch_quant(const CUtensorMap& mx, const CUtensorMap& mo, const QuantParams& p, bool want_t, cudaStream_t st) {
  if (!p.slot_src) return launch_quant_pk<D, MODE, PRO, STEPS, 0>(mx, mo, p, want_t, st);
  if (PRO && p.skip_padding && p.n_tiles > 3 * sm_count() * q_blocks(PRO, STEPS)) return launch_quant_pk<D, MODE, PRO, STEPS, PRO ? 2 : 1>(mx, mo, p, want_t, st);
  return launch_quant_pk<D, MODE, PRO, STEPS, 1>(mx, mo, p, want_t, st);
}

// Steps of a prologue tile. Two where both of an SM's blocks have tiles. One where there is no more than a tile an SM, or where in the
// last round most SMs have one tile only, which a block of 256 then works through with nothing beside it.
// One B200 (148 SMs), one head, launch in a row, one step / two steps, us at d = 64 (d = 128): 16 tiles 3.4 / 4.1 (4.2 / 4.9), 148 tiles
// 3.6 / 4.3 (4.4 / 5.1), 296 tiles 5.6 / 5.0 (6.9 / 6.5), 390 tiles 7.5 / 7.8 (9.6 / 9.7), 407 to 444 tiles 7.5 / 8.7 (9.6 / 11.1), 592 tiles
// 9.5 / 9.0 (12.1 / 11.5), 666 tiles 11.5 / 11.5 (14.8 / 14.4), 740 tiles 11.5 / 12.6 (15.1 / 16.3), 1184 tiles 17.3 / 16.7 (26.3 / 25.4);
// b4 s4096 h16 d128 41.9 / 43.3, behind a write of O 47.2 / 45.1. One with the channel-major copy, whose staging rows leave room for one
// block an SM at d = 128 (b4 s4096 h16, one step / two: 79 / 90 us, at d = 64 48 / 64).
static int prologue_steps(long long n_tiles, bool want_t) {
  if (want_t) return 1;
  const int sms = sm_count(), rest = (int)(n_tiles % (2 * sms));
  return rest > sms || rest == 0 || (n_tiles > 3 * sms && rest <= sms * 2 / 3) ? 2 : 1;
}

static int quant_cols(const fl_quant_args* a) { return (a->flags >> 16) > 0 ? (a->flags >> 16) : a->d; }

// rows of a batch row of x (the outputs have a->s): the tensor maps read the missing ones as zeros
static int quant_src_rows(const fl_quant_args* a) { return a->slot_src || (a->flags & FL_Q_ROWS) ? a->src_rows : a->s; }

static int check_quant_args(const fl_quant_args* a) {
  if (!a || !a->x || !a->codes) return FL_ERR_BAD_ARG;
  if (a->b <= 0 || a->s <= 0 || a->h <= 0 || (a->s % 128) != 0) return FL_ERR_BAD_ARG;
  if (a->d != 64 && a->d != 128) return FL_ERR_UNSUPPORTED;
  if (quant_cols(a) > a->d || quant_cols(a) % 8) return FL_ERR_BAD_ARG;
  if ((a->flags & (FL_Q_HADAMARD | FL_Q_HADAMARD_NVFP4_ONLY)) && a->d != 128) return FL_ERR_UNSUPPORTED;
  if ((a->flags & FL_Q_HADAMARD) && (a->flags & FL_Q_TOKEN_LOCAL)) return FL_ERR_UNSUPPORTED;
  if ((a->flags & FL_Q_D_PER_FACTOR) && !(a->flags & FL_Q_TOKEN_LOCAL)) return FL_ERR_BAD_ARG;
  if ((a->flags & FL_Q_HADAMARD_NVFP4_ONLY) && !a->x4) return FL_ERR_BAD_ARG;
  if (a->h > 65535) return FL_ERR_TOO_LARGE;
  if ((long long)a->b * (a->s / 128) * a->h > 0x7FFFFFFF) return FL_ERR_TOO_LARGE;
  if (a->row_stat && (a->row_stat_kind < 1 || a->row_stat_kind > 3)) return FL_ERR_BAD_ARG;
  if (a->slot_src && (!a->slot_rows || a->b != 1 || a->src_rows <= 0)) return FL_ERR_BAD_ARG;
  if (!a->slot_src && (a->flags & FL_Q_ROWS) && (a->src_rows <= 0 || a->src_rows > a->s || a->src_rows <= a->s - 128)) return FL_ERR_BAD_ARG;
  return FL_OK;
}

// what the one-thread-per-row kernel serves (same bits as the other one, fewer instructions, no shuffles)
static bool rows_kernel_serves(const fl_quant_args* a) {
  return (a->d == 128 || !(a->flags & (FL_Q_HADAMARD | FL_Q_HADAMARD_NVFP4_ONLY) || a->x4)) && !(a->d_out && a->o) && !a->codes_t &&
         !(a->flags & (FL_Q_TOKEN_LOCAL | FL_Q_LEGACY)) && !a->sf_tok && !a->sf_dim && !a->token_factors && !a->zero_acc && !a->lse_log2;
}
// MODE of an operand: bit 0 = rotate the codes, bit 1 = NVFP4 copy, bit 2 = rotate the copy only
static int quant_mode(const fl_quant_args* a) {
  if (a->flags & FL_Q_HADAMARD_NVFP4_ONLY) return 6;
  return ((a->flags & FL_Q_HADAMARD) ? 1 : 0) | (a->x4 ? 2 : 0);
}

// Packed sources: is more than an eighth of the tiles' rows past the end of a document? Then the kernels in which the warps of such rows
// leave their work out (PK = 2): 352 documents of 30 to 60 rows, h16/16, d = 128, step 869 -> 815 us; 210 of 100 to 200 454 -> 448; 6000
// rows in documents of 16 to 1024, h16/4, 182.5 -> 181.2. Not where the documents are long (16k rows in 4, 672 -> 677), and not in a
// launch of up to three rounds, which is over before the shorter way pays for the longer code (75 rows h16/8, mixed route, forward 14.4 ->
// 14.9; 1.1 rounds, prologue, d = 64, 8.4 -> 8.9; 1.2 rounds, rows, 9.7 -> 9.9; 2.7 rounds the same; 3.4 rounds, rows, 30.1 -> 29.4).
static bool mostly_padding(const fl_quant_args* const* args, int n) {
  long long rows = 0, aligned = 0;
  for (int i = 0; i < n; ++i) rows += (long long)args[i]->src_rows * args[i]->h, aligned += (long long)args[i]->s * args[i]->h;
  return args[0]->slot_src && 8 * rows < 7 * aligned;
}

static int quant_rows(const fl_quant_args* const* args, int n, cudaStream_t st, const DocWork& docs = {}) {
  QuantRowsMaps maps;
  QuantRowsParams p = {};
  int mode = 0;
  long long tiles = 0;
  for (int i = 0; i < n; ++i) {
    const fl_quant_args* a = args[i];
    const int m = quant_mode(a);
    if (m) mode = m;
    QuantOperand& o = p.op[i];
    o.e_tab = a->e_tab; o.fac = a->fac; o.x4 = a->x4; o.sf4 = a->sf4; o.tile_stats = a->tile_stats;
    o.row_stat = (uint32_t*)a->row_stat; o.row_stat_kind = a->row_stat_kind;
    o.s = a->s; o.h = a->h; o.first = (int)tiles; o.plain = m == 0;
    tiles += (long long)a->b * (a->s / 128) * a->h;
    int rc;
    if ((rc = make_rows_map_16(&maps.x[i], a->x, a->b, quant_src_rows(a), a->h, quant_cols(a), 128))) return rc;
    if ((rc = make_rows_map(&maps.c[i], a->codes, a->b, a->s, a->h, a->d, 128))) return rc;
  }
  if (tiles > 0x7FFFFFFF) return FL_ERR_TOO_LARGE;
  const fl_quant_args* a = args[0];
  p.n_ops = n; p.n_tiles = (int)tiles;
  p.slot_src = a->slot_src; p.slot_rows = a->slot_rows;
  p.skip_padding = mostly_padding(args, n);
  p.in_f16 = a->in_f16;
  p.docs = docs;
  p.ctl = dev_ctl(a->status, a->wait_cycles > 0 ? a->wait_cycles : kDefaultWaitCycles);
  int rc;
  if (a->d == 64) rc = launch_quant_rows<0, 64>(maps, p, st);
  else if (mode == 6) rc = launch_quant_rows<6, 128>(maps, p, st);
  else if (mode == 3) rc = launch_quant_rows<3, 128>(maps, p, st);
  else if (mode == 2) rc = launch_quant_rows<2, 128>(maps, p, st);
  else if (mode == 1) rc = launch_quant_rows<1, 128>(maps, p, st);
  else rc = launch_quant_rows<0, 128>(maps, p, st);
  return rc ? rc : launch_result("fl_quant_blocks: kernel launch");
}

}  // namespace fl

extern "C" int fl_quant_blocks(const fl_quant_args* a, void* stream) {
  using namespace fl;
  if (int rc = check_quant_args(a)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  if (rows_kernel_serves(a)) return quant_rows(&a, 1, st);
  const long long n_tiles = (long long)a->b * (a->s / 128) * a->h;
  const bool pro = a->d_out != nullptr && a->o != nullptr;
  const bool rot = (a->flags & FL_Q_HADAMARD) != 0, rot4 = (a->flags & FL_Q_HADAMARD_NVFP4_ONLY) != 0;
  const bool nv4 = a->x4 != nullptr;
  if (pro && (rot || rot4 || nv4)) return FL_ERR_UNSUPPORTED;     // the prologue rides on the dO launch, which does neither
  QuantParams p;
  p.lse = a->lse; p.codes = a->codes; p.codes_t = a->codes_t; p.e_tab = a->e_tab; p.fac = a->fac; p.sf_tok = a->sf_tok;
  p.sf_dim = a->sf_dim; p.token_factors = a->token_factors; p.x4 = a->x4; p.sf4 = a->sf4; p.d_out = a->d_out;
  p.lse_log2 = a->lse_log2; p.zero_acc = (uint16_t*)a->zero_acc; p.tile_stats = a->tile_stats;
  p.row_stat = (uint32_t*)a->row_stat; p.row_stat_kind = a->row_stat_kind;
  p.b = a->b; p.s = a->s; p.h = a->h; p.n_tiles = (int)n_tiles;
  p.slot_src = a->slot_src; p.slot_rows = a->slot_rows;
  p.skip_padding = mostly_padding(&a, 1);
  const bool packed = a->slot_src != nullptr;
  const int d_src = quant_cols(a);
  p.token_local = (a->flags & FL_Q_TOKEN_LOCAL) ? 1 : 0;
  p.d_per_factor = (a->flags & FL_Q_D_PER_FACTOR) ? 1 : 0;
  p.in_f16 = a->in_f16;
  p.lse_shift = a->lse_shift; p.d_multiplier = a->d_multiplier;
  p.ctl = dev_ctl(a->status, a->wait_cycles > 0 ? a->wait_cycles : kDefaultWaitCycles);
  CUtensorMap mx, mo;
  int rc;
  const bool wt = a->codes_t != nullptr;
  const int steps = pro ? prologue_steps(n_tiles, wt) : 1, box = QT / steps;          // rows of a step
  if ((rc = make_rows_map_16(&mx, a->x, a->b, quant_src_rows(a), a->h, d_src, box))) return rc;
  p.o_packed = (packed && (a->flags & FL_Q_O_PACKED)) ? 1 : 0;
  if ((rc = make_rows_map_16(&mo, pro ? a->o : a->x, a->b, !packed || p.o_packed ? quant_src_rows(a) : a->s, a->h, d_src, box))) return rc;
  if (a->d == 64) {
    if (pro) rc = steps == 2 ? launch_quant<64, 0, true, 2>(mx, mo, p, wt, st) : launch_quant<64, 0, true>(mx, mo, p, wt, st);
    else rc = nv4 ? launch_quant<64, 2, false>(mx, mo, p, wt, st) : launch_quant<64, 0, false>(mx, mo, p, wt, st);
  } else if (pro) {
    rc = steps == 2 ? launch_quant<128, 0, true, 2>(mx, mo, p, wt, st) : launch_quant<128, 0, true>(mx, mo, p, wt, st);
  } else if (rot4) {
    rc = launch_quant<128, 6, false>(mx, mo, p, wt, st);
  } else if (rot) {
    rc = nv4 ? launch_quant<128, 3, false>(mx, mo, p, wt, st) : launch_quant<128, 1, false>(mx, mo, p, wt, st);
  } else {
    rc = nv4 ? launch_quant<128, 2, false>(mx, mo, p, wt, st) : launch_quant<128, 0, false>(mx, mo, p, wt, st);
  }
  if (rc) return rc;
  return launch_result("fl_quant_blocks: kernel launch");
}

namespace fl {
// do the three go as one launch of the one-thread-per-row kernel?
static bool one_launch(const fl_quant_args* q, const fl_quant_args* k, const fl_quant_args* v) {
  const int mq = quant_mode(q), mk = quant_mode(k), mv = quant_mode(v);
  return rows_kernel_serves(q) && rows_kernel_serves(k) && rows_kernel_serves(v) && mq == mk && mv == 0 && q->d == k->d && q->d == v->d &&
         q->in_f16 == k->in_f16 && q->in_f16 == v->in_f16 && q->slot_src == k->slot_src && q->slot_src == v->slot_src;
}

// Work lists: does a block of the quantiser's launch make them in the time that a launch of their own would take? Its 128 threads take
// eight times as many turns over documents and tiles as the 1024 there. Up to 1536 of these it always does (2560 where the documents
// are few or short), beyond where the quantiser beside it has work enough: tiles of 64 columns for each tile of the buffer, more of them
// where full tiles of many documents load the memory (a buffer sized for any division has empty tiles between). Above 4096 it was not
// measured. One B200, quantiser with the lists / with the launch, us:
// d = 64, documents of a tile: 75 tiles h16/4 7 us less; 1536 h1/1 30.9 / 31.6; 2048 h1/1 48 / 38, h4/1 64 / 62, h4/2 74 / 78; 3000 h1/1
//   74 / 53, h4/2 115 / 110, h6/2 131 / 132; 4096 h1/1 104 / 71, h4/2 158 / 147, h6/2 180 / 179;
// documents of 32 rows: 2048 h1/1 33 / 34; 3000 h2/1 62 / 59, h4/1 76 / 79; 4096 h2/1 92 / 79, h4/1 110 / 106, h4/2 125 / 137;
// d = 128: 2048 h1/1 61 / 71; 3000 h1/1 98 / 99; 4096 h1/1 136 / 131, h2/1 158 / 169, with NVFP4 copies h1/1 152 / 170;
// whole forward calls with cu_seqlens (twice as many tiles as documents, each of a tile), d = 64: 1000 documents h1/1 62 / 70, 1500 h1/1
//   101 / 97, h4/1 236 / 243, 2040 h1/1 137 / 126, h4/1 323 / 327.
static bool lists_hide(const fl_quant_args* q, const fl_quant_args* k, const fl_quant_args* v, int n_docs, int tiles) {
  const int most = max(n_docs, tiles);
  const float full = min((float)n_docs, q->src_rows / 128.f) * min(1.f, (float)n_docs / tiles);
  const float col = q->d == 128 ? 2.75f : 1.f, score = q->x4 ? 3.75f : col;      // a tile's time in tiles of 64 columns
  return most <= 1536 || (most <= 2560 && full <= 1100) || (most <= 4096 && score * (q->h + k->h) + col * v->h >= 3.9f + full * (6.f / 4096));
}
}  // namespace fl

extern "C" int fl_quant_qkv(const fl_quant_args* q, const fl_quant_args* k, const fl_quant_args* v, void* stream) {
  using namespace fl;
  const fl_quant_args* a[3] = {q, k, v};
  for (const fl_quant_args* x : a)
    if (int rc = check_quant_args(x)) return rc;
  if (one_launch(q, k, v)) return quant_rows(a, 3, (cudaStream_t)stream);
  for (const fl_quant_args* x : a)
    if (int rc = fl_quant_blocks(x, stream)) return rc;
  return FL_OK;
}

extern "C" int fl_quant_qkv_work(const fl_quant_args* q, const fl_quant_args* k, const fl_quant_args* v, const int32_t* doc_start,
                                 const int32_t* doc_len, int32_t n_docs, int32_t capacity, int32_t window_left_p1,
                                 int32_t window_right_p1, int32_t causal, int32_t ordered, int32_t* work, void* stream) {
  using namespace fl;
  const fl_quant_args* a[3] = {q, k, v};
  for (const fl_quant_args* x : a)
    if (int rc = check_quant_args(x)) return rc;
  if (!doc_start || !doc_len || !work || n_docs <= 0 || capacity <= 0 || (capacity % 128)) return FL_ERR_BAD_ARG;
  if (one_launch(q, k, v) && q->slot_src && lists_hide(q, k, v, n_docs, capacity / 128))
    return quant_rows(a, 3, (cudaStream_t)stream,
                      DocWork{doc_start, doc_len, n_docs, capacity, window_side(window_left_p1), causal ? 0 : window_side(window_right_p1),
                              ordered, (int4*)work});
  if (int rc = fl_quant_qkv(q, k, v, stream)) return rc;
  return fl_doc_work(doc_start, doc_len, n_docs, capacity, window_left_p1, window_right_p1, causal, ordered, work, q->status, stream);
}
