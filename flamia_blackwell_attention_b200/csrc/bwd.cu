// Backward main kernel for sm_100a (head_dim 128 or 64): dK, dV and the pre-scaled f16 dQ accumulator from block-scaled
// operands, software-pipelined over 64-query half tiles, on a persistent grid.
//
// Replaces the reference's FlashAttentionBackwardSm100FP4 (flash_attn/cute/flash_bwd_sm100_fp4.py:82; driver
// flash_attn/cute/interface_bwd_fp4.py:1207) for the E4M3 backward. One CTA per SM walks a static list of work items
// (128-key tile, kv head, batch | document): under the causal mask the items are ordered longest first and dealt out in
// zigzag rounds (round k gives CTA c item k G + c or k G + G - 1 - c), so every CTA gets nearly the same number of query
// tiles. All pipelines run ACROSS items: the K / V tiles of the next item are loaded into a second buffer while the
// current item's last query tiles are processed, the first S^T / dP^T products of the next item are issued while the
// compute warpgroups write the current item's dK / dV, and barriers, tensor memory and tensor maps are set up once per CTA.
// An item walks the query tiles that see its key tile (x the query heads of the GQA group), each as two 64-query halves
// x = 0, 1 that run one step apart, so the tensor core works on one half while the other half's elementwise math runs:
//   S^T_x  = K Q_x^T                  kind::f8f6f4, N = 64 (token-block factors folded into the exponent argument)
//   P'     = 2^(S^T c - lse_log2) = 2^8 P        -> P-hat = E4M3(P')                   [tensor memory]
//   dV    += P-hat^T dO_x             kind::mxf8f6f4.block_scale, B scale = dO's UE8M0 per 32 queries
//   dP^T_x = V dO_x^T                 kind::f8f6f4
//   dS     = P' (b dP^T + D''), b = f_V f_dO 2^-8, D'' = -2^-8 rowsum(O dO)
//   dS-hat : one UE8M0 exponent per 32 keys x 32 queries, E4M3 codes (the same codes feed dK and dQ)
//   dK    += dS-hat^T Q_x             block-scaled, A from tensor memory
//   dQ^T_x = K^T dS-hat^T             block-scaled, M = head dim, N = 64 queries; A = K tile and B = dS-hat (shared
//                                     memory) both MN-major; the f16 pre-scale B_m is folded into the A scale bytes
//   dQ^T_x -> f16 -> TMA reduce-add into the (b, h, d, s) accumulator
//   d = 64: block-scaled products need M = 128, so the product is taken the other way round, dQ_x = dS-hat_x K with
//   A = dS-hat (shared memory, MN-major; its second 64-row block is whatever follows in memory and only fills the
//   unused rows 64..127 of the result) and B = the K tile; rows = queries, accumulator layout (b, h, s, d)
//   compute warpgroups: two, one per half (64 queries each), or four of 32 queries (bwd_qw); thread = key row = TMEM lane
//   four warps of dQ reduction (thread = head-dim row), one TMA producer warp
//   three UMMA issuer warps: dQ^T, dV, dK | S^T | dP^T
// TMEM: [0,64) / [64,128) S^T_x; [128,256) dV; [256,320) / [320,384) dP^T_x, then dQ^T_x; [384,512) dK.
// P-hat, dS-hat and the scale tiles of a half go to the OTHER half's S^T columns (P-hat +0, dS-hat +16, scale tiles +32..+56): the
// compute warps read all 64 scores of a row into registers at once, so their own S^T columns take the next scores while they
// work, and a half goes from one iteration to the next without waiting for the tensor core. The regions alternate,
//   region 0: S0(g) -> read -> P1, dS1(g - 1) -> dV dK dQ of (g - 1, 1) -> S0(g + 1) ...
//   region 1: S1(g) -> read -> P0, dS0(g)     -> dV dK dQ of (g, 0)     -> S1(g + 1) ...
// so the issue order is [dQ dV dK](g, 0), S1(g + 1), dP0(g + 1), [dQ dV dK](g, 1), S0(g + 2), dP1(g + 1): one wait of the issuer per
// half and about 830 clocks of products behind it (an mbarrier wait costs the issuer 100 to 150 clocks even when the phase
// has completed, and the tensor pipe takes about eight instructions ahead: with P-hat and dS-hat announced separately and S^T
// issued after them the pipe drained at each of four waits per half, and the compute warps waited 1100 to 1700 of an
// iteration's 3800 clocks for their scores). Half 0 runs ahead by up to one iteration.
// Every wait is bounded (sm100.cuh).
// Item epilogue: the compute warpgroups read dV (warpgroup 0) / dK (warpgroup 1) out of tensor memory, release the
// accumulators to the next item's products, and write their rows through the finished item's K / V tile buffers (dead by
// then) with TMA stores, 64 columns at a time; only then may the producer refill those buffers (two items ahead).
// FL_MODE_FP4 (the mixed route): S^T_x is recomputed at the forward's precision, K4 Q4_x^T with
// kind::mxf4nvf4.block_scale.scale_vec::4X on the NVFP4 copies; everything after P' is the E4M3 path above. The 16 scale
// columns of that product (tcgen05.cp of the K and Q atoms) are parked in dP^T columns whose dQ^T has been read out and whose
// next dP^T is issued right behind the S^T (the tensor pipe runs in issue order). The second half's Q scales are columns
// 2, 3 of each atom.
// VAR = 1 (FL_A_DQ_ROWLOCAL, the reference's ds_dq_rowlocal="all", flash_bwd_sm100_fp4.py:3637-3642): the dQ side of
// dS-hat gets its own codes with one exponent per (query row, 32-key block) instead of sharing the 32 x 32 block's.
// VAR = 2 (FL_A_TOKEN_LOCAL + row-local, flash_bwd_sm100_fp4.py:152-158): every token of Q, K, V, dO carries its own
// power-of-two factor. Per-key factors are per-thread scalars here, per-query factors are read per element; S and dP
// take f_K f_Q and f_V f_dO in the elementwise math; dV takes f_dO inside a block-scaled P-hat (one exponent per key row
// x 32 queries); dK takes f_Q inside its dS-hat codes, dQ takes f_K inside its own; the operand scale tiles are unit.
// What bounds these kernels are the loads of the per-query tables: each returns 512 bytes to a warp, four clocks of the 2 350 of a half
// tile. VAR = 3 (FL_A_D_PER_FACTOR: D'' comes divided by f_dO, exactly, as f_dO is a power of two) takes 40 of them a warp: P' f_dO, which
// P-hat needs, is all that dS = (P' f_dO) (f_V dP + D'' / f_dO) needs, too. VAR = 2, for callers with D'' as it is, takes 56 (48 if P' f_dO is
// kept for its codes, in 32 registers more, which costs 1 to 3 %). b2 s8192 h32/8 d128 causal, kernel alone, one B200: VAR = 2 with 48 loads
// 2445 us, with 56 2381 to 2431, VAR = 3 2325 to 2360; the same bits.
#include "flamia_internal.h"

namespace fl {

struct BwdParams {
  const float* fac_q;
  const float* fac_k;
  const float* fac_v;
  const float* fac_do;
  const float* lse_log2;
  const float* d_rows;
  const float* dq_scale;
  const float* dq_scale_rows;   // (b, s_q) per query row instead of dq_scale per query tile, or null
  const float* dk_mult;         // (b, h_kv) factor on dK (Q's mantissa with float descales), or null
  const int32_t* slot_src;      // packed output: packed row of each 128-row slot of the aligned buffer (-1: empty), or null
  const int32_t* slot_rows;     // packed output: real rows of each slot
  const uint8_t* sfq4;   // FL_MODE_FP4: E4M3 scale atoms of the NVFP4 Q / K copies (1 KB per 128-row tile)
  const uint8_t* sfk4;
  void* dk;
  void* dv;
  const int32_t* doc_start;
  const int32_t* doc_len;
  const int32_t* seqused_k;   // batched form: valid keys per batch row, or null
  int32_t* dq_order;     // deterministic dQ: (b, h, s_q / 128, 2) counters, zero on entry, or null
  int n_docs;
  int b, s_q, s_k, h, h_kv;
  int q_len, k_len;      // batched form: a batch row's queries and keys (s_q, s_k, or fewer where those are rounded up to whole tiles)
  int d_out;             // columns of a gradient row (D, or fewer: zero-padded head dims)
  float scale_log2;
  float softmax_scale;
  float cap_a, cap_b;    // soft cap c: x = cap_a tanh(s * factor * cap_b) in log2 units, cap_a = c log2 e, cap_b = 1 / cap_a
  int causal;
  int win_l, win_r;      // sliding window sides, -1 = unlimited (causal: the right side is 0)
  int out_f16;
  int had_dk;
  const int4* work;      // documents: the backward entries of fl_doc_work's list, or null
  const int4* work_head;
  FastDiv div_item, div_h;   // items per (causal: key tile; otherwise: kv head), kv heads
  int grp;               // query heads per kv head
  int n_items;           // work items: key tiles x kv heads x batch rows (documents: tile slots x kv heads)
  int n_tile;            // key tiles per batch row (documents: tile slots of the packed buffer)
  int zigzag;            // deal the items out in zigzag rounds (causal: they are ordered longest first)
  DevCtl ctl;
};

struct BTile {
  int bat;    // batch coordinate of the tensor maps (0 for packed documents)
  int hkv;    // kv head
  int k0;     // first key row of the tile (row index inside the batch entry)
  int nk;     // key rows of the tile inside the document / batch row (<= 128; 0 = an empty tile slot)
  int nv;     // of those, the keys that take part (fewer under seqused_k; <= 0: none, the tile's gradients are zero)
  int krel;   // document-relative index of key row k0
  int q0;     // first query row of the document (row index inside the batch entry)
  int sq;     // queries of the document
  int off;    // causal alignment: key j (document-relative) is visible to query i iff j <= i + off
  int m_lo;   // first query tile that sees this key tile
  int n_m;    // number of query tiles that see it
};

// barriers; [2] = one per half, stage or buffer, [3] = one per stage of the score operand's ring
// (B ring: [stage][half])
enum { BB_KV = 0, BB_KVE = 2, BB_AFULL = 4, BB_AEMPTY = 7, BB_BFULL = 10, BB_BEMPTY = 14, BB_S = 18, BB_DP = 20, BB_GRANT = 22,
       BB_DS = 24, BB_DQF = 26, BB_DQE = 28, BB_EPI = 30, BB_R1 = 34, BB_R2 = 35, BB_ACC = 36, BB_ACCFREE = 37, BB_SDR = 38,
       BB_EPX = 39, BB_ROT = 41, BB_COUNT = 42 };
// TMEM columns; the per-half regions are at + 64 * x
enum { TC_S = 0, TO_P = 0, TO_DS = 16, TO_SFA_P = 32, TO_SFB_DO = 36, TO_SFB_Q = 40, TO_SFA_DQ = 44, TO_SFA_DK = 48,
       TO_SFB_DQ = 52, TC_DV = 128, TC_DP = 256, TC_DK = 384 };

// bits of the warp's largest |v| (the f32 form of the instruction is faster than masking the sign and reducing integers:
// -8 % on the row-local backward, which runs it once per dS column)
__device__ __forceinline__ uint32_t warp_max_abs_f32(float v) {
  float r;
  asm volatile("redux.sync.max.abs.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return __float_as_uint(r);
}
template <int N>
__device__ __forceinline__ void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ float4 lds128(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sts8(uint32_t addr, uint32_t v) { asm volatile("st.shared.b8 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
// 448 * 2^(e - 127) >= amax for the returned UE8M0 byte (bits = the non-negative float's pattern), clamped to [1, 254]
__device__ __forceinline__ uint32_t exp448(uint32_t bits) {
  const int e = (int)((bits + 0x00200000u) >> 23) - 8;
  return (uint32_t)min(max(e, 1), 254);
}
__device__ __forceinline__ float pow2_inv(uint32_t ebyte) { return __uint_as_float((uint32_t)(254 - (int)ebyte) << 23); }

// k-th work item of CTA c on a grid of G CTAs (>= n_items: the CTA is done)
__device__ __forceinline__ int bwd_item(int k, int G, int c, int zigzag) {
  return k * G + ((zigzag && (k & 1)) ? (G - 1 - c) : c);
}

// Work item L -> its key tile. Causal: tiles slowest, so that the item index orders the items longest first (a key tile
// near the start of the sequence is seen by the most query tiles). Otherwise tiles fastest: the CTAs that run at the same
// time work on one head and share its Q / dO tiles in L2.
template <bool DOCS>
__device__ __forceinline__ void bwd_decode(const BwdParams& p, int L, BTile& t) {
  if (!DOCS || p.doc_start == nullptr) {
    const int q = p.div_item.div(L), rq = L - q * p.div_item.d;
    const int tile = p.causal ? q : rq, rem = p.causal ? rq : q;
    t.bat = p.div_h.div(rem); t.hkv = rem - t.bat * p.h_kv;
    t.k0 = tile * 128; t.nk = min(128, p.k_len - t.k0); t.krel = t.k0; t.q0 = 0; t.sq = p.q_len; t.off = p.k_len - p.q_len;
    t.nv = p.seqused_k ? min(t.nk, p.seqused_k[t.bat] - t.k0) : t.nk;
  } else {
    // documents sit at 128-aligned starts of one packed batch entry; tile slot x -> (document, key tile of it)
    int x = p.div_h.div(L), dsel = -1, len = 0, st = 0;
    t.hkv = L - x * p.h_kv;
    if (p.work) {          // longest first; checked when the list was made
      const int4 e = __ldg(p.work + x);
      st = e.x; len = e.y; x = e.z; dsel = 0;
    } else {
      for (int dI = 0; dI < p.n_docs; ++dI) {
        doc_entry(p.doc_start, p.doc_len, dI, p.s_k, p.ctl.status, st, len);
        const int nb = (len + 127) / 128;
        if (x < nb) { dsel = dI; break; }
        x -= nb;
      }
    }
    if (dsel < 0) { t.nk = 0; t.bat = 0; t.k0 = 0; t.krel = 0; t.q0 = 0; t.sq = 0; t.off = 0; }
    else { t.bat = 0; t.k0 = st + x * 128; t.nk = min(128, len - x * 128); t.krel = x * 128; t.q0 = st; t.sq = len; t.off = 0; }
    t.nv = t.nk;
  }
  // query tiles that see this key tile: the first query that sees its first key, the last one that sees its last key
  int m_hi = (t.sq + 127) / 128, m_lo = 0;
  if (p.win_r >= 0 && t.krel - t.off - p.win_r > 0) m_lo = (t.krel - t.off - p.win_r) / 128;
  if (p.win_l >= 0) m_hi = min(m_hi, max(0, t.krel + t.nk - 1 - t.off + p.win_l) / 128 + 1);
  t.m_lo = m_lo;
  t.n_m = (t.nv > 0 && m_hi > m_lo) ? (m_hi - m_lo) : 0;
}

// Deterministic dQ: how many key tiles before this one also see query tile m of the document (they add their partial sums
// first). The key tiles that see a query tile are a contiguous range; without a left window it starts at key tile 0.
__device__ __forceinline__ int bwd_order_rank(const BwdParams& p, const BTile& t, int m) {
  const int kt = t.krel / 128;
  if (p.win_l < 0) return kt;
  // first key tile whose last query tile is not below m (key tiles are full except the document's last one)
  int klo = 0;
  while (klo < kt && max(0, klo * 128 + 127 - t.off + p.win_l) / 128 < m) ++klo;
  return kt - klo;
}
__device__ __forceinline__ int ld_acquire_gpu(const int32_t* ptr) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(int32_t* ptr, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(ptr), "r"(v) : "memory");
}

// Shared memory of one CTA (dynamic, from a 1024-byte boundary; the kernel has no static shared memory, so that the 8-bit route
// at d = 128 fits the 227 KB to the byte).
struct BwdMisc {
  uint64_t bars[BB_COUNT];
  uint32_t tmem_base;
  int abort;
  BTile tile[2];            // the items in flight (written by the producer, item k in slot k & 1)
  // ring B's scalars [stage][half]: Q's and dO's factors of the half's two 32-query blocks, their UE8M0 bytes (Q's two, dO's two) and four times
  // the exponent of the query tile's pre-scale, as bytes. Read
  // from global memory by the producer: a load that misses in a compute warp stalls it at its next scoreboard wait (every
  // second iteration, by 700 clocks), whatever the distance to the value's use.
  alignas(16) float scal[2][2][8];
  // block factors of the item's four key blocks, K's then V's [slot]: read ahead by the producer for the same reason (from global memory they
  // stood 700 clocks in front of an item's first scores)
  alignas(16) float kfac[2][8];
};
template <int D, bool FP4, bool TL>
struct BwdSmem {
  static constexpr int TILE = 128 * D;
  static constexpr int A_TILE = FP4 ? 8192 : TILE;                  // the score operand: Q, or its NVFP4 copy
  static constexpr bool EPI2 = D == 128 && !FP4 && !TL;             // a second way out for the gradient rows, see the item epilogue
  static constexpr int K = 0;                                       // 2 buffers (items alternate)
  static constexpr int V = K + 2 * TILE;                            // 2 buffers
  static constexpr int DO = V + 2 * TILE;                           // 2 stages
  static constexpr int A = DO + 2 * TILE;                           // 3 stages
  static constexpr int Q = FP4 ? A + 3 * A_TILE : A;                // FP4: the E4M3 Q tiles (dK), 2 stages; else the A ring
  static constexpr int DS = Q + (FP4 ? 2 : 3) * TILE;               // per half: 128 key rows x 64 query bytes, 64 B swizzle
  static constexpr int DQ = DS + 2 * 8192;                          // per half: 128 head-dim rows x 64 queries f16, 128 B swizzle
  static constexpr int OUT = DQ + 2 * 16384;                        // gradient rows' way out: EPI2 or d = 64, 2 x 16 KB
  static constexpr int K4 = OUT + ((EPI2 || D == 64) ? 2 * 16384 : 0);   // FP4: NVFP4 K tiles, 2 x 8 KB
  static constexpr int SF = K4 + (FP4 ? 2 * 8192 : 0);              // FP4: scale atoms, K 2 x 1 KB then Q 3 x 1 KB
  static constexpr int VEC = SF + (FP4 ? 5 * 1024 : 0);             // 2 stages x 2 halves x {lse_log2[64], D''[64]; TL: f_Q[64], f_dO[64]}
  static constexpr int VEC_HALF = TL ? 1024 : 512;
  // per half three scale atoms of 512 bytes (dK's A side, dQ's query side, P-hat's), written by the compute warps and copied by
  // the issuer. EPI2: inside the half's own part of OUT, in use only between an item's last product and the next item's first dS.
  static constexpr int ATOM_STRIDE = EPI2 ? 16384 : 1536;
  static constexpr int ATOMS = EPI2 ? OUT : VEC + 4 * VEC_HALF;
  static constexpr int MISC = EPI2 ? VEC + 4 * VEC_HALF : ATOMS + 2 * ATOM_STRIDE;
  static constexpr int BYTES = MISC + 1024;
  static_assert(sizeof(BwdMisc) <= 1024 && BYTES <= 227 * 1024);
};

// Queries per compute warpgroup, and with them the number of compute warpgroups. Two of 64 queries are enough where an iteration
// is a chain of hand-overs (four lost 6 % to narrower loads and more arrivals). The row-local dQ side adds a warp reduction per
// column: two warps a scheduler no longer cover its latencies, four of 32 queries do (b2 s4096 h16/4, one B200: row-local
// 379 -> 292 us, token-local 456 -> 420), and the code of one query block is half as long (59 KB instead of 61 with a rolled loop).
constexpr int bwd_qw(int var) { return var >= 1 ? 32 : 64; }
constexpr int bwd_threads(int var) { return (128 / bwd_qw(var) + 2) * 128; }     // + the dQ reduction, + issuers and producer

// FULL: the variants that also serve the rarer call forms (deterministic dQ order, per-query-row pre-scale, packed
// outputs, the dK mantissa factor), each behind a run-time check of its pointer. A template flag, so that the kernels
// of the plain calls carry none of that code: the loop is sensitive to every register and instruction added to it.
template <int D, bool FP4, int VAR, bool SC, bool FULL = false>
__global__ void __launch_bounds__(bwd_threads(VAR), 1)
bwd_kernel_pipelined(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ CUtensorMap tm_acc, const __grid_constant__ CUtensorMap tm_q4,
                     const __grid_constant__ CUtensorMap tm_k4, const __grid_constant__ CUtensorMap tm_dk,
                     const __grid_constant__ CUtensorMap tm_dv, const BwdParams p) {
  using SM = BwdSmem<D, FP4, (VAR >= 2)>;
  constexpr int TILE_BYTES = 128 * D;
  constexpr uint64_t OP_SWZ = (D == 128) ? SWZ_128 : SWZ_64;     // operand tiles: rows of D bytes
  constexpr uint32_t OP_SBO = 8 * D;
  constexpr bool EPI2 = SM::EPI2;
  extern __shared__ __align__(1024) uint8_t smem[];
  BwdMisc& misc = *reinterpret_cast<BwdMisc*>(smem + SM::MISC);
  uint64_t* const bars = misc.bars;
  BTile* const tile_s = misc.tile;
  constexpr bool RL = VAR >= 1, TL = VAR >= 2, FOLD = VAR == 3;
  constexpr int QW = bwd_qw(VAR), NQ = QW / 32, NWG = 128 / QW;      // queries, query blocks per warpgroup; warpgroups
  // Who gives a K / V buffer and its slot of tile_s back: the compute warps (gradient rows written, slot no longer read), each warp of
  // the reduction and each issuer (slot read; an item without query tiles does not hold these up, and an ordered dQ can keep the
  // reduction behind). One thread a compute warpgroup is enough where the warps work on a copy of the slot (two warpgroups; what
  // they write through the buffer is stored behind a barrier of the warpgroup) and is kept for the plain 8-bit route (every warp: b4 s4096 h16 914 -> 930 us);
  // the others are faster with an arrival per warp, spills go (d = 64 b8 s1000 209 -> 201 us, token scales b2 s8192 4900 -> 4350).
  constexpr bool KVE_EACH = !(NWG == 2 && SM::EPI2);
  constexpr int N_KVE = (KVE_EACH ? 4 * NWG : NWG) + 4 + (FP4 ? 2 : 3);
  constexpr int W_RED = 4 * NWG, W_GRAD = W_RED + 4, W_PROD = W_RED + 5, W_S = W_RED + 6, W_DP = W_RED + 7;    // warps

  if (smem_u32(smem) & 1023) {           // (never the case without static shared memory; the swizzles depend on it)
    if (threadIdx.x == 0 && p.ctl.status) atomicCAS(p.ctl.status, 0, FL_DEV_WAIT_TIMEOUT | 63);
    return;
  }
  // (the warp index through a shuffle: the compiler then knows that it is the same in all lanes)
  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
  const int G = gridDim.x, cta = blockIdx.x;
  const int grp = p.grp;
  int n_items = p.n_items;

  if (tid == W_PROD * 32) {
    misc.abort = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars[BB_KV + i], 1); mbar_init(&bars[BB_KVE + i], N_KVE);
      mbar_init(&bars[BB_BFULL + 2 * i], 1); mbar_init(&bars[BB_BEMPTY + 2 * i], 1);
      mbar_init(&bars[BB_BFULL + 2 * i + 1], 1); mbar_init(&bars[BB_BEMPTY + 2 * i + 1], 1);
      mbar_init(&bars[BB_S + i], 1); mbar_init(&bars[BB_DP + i], 1);
      mbar_init(&bars[BB_GRANT + i], 2 * NWG); mbar_init(&bars[BB_DS + i], 2 * NWG);      // one arrival per warp of the half
      mbar_init(&bars[BB_DQF + i], 1); mbar_init(&bars[BB_DQE + i], 4);
      mbar_init(&bars[BB_EPI + i], 4); mbar_init(&bars[BB_EPI + 2 + i], 4);      // [warpgroup]
      mbar_init(&bars[BB_EPX + i], EPI2 ? 2 * NWG : 1);
    }
    for (int i = 0; i < 3; ++i) { mbar_init(&bars[BB_AFULL + i], 1); mbar_init(&bars[BB_AEMPTY + i], 1); }
    mbar_init(&bars[BB_R1], 4);
    mbar_init(&bars[BB_R2], 4);
    mbar_init(&bars[BB_ACC], 1);
    mbar_init(&bars[BB_ACCFREE], 4 * NWG);
    mbar_init(&bars[BB_SDR], 2 * NWG);
    mbar_init(&bars[BB_ROT], 8);
    fence_barrier_init();
    tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_acc); tma_prefetch_desc(&tm_dk); tma_prefetch_desc(&tm_dv);
    if (FP4) { tma_prefetch_desc(&tm_q4); tma_prefetch_desc(&tm_k4); }
    grid_dependency();                     // (the others wait at the barrier below)
  }
  if (warp == 0) {
    tmem_alloc(&misc.tmem_base, 512);
    tmem_relinquish();
  }
  if (!EPI2) {      // (atom bytes that nobody writes are scale 1; with EPI2 no product looks at them)
    for (int i = tid; i < 2 * SM::ATOM_STRIDE / 4; i += bwd_threads(VAR)) reinterpret_cast<uint32_t*>(smem + SM::ATOMS)[i] = 0x7F7F7F7Fu;
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (FULL && p.work) n_items = *reinterpret_cast<const volatile int*>(&p.work_head->y) * p.h_kv;
  const uint32_t tmem = misc.tmem_base;
  volatile int* abortp = &misc.abort;
  // (a status word already set by an earlier launch is not looked at: a kernel that runs after one that gave up does no harm)

  // registers per warpgroup: 2 x 176 + 2 x 80 (= the launch's 512 x 128 / 128), or 4 x 96 + 2 x 48 (= 768 x 80 / 128)
  if (warp >= W_RED) reg_dealloc<NWG == 2 ? 80 : 48>();
  if (warp == W_PROD) {
    // =================================================================== TMA producer
    if (lane == 0) {
      int gi = 0;                          // query-tile iterations issued so far, over all items
      bool ok = true;
      for (int k = 0; ok; ++k) {
        const int L = bwd_item(k, G, cta, p.zigzag);
        if (L >= n_items) break;
        const int kb = k & 1;
        // the buffers of item k - 2 (and its slot of tile_s) are free once the compute warpgroups have written its
        // gradient rows out of them and every other role has read the slot
        if (k >= 2 && !(ok = mbar_wait(&bars[BB_KVE + kb], ((k >> 1) - 1) & 1, p.ctl, abortp, 11))) break;
        BTile t;
        bwd_decode<FULL>(p, L, t);
        tile_s[kb] = t;
        if (t.nk > 0) {
          tma_load_4d(smem + SM::K + kb * TILE_BYTES, &tm_k, &bars[BB_KV + kb], 0, t.hkv, t.k0, t.bat);
          tma_load_4d(smem + SM::V + kb * TILE_BYTES, &tm_v, &bars[BB_KV + kb], 0, t.hkv, t.k0, t.bat);
          if (FP4) {
            tma_load_4d(smem + SM::K4 + kb * 8192, &tm_k4, &bars[BB_KV + kb], 0, t.hkv, t.k0, t.bat);
            bulk_load(smem + SM::SF + kb * 1024, p.sfk4 + (((size_t)t.bat * p.h_kv + t.hkv) * (p.s_k / 128) + t.k0 / 128) * 1024,
                      1024, &bars[BB_KV + kb]);
          }
        }
        if (!TL) {
          const size_t at = ((size_t)t.bat * p.h_kv + t.hkv) * (p.s_k / 32) + t.k0 / 32;
          float f[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) { f[i] = __ldg(p.fac_k + at + i); f[4 + i] = __ldg(p.fac_v + at + i); }
#pragma unroll
          for (int i = 0; i < 8; ++i) misc.kfac[kb][i] = f[i];
        }
        // (the loads are on their way: what they bring is expected with the arrival, which also makes the slot visible)
        if (t.nk > 0) mbar_arrive_expect_tx(&bars[BB_KV + kb], 2 * TILE_BYTES + (FP4 ? 8192 + 1024 : 0));
        else mbar_arrive(&bars[BB_KV + kb]);  // an empty tile slot: the phase still completes, every role moves on
        const int n_it = t.n_m * grp;
        int head = t.hkv * grp, m = t.m_lo;
        for (int it = 0; it < n_it; ++it, ++gi) {
          // ring A: the scores' query operand, three stages of a whole query tile. Ring B: dO, the row vectors, FP4: the E4M3 Q; two
          // stages in halves of 64 queries, each given back when its half is done: a whole period to load the next one in
          // (as whole tiles it was half a period, less than a load takes)
          const int sa = gi % 3, ra = gi / 3, sb = gi & 1, rb = gi >> 1;
          const int qrow = t.q0 + m * 128;
          const size_t ro = ((size_t)t.bat * p.h + head) * p.s_q + qrow;
          float4 fq = {1.f, 1.f, 1.f, 1.f}, fd = {1.f, 1.f, 1.f, 1.f};       // token-local: unit block factors
          float bsc = 1.f;
          if (!TL) {
            fq = __ldg(reinterpret_cast<const float4*>(p.fac_q + ro / 32));
            fd = __ldg(reinterpret_cast<const float4*>(p.fac_do + ro / 32));
          }
          if (!(FULL && p.dq_scale_rows)) bsc = __ldg(p.dq_scale + (size_t)t.bat * (p.s_q / 128) + qrow / 128);
          if (gi >= 3 && !(ok = mbar_wait(&bars[BB_AEMPTY + sa], (ra - 1) & 1, p.ctl, abortp, 10))) break;
          mbar_arrive_expect_tx(&bars[BB_AFULL + sa], SM::A_TILE + (FP4 ? 1024 : 0));
          tma_load_4d(smem + SM::A + sa * SM::A_TILE, FP4 ? &tm_q4 : &tm_q, &bars[BB_AFULL + sa], 0, head, qrow, t.bat);
          if (FP4)
            bulk_load(smem + SM::SF + 2048 + sa * 1024, p.sfq4 + (((size_t)t.bat * p.h + head) * (p.s_q / 128) + qrow / 128) * 1024,
                      1024, &bars[BB_AFULL + sa]);
#pragma unroll 1
          for (int x = 0; x < 2; ++x) {
            uint64_t* const full = &bars[BB_BFULL + 2 * sb + x];
            if (gi >= 2 && !(ok = mbar_wait(&bars[BB_BEMPTY + 2 * sb + x], (rb - 1) & 1, p.ctl, abortp, 10))) break;
            float* const sc = misc.scal[sb][x];
            *reinterpret_cast<float4*>(sc) = x == 0 ? make_float4(fq.x, fq.y, fd.x, fd.y) : make_float4(fq.z, fq.w, fd.z, fd.w);
            auto e8 = [](float f) { return (__float_as_uint(f) >> 23) & 0xFF; };
            const uint32_t lb = (e8(bsc) - 127u) & 0xFF;
            sc[4] = __uint_as_float(x == 0 ? e8(fq.x) | e8(fq.y) << 8 | e8(fd.x) << 16 | e8(fd.y) << 24
                                           : e8(fq.z) | e8(fq.w) << 8 | e8(fd.z) << 16 | e8(fd.w) << 24);
            sc[5] = __uint_as_float(lb * 0x01010101u);
            mbar_arrive_expect_tx(full, TILE_BYTES / 2 + SM::VEC_HALF + (FP4 ? TILE_BYTES / 2 : 0));
            const int half = sb * TILE_BYTES + x * (TILE_BYTES / 2), vec = SM::VEC + (2 * sb + x) * SM::VEC_HALF;
            bulk_load(smem + vec, p.lse_log2 + ro + 64 * x, 256, full);
            tma_load_4d(smem + SM::DO + half, &tm_do, full, 0, head, qrow + 64 * x, t.bat);
            if (FP4) tma_load_4d(smem + SM::Q + half, &tm_q, full, 0, head, qrow + 64 * x, t.bat);
            bulk_load(smem + vec + 256, p.d_rows + ro + 64 * x, 256, full);
            if (TL) {
              bulk_load(smem + vec + 512, p.fac_q + ro + 64 * x, 256, full);
              bulk_load(smem + vec + 768, p.fac_do + ro + 64 * x, 256, full);
            }
          }
          if (!ok) break;
          if (++m == t.m_lo + t.n_m) { m = t.m_lo; ++head; }
        }
      }
    }
  } else if (warp == W_GRAD) {
    // =================================================================== UMMA issuer of the gradient products
    // The whole warp stays converged through the waits and the descriptor arithmetic (warp-uniform values); one elected
    // lane issues. Descriptors are built once; the loops only add byte offsets. Three warps issue (this one dQ^T, dV, dK; the
    // others S^T and dP^T): alone, one warp's waits and descriptor moves took longer than the products. Each loop exists once, with the
    // half as a run-time value: the roles' loops share the instruction cache.
    const uint32_t tm = __shfl_sync(0xFFFFFFFFu, tmem, 0);
    const uint32_t base = smem_u32(smem);
    const uint64_t dQ0 = smem_desc(base + SM::Q, 16, OP_SBO, OP_SWZ), dDO0 = smem_desc(base + SM::DO, 16, OP_SBO, OP_SWZ),
                   dDS0 = D == 128 ? smem_desc(base + SM::DS, 16, 512, SWZ_64)
                                   : smem_desc(base + SM::DS, 8192, 512, SWZ_64),   // d = 64: dS-hat as A, next M block 8 KB further
                   dAT0 = smem_desc(base + SM::ATOMS, 0, 128, SWZ_NONE), dK0 = smem_desc(base + SM::K, 16, OP_SBO, OP_SWZ);
    int gi = 0;
    bool ok = true;
    for (int k = 0; ok; ++k) {
      const int L = bwd_item(k, G, cta, p.zigzag);
      if (L >= n_items) break;
      const int kb = k & 1;
      if (!(ok = mbar_wait(&bars[BB_KV + kb], (k >> 1) & 1, p.ctl, abortp, 20))) break;
      const int n_it = tile_s[kb].n_m * grp;
      mbar_arrive_warp(&bars[BB_KVE + kb]);
      const uint64_t dK_k = desc_adv(dK0, kb * TILE_BYTES);
      // the first products of an item overwrite dV / dK: the previous item's rows must have left tensor memory (an item without
      // query tiles issues nothing, but its accumulator hand-over still takes place once)
      if (k > 0 && !(ok = mbar_wait(&bars[BB_ACCFREE], (k - 1) & 1, p.ctl, abortp, 25))) break;
#pragma unroll 1
      for (int t = 0; t < 2 * n_it; ++t) {
        const int g = gi + (t >> 1), x = t & 1, sa = g % 3, sb = g & 1;
        // dQ^T_x, dV, dK of iteration g (P-hat and dS-hat of half x stand in the other half's region); dQ^T first: the reduction
        // warps read it while the rest runs, and dP^T_x of the next iteration takes its columns
        const uint32_t ro = tm + TC_S + 64 * (1 - x), t_dq = tm + TC_DP + 64 * x;
        const uint64_t qx = desc_adv(dQ0, (FP4 ? sb : sa) * TILE_BYTES + x * 64 * D), dox = desc_adv(dDO0, sb * TILE_BYTES + x * 64 * D),
                       at = desc_adv(dAT0, x * SM::ATOM_STRIDE), dsx = desc_adv(dDS0, x * 8192);
        uint64_t* const b_free = &bars[BB_BEMPTY + 2 * sb + x];
        if (!(ok = mbar_wait(&bars[BB_DS + x], g & 1, p.ctl, abortp, 24))) break;
        tc_fence_after();
        if (elect_one()) {
          tmem_cp_sf_atom(ro + TO_SFB_DQ, desc_adv(at, 512));
          tmem_cp_sf_atom(ro + TO_SFA_DK, at);
          if (TL) tmem_cp_sf_atom(ro + TO_SFA_P, desc_adv(at, 1024));
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {   // K = 128 keys
            if (D == 128)      // A = K tile (M = head dim), B = dS-hat half (N = 64 queries)
              umma_mxf8_ss(t_dq, desc_adv(dK_k, kk * 32 * D), desc_adv(dsx, kk * 2048), idesc_bs(128, 64, 0, 0, 1, 1, 1, kk, kk),
                           ro + TO_SFA_DQ, ro + TO_SFB_DQ, kk > 0);
            else               // A = dS-hat half (M = 64 queries + 64 unused rows), B = K tile (N = head dim)
              umma_mxf8_ss(t_dq, desc_adv(dsx, kk * 2048), desc_adv(dK_k, kk * 32 * D), idesc_bs(128, 64, 0, 0, 1, 1, 1, kk, kk),
                           ro + TO_SFB_DQ, ro + TO_SFA_DQ, kk > 0);
          }
          tc_commit(&bars[BB_DQF + x]);
#pragma unroll
          for (int kk = 0; kk < 2; ++kk)     // K = 64 queries: two instructions of 32
            umma_mxf8_ts(tm + TC_DV, ro + TO_P + 8 * kk, desc_adv(dox, kk * 32 * D),
                         idesc_bs(128, D, 0, 0, 0, 1, 1, kk, kk), ro + TO_SFA_P, ro + TO_SFB_DO, t | kk);
#pragma unroll
          for (int kk = 0; kk < 2; ++kk)
            umma_mxf8_ts(tm + TC_DK, ro + TO_DS + 8 * kk, desc_adv(qx, kk * 32 * D),
                         idesc_bs(128, D, 0, 0, 0, 1, 1, kk, kk), ro + TO_SFA_DK, ro + TO_SFB_Q, t | kk);
          tc_commit(b_free);
          if (x == 1) tc_commit(&bars[BB_AEMPTY + sa]);
        }
        __syncwarp();
      }
      if (!ok) break;
      if (elect_one()) tc_commit(&bars[BB_ACC]);       // every product of the item has completed when this arrives
      __syncwarp();
      gi += n_it;
    }
  } else if (warp == W_S || (!FP4 && warp == W_DP)) {
    // =================================================================== UMMA issuer of the score products
    // Step t of an item (y = t & 1, j = t >> 1) follows the gradient products of (j, y) and issues S^T_{1-y} of iteration
    // j + 1 + y and dP^T_y of iteration j + 1; steps -3 to -1 are the item's first products, which run while the compute
    // warpgroups write the previous item's rows. One warp issues S^T, one dP^T: dP^T_y goes out as soon as dQ^T_y has been read
    // out of its columns (the longest chain of an iteration: dS -> dQ^T -> read -> dP^T -> dS), whatever S^T waits for. FP4: one
    // warp, S^T first, because its scale columns stand in dP^T's.
    const bool role_s = FP4 || warp == W_S, role_p = FP4 || warp == W_DP;
    constexpr uint32_t ID_N64 = idesc_f8(128, 64, 0, 0);
    const uint32_t tm = __shfl_sync(0xFFFFFFFFu, tmem, 0);
    const uint32_t base = smem_u32(smem);
    const uint64_t dA0 = FP4 ? smem_desc(base + SM::A, 16, 512, SWZ_64) : smem_desc(base + SM::A, 16, OP_SBO, OP_SWZ),
                   dDO0 = smem_desc(base + SM::DO, 16, OP_SBO, OP_SWZ), dSF0 = smem_desc(base + SM::SF, 0, 128, SWZ_NONE),
                   dK0 = FP4 ? smem_desc(base + SM::K4, 16, 512, SWZ_64) : smem_desc(base + SM::K, 16, OP_SBO, OP_SWZ),
                   dV0 = smem_desc(base + SM::V, 16, OP_SBO, OP_SWZ);
    int gi = 0, sdr = 0;                   // iterations so far; uses of BB_SDR so far
    bool ok = true;
    for (int k = 0; ok; ++k) {
      const int L = bwd_item(k, G, cta, p.zigzag);
      if (L >= n_items) break;
      const int kb = k & 1;
      if (!(ok = mbar_wait(&bars[BB_KV + kb], (k >> 1) & 1, p.ctl, abortp, 21))) break;
      const int n_it = tile_s[kb].n_m * grp;
      mbar_arrive_warp(&bars[BB_KVE + kb]);
      const uint64_t dK_k = desc_adv(dK0, kb * (FP4 ? 8192 : TILE_BYTES)), dV_k = desc_adv(dV0, kb * TILE_BYTES);
#pragma unroll 1
      for (int t = -3; t < 2 * n_it - 2; ++t) {
        const int y = t & 1, j = t >> 1;
        const bool do_s = role_s && j + 1 + y < n_it, do_p = role_p && j + 1 >= 0 && j + 1 < n_it;
        const int gs = gi + j + 1 + y, gp = gi + j + 1, xs = 1 - y;
        // the half's dP^T columns hold its previous dQ^T until the reduction warps have read it. FP4: the 16 scale columns of S^T
        // stand in them, too
        auto dq_read = [&](int g) -> bool { return g == 0 || mbar_wait(&bars[BB_DQE + y], (g - 1) & 1, p.ctl, abortp, 22); };
        // The region S^T goes to: its last user were the gradient products of (j, y) (their completion also says that the scores
        // before have been read: the P-hat that took their place waited for that); at an item's start those of the item
        // before, and for half 0's second tile its own first scores.
        if (role_s && t != -2) {
          const int gl = t >= 0 ? gi + j : gi - 1;
          if (t == -1) { if (do_s && !(ok = mbar_wait(&bars[BB_SDR], sdr++ & 1, p.ctl, abortp, 26))) break; }
          else if (gl >= 0 && !(ok = mbar_wait(&bars[BB_BEMPTY + 2 * (gl & 1) + y], (gl >> 1) & 1, p.ctl, abortp, 28))) break;
        }
        if (FP4 && !(ok = dq_read(t == -3 ? gi : gp))) break;
        if (do_s) {
          const int st = gs % 3;
          // (the second half finds the stage loaded: the first half's product of the same iteration was issued before)
          if (xs == 0 && !(ok = mbar_wait(&bars[BB_AFULL + st], (gs / 3) & 1, p.ctl, abortp, 21))) break;
          tc_fence_after();
          const uint64_t ax = desc_adv(dA0, st * SM::A_TILE + xs * (SM::A_TILE / 2));
          const uint32_t t_s = tm + TC_S + 64 * xs, park = tm + TC_DP + 64 * y;
          const uint64_t sfk = desc_adv(dSF0, kb * 1024), sfq = desc_adv(dSF0, 2048 + st * 1024);
          if (elect_one()) {
            if (FP4) {
#pragma unroll
              for (int kk = 0; kk < 2; ++kk) {
                tmem_cp_sf_atom(park + 4 * kk, desc_adv(sfk, 512 * kk));
                tmem_cp_sf_atom(park + 8 + 4 * kk, desc_adv(sfq, 512 * kk));
              }
#pragma unroll
              for (int kk = 0; kk < 2; ++kk)   // K = 64 elements = 32 bytes per instruction
                umma_nvf4_ss(t_s, desc_adv(dK_k, 32 * kk), desc_adv(ax, 32 * kk), idesc_bs(128, 64, 1, 1, 0, 0, 0, 0, 0), park + 4 * kk,
                             park + 8 + 4 * kk + 2 * xs, kk > 0);
            } else {
#pragma unroll
              for (int kk = 0; kk < D / 32; ++kk) umma_f8_ss(t_s, desc_adv(dK_k, 32 * kk), desc_adv(ax, 32 * kk), ID_N64, kk > 0);
            }
            tc_commit(&bars[BB_S + xs]);
          }
          __syncwarp();
        }
        if (do_p) {
          const int st = gp & 1;
          if (!FP4 && !(ok = dq_read(gp))) break;
          if (!(ok = mbar_wait(&bars[BB_BFULL + 2 * st + y], (gp >> 1) & 1, p.ctl, abortp, 27))) break;
          // Half 1's P-hat and dS-hat go to the region that the products of (gp - 1, 1) read last. Otherwise the grant of the scores in
          // between says that they have (S^T is issued behind them); an item's last iteration has none, and dP^T waits in their
          // stead. (Waiting in the compute warps cost the 8-bit kernel 2 %: b4 s4096 h16 step 917 -> 931 us; here 909 -> 912, within noise.)
          if (y == 1 && j >= 0 && j + 2 == n_it && !(ok = mbar_wait(&bars[BB_BEMPTY + 2 * (st ^ 1) + 1], ((gp - 1) >> 1) & 1, p.ctl, abortp, 29))) break;
          tc_fence_after();
          const uint64_t doy = desc_adv(dDO0, st * TILE_BYTES + y * 64 * D);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < D / 32; ++kk)
              umma_f8_ss(tm + TC_DP + 64 * y, desc_adv(dV_k, 32 * kk), desc_adv(doy, 32 * kk), ID_N64, kk > 0);
            tc_commit(&bars[BB_DP + y]);
          }
          __syncwarp();
        }
      }
      gi += n_it;
    }
  } else if (warp >= W_RED && warp < W_GRAD) {
    // =================================================================== dQ reduction (thread = head-dim row)
    const int r = tid & 127;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    bool ok = true;
    int gi = 0, gt = 0;                     // iterations and half steps so far, over all items
    for (int k = 0; ok; ++k) {
      const int L = bwd_item(k, G, cta, p.zigzag);
      if (L >= n_items) break;
      const int kb = k & 1;
      if (!(ok = mbar_wait(&bars[BB_KV + kb], (k >> 1) & 1, p.ctl, abortp, 43))) break;
      const BTile T = tile_s[kb];
      mbar_arrive_warp(&bars[BB_KVE + kb]);
      const int n_it = T.n_m * grp;
      int head = T.hkv * grp, m = T.m_lo;
#pragma unroll 1
      for (int t = 0; t < 2 * n_it; ++t, ++gt) {
        const int it = t >> 1, y = t & 1, g = gi + it;
        if (t > 0 && y == 0 && ++m == T.m_lo + T.n_m) { m = T.m_lo; ++head; }
        // the staging buffer of this half was last read by the reduction of step gt - 2
        if (tid == W_RED * 32) tma_store_wait_read<1>();
        mbar_arrive_warp(&bars[BB_R1]);
        if (!(ok = mbar_wait(&bars[BB_R1], gt & 1, p.ctl, abortp, 41))) break;
        if (!(ok = mbar_wait(&bars[BB_DQF + y], g & 1, p.ctl, abortp, 40))) break;
        tc_fence_after();
        const uint32_t rowp = smem_u32(smem) + SM::DQ + y * 16384 + r * 128;
        // d = 128: thread = head-dim row of dQ^T, 64 query columns. d = 64: thread = query row (the first 64 lanes; the
        // other two warps hold the product's unused rows), 64 head-dim columns. Either way 64 f16 = one 128-byte row.
        if (D == 128 || warp < W_RED + 2) {
          uint32_t v[64], w[32];
          auto narrow = [&](int n) {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              if (e >= n) continue;
              __half2 hh = __floats2half2_rn(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
              w[e] = *reinterpret_cast<uint32_t*>(&hh);
            }
          };
          const uint32_t t_dq = lane_base + TC_DP + 64 * y;
          if constexpr (NWG == 2) {
            FL_TMEM_LD_32(t_dq, v);
            FL_TMEM_LD_32(t_dq + 32, (v + 32));
            tc_wait_ld();
          } else {                             // (48 registers: half the columns at a time)
            FL_TMEM_LD_32(t_dq, v);
            tc_wait_ld();
            narrow(16);
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4)     // 8 f16 = 16 bytes per chunk; 128 B swizzle by the row
              sts128(rowp + ((q4 ^ (r & 7)) << 4), w[4 * q4], w[4 * q4 + 1], w[4 * q4 + 2], w[4 * q4 + 3]);
            FL_TMEM_LD_32(t_dq + 32, v);
            tc_wait_ld();
          }
          tc_fence_before();                   // the columns go back (to dP^T) before the rows are stored
          mbar_arrive_warp(&bars[BB_DQE + y]);
          narrow(NWG == 2 ? 32 : 16);
          constexpr int Q0 = NWG == 2 ? 0 : 4;
#pragma unroll
          for (int q4 = Q0; q4 < 8; ++q4)
            sts128(rowp + ((q4 ^ (r & 7)) << 4), w[4 * (q4 - Q0)], w[4 * (q4 - Q0) + 1], w[4 * (q4 - Q0) + 2], w[4 * (q4 - Q0) + 3]);
        } else {
          tc_fence_before();
          mbar_arrive_warp(&bars[BB_DQE + y]);
        }
        fence_proxy_async();
        mbar_arrive_warp(&bars[BB_R2]);
        if (!(ok = mbar_wait(&bars[BB_R2], gt & 1, p.ctl, abortp, 42))) break;
        const bool det = FULL && p.dq_order != nullptr;
        if (!det) {
          if (tid == W_RED * 32) {
            if (D == 128) tma_reduce_add_4d(&tm_acc, smem + SM::DQ + y * 16384, T.q0 + m * 128 + 64 * y, 0, head, T.bat);
            else tma_reduce_add_4d(&tm_acc, smem + SM::DQ + y * 16384, 0, T.q0 + m * 128 + 64 * y, head, T.bat);
            tma_store_commit();
          }
        } else if (warp == W_RED) {              // (the whole warp stays converged: lane 0 works, the others follow its result)
          int go = 1;
          int32_t* order = nullptr;
          int rank = 0;
          {
            // deterministic order: the key tiles before this one have added their partial sums of this half
            order = p.dq_order + ((((size_t)T.bat * p.h + head) * (p.s_q / 128) + T.q0 / 128 + m) * 2 + y);
            rank = bwd_order_rank(p, T, m);
            if (lane == 0) {
              const long long t_start = clock64();
              while (ld_acquire_gpu(order) != rank) {
                if (*abortp || clock64() - t_start > p.ctl.wait_cycles) {
                  if (!*abortp) *abortp = 44;
                  go = 0;
                  break;
                }
              }
            }
            go = __shfl_sync(0xFFFFFFFFu, go, 0);
          }
          if (go && lane == 0) {
            if (D == 128) tma_reduce_add_4d(&tm_acc, smem + SM::DQ + y * 16384, T.q0 + m * 128 + 64 * y, 0, head, T.bat);
            else tma_reduce_add_4d(&tm_acc, smem + SM::DQ + y * 16384, 0, T.q0 + m * 128 + 64 * y, head, T.bat);
            tma_store_commit();
            if (order) {
              tma_store_wait<0>();                // the addition has completed, not only read its source
              __threadfence();
              st_release_gpu(order, rank + 1);
            }
          }
          __syncwarp();
          if (!go) ok = false;           // the other warps of the group see the flag at their next wait
        }
        if (!ok) break;
      }
      gi += n_it;
    }
    if (tid == W_RED * 32) tma_store_wait<0>();
  } else if (warp < W_RED) {
    reg_alloc<NWG == 2 ? 176 : 96>();
    // =================================================================== compute (thread = key row, QW query columns)
    const int x = warp / (2 * NWG);                  // the half this warpgroup works for
    const int qb = NWG == 2 ? 0 : (warp >> 2) & 1;   // its first 32-query block of the half
    const int wq = warp & 3;                         // lane quadrant = 32-key block of the tile
    const int r = wq * 32 + lane;                    // key row of the tile = TMEM lane
    const uint32_t lane_base = tmem + ((uint32_t)(wq * 32) << 16);
    const uint32_t t_sx = lane_base + TC_S + 64 * x + 32 * qb, t_dpx = lane_base + TC_DP + 64 * x + 32 * qb;
    const uint32_t t_ox = lane_base + TC_S + 64 * (1 - x);           // where P-hat, dS-hat and the scale columns go
    const uint32_t ds_row = smem_u32(smem) + SM::DS + x * 8192 + r * 64;
    // this thread's bytes of the scale atoms (row r of a 128-row atom: word (r % 32) * 4 + r / 32; query rows 0..63 likewise)
    const uint32_t at = smem_u32(smem) + SM::ATOMS + x * SM::ATOM_STRIDE;
    const uint32_t at_row = at + lane * 16 + wq * 4 + qb, at_q = at + 512 + lane * 16 + 4 * qb + wq;
    uint64_t* const bar_epi = &bars[BB_EPI + (warp >> 2)];
    bool ok = true;
    int gi = 0, epi = 0, epx = 0;                    // iterations so far; uses of the epilogue barriers so far
    [[maybe_unused]] int n_rot = 0;                                   // rotated items so far
    int cg = 0;                                      // grants used so far
    int pending_kve = -1;                            // the K / V buffer whose gradient stores are still to be confirmed
    auto free_kv = [&](int buf) {
      if (r == 0) tma_store_wait_read<0>();
      if (KVE_EACH) mbar_arrive_warp(&bars[BB_KVE + buf]);
      else if (r == 0) mbar_arrive(&bars[BB_KVE + buf]);
    };
    for (int k = 0; ok; ++k) {
      const int L = bwd_item(k, G, cta, p.zigzag);
      if (L >= n_items) break;
      const int kb = k & 1;
      if (!(ok = mbar_wait(&bars[BB_KV + kb], (k >> 1) & 1, p.ctl, abortp, 39))) break;
      const BTile Tcopy = tile_s[kb];
      const BTile& T = NWG == 4 ? tile_s[kb] : Tcopy;
      const int hkv = T.hkv;
      const int n_it = T.n_m * grp;
      const bool key_valid = r < T.nv;
      const size_t bh_k = (size_t)T.bat * p.h_kv + hkv;
      const float4 kf = lds128(smem_u32(misc.kfac[kb]));
      // token-local: this key's own factors; otherwise its 32-key block's
      const float fk_true = TL ? p.fac_k[bh_k * p.s_k + T.k0 + r] : misc.kfac[kb][wq];
      const float fk = fk_true * p.scale_log2;
      const float fv8 = (TL ? p.fac_v[bh_k * p.s_k + T.k0 + r] : misc.kfac[kb][4 + wq]) * 0.00390625f;   // f_V 2^-8
      uint32_t ek_word = TL ? 0x7F7F7F7Fu : 0u;        // UE8M0 bytes of the tile's four key blocks (unit when token-local)
      if (!TL) {
        const float k4[4] = {kf.x, kf.y, kf.z, kf.w};
#pragma unroll
        for (int kbk = 0; kbk < 4; ++kbk) ek_word |= ((__float_as_uint(k4[kbk]) >> 23) & 0xFF) << (8 * kbk);
      }
      const int krel = T.krel + r - T.off;
      const int vis_from = p.win_r >= 0 ? krel - p.win_r : 0;    // queries in [vis_from, vis_to] see this key
      const int vis_to = min(p.win_l >= 0 ? krel + p.win_l : 0x7FFFFFFF, T.sq - 1);
      int m = T.m_lo;
      for (int it = 0; it < n_it; ++it) {
        const int g = gi + it, st = g & 1;
        const int q_first = m * 128 + 64 * x + 32 * qb;                    // document-relative query of column 0
        bool full = false;
        // which of the queries see this key, a bit each (tested bit by bit the mask takes a third of the instructions that
        // comparisons take, and they stand in the loop whether they run or not)
        uint32_t see[2] = {0u, 0u};
        auto masks = [&]() {
          full = key_valid && (q_first >= vis_from) && (q_first + QW - 1 <= vis_to);
          if (!full) {
            const int lo = max(vis_from - q_first, 0), n = key_valid ? max(min(vis_to - q_first + 1, QW) - lo, 0) : 0;
            const uint64_t b = lo < QW && n > 0 ? (~0ull >> (64 - n)) << lo : 0ull;
            see[0] = (uint32_t)b;
            see[1] = (uint32_t)(b >> 32);
          }
          if (++m == T.m_lo + T.n_m) m = T.m_lo;                              // (the next iteration's from here on)
        };
        auto visible = [&](int j) { return (see[j >> 5] & (1u << (j & 31))) != 0; };
        const uint32_t v_lse = smem_u32(smem) + SM::VEC + (2 * st + x) * SM::VEC_HALF + 128 * qb, v_dpp = v_lse + 256;
        [[maybe_unused]] const uint32_t v_fq = v_lse + 512, v_fdo = v_lse + 768;      // token-local: the per-query factors
        uint32_t edo2 = 0, eq2 = 0, ekb_word = 0, lq[NQ];
        float c[NQ], b8[NQ];
        auto row_vectors = [&]() -> bool {         // they are there, and so are the half's scalars
          if (!mbar_wait(&bars[BB_BFULL + 2 * st + x], (g >> 1) & 1, p.ctl, abortp, 30)) return false;
          const float4 sc4 = lds128(smem_u32(misc.scal[st][x]));
          const float sc[4] = {sc4.x, sc4.y, sc4.z, sc4.w};
          // (the words' sixteen instructions, once in the producer: d = 64 8 x 1024 x 12 93.2 -> 91.7 us, mixed route b4 s4096 h16 503 -> 496)
          const float2 words = *reinterpret_cast<const float2*>(&misc.scal[st][x][4]);
          if constexpr (SC && D == 128) {        // from the factors (b5 s1536 h4/1 dense, mixed route 127 -> 120 us, 8-bit 120 -> 119; d = 64 +0.6 %)
            auto e8 = [](float f) { return (__float_as_uint(f) >> 23) & 0xFF; };
            eq2 = e8(sc[0]) | (e8(sc[1]) << 8);
            edo2 = e8(sc[2]) | (e8(sc[3]) << 8);
          } else {
            eq2 = __float_as_uint(words.x) & 0xFFFF;
            edo2 = __float_as_uint(words.x) >> 16;
          }
          ekb_word = __vadd4(ek_word, __float_as_uint(words.y));
#pragma unroll
          for (int qh = 0; qh < NQ; ++qh) {        // a pre-scale per query row: folded into the dQ side's B scale bytes
            lq[qh] = 0;
            if (FULL && p.dq_scale_rows)
              lq[qh] = (uint32_t)((int)((__float_as_uint(p.dq_scale_rows[(size_t)T.bat * p.s_q + T.q0 + q_first + 32 * qh + lane]) >> 23) & 0xFF) - 127);
          }
          // FP4: the block scales of S were applied by the tensor core; only the softmax scale remains
#pragma unroll
          for (int qh = 0; qh < NQ; ++qh) {
            c[qh] = FP4 ? p.scale_log2 : fk * (qb ? sc[1] : sc[qh]);
            b8[qh] = fv8 * (qb ? sc[3] : sc[2 + qh]);
          }
          return true;
        };
        // Where the scores are waited for anyway, what they are not needed for stands behind their load from tensor memory, which takes its
        // time: of an iteration of 3250 clocks the masks took 250 and the row vectors 130 (b4 s4096 h16 causal, kernel alone: 467 ->
        // 460.5 us, masks alone 462.6; dense 821 -> 809). Not where registers are short or the order of waits matters more: mixed route masks
        // alone (475 us either way, both +0.3 %), d = 64 +1 %, token-local +5 %.
        constexpr bool LATE_MASK = D == 128 && VAR == 0 && !SC, LATE_VEC = LATE_MASK && !FP4;
        if constexpr (!LATE_MASK) masks();
        if constexpr (!LATE_VEC) {
          if (!(ok = row_vectors())) break;
        }

        // ---- P' = 2^(s c - lse2)
        if (!(ok = mbar_wait(&bars[BB_S + x], g & 1, p.ctl, abortp, 31))) break;
        tc_fence_after();
        uint32_t pv[QW];
        FL_TMEM_LD_32(t_sx, pv);
        if constexpr (NQ == 2) FL_TMEM_LD_32(t_sx + 32, (pv + 32));
        if constexpr (LATE_MASK) masks();
        if constexpr (LATE_VEC) {
          if (!(ok = row_vectors())) break;
        }
        tc_wait_ld();
        // the scores are in registers: this region may take the other half's P-hat and dS-hat (half 0's iteration waits for S1 of
        // the same iteration; half 1's for S0 of the next one, which is issued before, or of this one where that was the last)
        tc_fence_before();
        if (x == 1 || it > 0 || n_it == 1) mbar_arrive_warp(&bars[BB_GRANT + (1 - x)]);
        if (x == 0 && it == 0 && n_it > 1) mbar_arrive_warp(&bars[BB_SDR]);
        float pf[QW];
        uint32_t pw[QW / 4];                   // P-hat's codes, kept until the region they go to is free
        [[maybe_unused]] uint32_t ep = 0;
        if constexpr (SC) {
          // soft cap: x = cap_a tanh(s c cap_b); P-hat is taken from P' right here, and what stays in pf is
          // P' (1 - tanh^2), the factor dS needs (the reference's score_mod_bwd, flash_attn/cute/utils.py:178-187)
#pragma unroll
          for (int j4 = 0; j4 < QW / 4; ++j4) {
            const float4 l4 = lds128(v_lse + 16 * j4);
            const float l[4] = {l4.x, l4.y, l4.z, l4.w};
            float pp[4], df[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float th = tanh_fast(__uint_as_float(pv[4 * j4 + e]) * (c[j4 >> 3] * p.cap_b));
              pp[e] = ex2(fmaf(p.cap_a, th, -l[e]));
              df[e] = fmaf(-th, th, 1.0f);
              if (!full) pp[e] = visible(4 * j4 + e) ? pp[e] : 0.f;
            }
            pw[j4] = cvt_e4m3x4(pp[0], pp[1], pp[2], pp[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) pf[4 * j4 + e] = pp[e] * df[e];
          }
        } else {
#pragma unroll
          for (int j4 = 0; j4 < QW / 4; ++j4) {
            const float4 l4 = lds128(v_lse + 16 * j4);
            // t = lse2 - s c (token-local: c = f_K f_Q(query)), two columns per instruction; P' = 2^-t
            uint64_t c01, c23;
            if (TL) {
              const float4 f4 = lds128(v_fq + 16 * j4);
              const uint64_t nfk2 = pack2(-fk, -fk);
              c01 = mul2(pack2(f4.x, f4.y), nfk2);
              c23 = mul2(pack2(f4.z, f4.w), nfk2);
            } else {
              c01 = c23 = pack2(-c[j4 >> 3], -c[j4 >> 3]);
            }
            float t0, t1, t2, t3;
            unpack2(fma2(pack2(__uint_as_float(pv[4 * j4 + 0]), __uint_as_float(pv[4 * j4 + 1])), c01, pack2(l4.x, l4.y)), t0, t1);
            unpack2(fma2(pack2(__uint_as_float(pv[4 * j4 + 2]), __uint_as_float(pv[4 * j4 + 3])), c23, pack2(l4.z, l4.w)), t2, t3);
            pf[4 * j4 + 0] = ex2_neg(t0);
            pf[4 * j4 + 1] = ex2_neg(t1);
            pf[4 * j4 + 2] = ex2_neg(t2);
            pf[4 * j4 + 3] = ex2_neg(t3);
          }
          if (!full) {      // diagonal / tail tiles only
#pragma unroll
            for (int j = 0; j < QW; ++j) pf[j] = visible(j) ? pf[j] : 0.f;
          }
          if constexpr (TL) {
            static_assert(!TL || QW == 32, "one query block per warpgroup");
            // block-scaled P-hat carrying f_dO(query): one exponent per (this key row, 32 queries). (Its atom's last reader, the dV
            // product of the iteration before, has completed when dP^T has: the byte is written below.) FOLD: pf keeps the product, else it is
            // taken again for the codes (32 registers less).
            float am = 0.f;
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              const float4 f4 = lds128(v_fdo + 16 * j4);
              const int j = 4 * j4;
              float t0, t1, t2, t3;
              unpack2(mul2(pack2(pf[j + 0], pf[j + 1]), pack2(f4.x, f4.y)), t0, t1);
              unpack2(mul2(pack2(pf[j + 2], pf[j + 3]), pack2(f4.z, f4.w)), t2, t3);
              am = fmax3_abs(fmax3_abs(am, t0, t1), t2, t3);   // all >= 0
              if (FOLD) { pf[j + 0] = t0; pf[j + 1] = t1; pf[j + 2] = t2; pf[j + 3] = t3; }
            }
            ep = exp448(__float_as_uint(am));
            const float inv = pow2_inv(ep);
            const uint64_t inv2 = pack2(inv, inv);
#pragma unroll
            for (int w = 0; w < 8; ++w) {
              float a0, a1, a2, a3;
              uint64_t t01 = pack2(pf[4 * w], pf[4 * w + 1]), t23 = pack2(pf[4 * w + 2], pf[4 * w + 3]);
              if (!FOLD) {
                const float4 f4 = lds128(v_fdo + 16 * w);
                t01 = mul2(t01, pack2(f4.x, f4.y));
                t23 = mul2(t23, pack2(f4.z, f4.w));
              }
              unpack2(mul2(t01, inv2), a0, a1);
              unpack2(mul2(t23, inv2), a2, a3);
              pw[w] = cvt_e4m3x4(a0, a1, a2, a3);
            }
          } else {
#pragma unroll
            for (int w = 0; w < QW / 4; ++w) pw[w] = cvt_e4m3x4(pf[4 * w], pf[4 * w + 1], pf[4 * w + 2], pf[4 * w + 3]);
          }
        }
        if (it == 0 && pending_kve >= 0) {
          // the previous item's gradient stores have long read their shared-memory source: its K / V buffer goes back (and, where
          // the scale atoms share the way out's memory, every warp of the half has to know)
          free_kv(pending_kve);
          pending_kve = -1;
          if (EPI2) {
            mbar_arrive_warp(&bars[BB_EPX + x]);
            if (!(ok = mbar_wait(&bars[BB_EPX + x], epx & 1, p.ctl, abortp, 38))) break;
            ++epx;
          }
        }

        // ---- dS = P' (b dP + D''), block exponent per (this warp's 32 keys, 32 queries)
        if (!(ok = mbar_wait(&bars[BB_DP + x], g & 1, p.ctl, abortp, 32))) break;
        tc_fence_after();
        FL_TMEM_LD_32(t_dpx, pv);
        if constexpr (NQ == 2) FL_TMEM_LD_32(t_dpx + 32, (pv + 32));
        tc_wait_ld();
        uint32_t ebyte[NQ];
#pragma unroll
        for (int qh = 0; qh < NQ; ++qh) {
        float am = 0.f;
#pragma unroll
        for (int j4 = 8 * qh; j4 < 8 * qh + 8; ++j4) {
          const float4 d4 = lds128(v_dpp + 16 * j4);
          const int j = 4 * j4;
          if (TL) {
            // b = f_V(key) f_dO(query) per column (FOLD: f_dO is in pf, and D'' comes divided by it); the dK side's maximum and codes
            // carry f_Q(query) (kept in pv), the dQ side's f_K(key)
            const float4 q4 = lds128(v_fq + 16 * j4);
            const uint64_t fv2 = pack2(fv8, fv8);
            uint64_t b01 = fv2, b23 = fv2;
            if (!FOLD) {
              const float4 f4 = lds128(v_fdo + 16 * j4);
              b01 = mul2(pack2(f4.x, f4.y), fv2);
              b23 = mul2(pack2(f4.z, f4.w), fv2);
            }
            const uint64_t u01 = fma2(pack2(__uint_as_float(pv[j + 0]), __uint_as_float(pv[j + 1])), b01, pack2(d4.x, d4.y));
            const uint64_t u23 = fma2(pack2(__uint_as_float(pv[j + 2]), __uint_as_float(pv[j + 3])), b23, pack2(d4.z, d4.w));
            const uint64_t p01 = mul2(pack2(pf[j + 0], pf[j + 1]), u01), p23 = mul2(pack2(pf[j + 2], pf[j + 3]), u23);
            unpack2(mul2(p01, pack2(fk_true, fk_true)), pf[j + 0], pf[j + 1]);
            unpack2(mul2(p23, pack2(fk_true, fk_true)), pf[j + 2], pf[j + 3]);
            float w0, w1, w2, w3;
            unpack2(mul2(p01, pack2(q4.x, q4.y)), w0, w1);
            unpack2(mul2(p23, pack2(q4.z, q4.w)), w2, w3);
            am = fmax3_abs(fmax3_abs(am, w0, w1), w2, w3);
            pv[j] = __float_as_uint(w0); pv[j + 1] = __float_as_uint(w1);
            pv[j + 2] = __float_as_uint(w2); pv[j + 3] = __float_as_uint(w3);
          } else {
            // two columns per instruction
            const uint64_t b2 = pack2(b8[qh], b8[qh]);
            const uint64_t u01 = fma2(pack2(__uint_as_float(pv[j + 0]), __uint_as_float(pv[j + 1])), b2, pack2(d4.x, d4.y));
            const uint64_t u23 = fma2(pack2(__uint_as_float(pv[j + 2]), __uint_as_float(pv[j + 3])), b2, pack2(d4.z, d4.w));
            unpack2(mul2(pack2(pf[j + 0], pf[j + 1]), u01), pf[j + 0], pf[j + 1]);
            unpack2(mul2(pack2(pf[j + 2], pf[j + 3]), u23), pf[j + 2], pf[j + 3]);
            am = fmax3_abs(fmax3_abs(am, pf[j], pf[j + 1]), pf[j + 2], pf[j + 3]);
          }
        }
        ebyte[qh] = exp448(warp_max_abs_f32(am));                          // 448 * 2^(e-127) >= amax
        }
        if (!full) {      // diagonal / tail tiles only
          // masked entries hold P' = 0, but their dP^T or D'' may come from rows outside the document (padding or whatever
          // the buffer held: possibly Inf / NaN), and 0 * NaN is NaN: select again after the multiply. (The maxima above
          // ignore NaN, so the block exponents are those of the visible entries.)
#pragma unroll
          for (int j = 0; j < QW; ++j) {
            pf[j] = visible(j) ? pf[j] : 0.f;
            if (TL) pv[j] = visible(j) ? pv[j] : 0u;
          }
        }
        // dK's A scales: row = key; bytes = the half's two query blocks
        if constexpr (NQ == 2) sts32(at_row, ebyte[0] | (ebyte[1] << 8));
        else sts8(at_row, ebyte[0]);
        if (TL) sts8(at_row + 1024, ep);
        uint32_t dsw[QW / 4];
#pragma unroll
        for (int qh = 0; qh < NQ; ++qh) {
          const float inv = pow2_inv(ebyte[qh]);                           // 2^(127 - e)
          const uint64_t inv2 = pack2(inv, inv);
          auto ds = [&](int j) { return TL ? __uint_as_float(pv[j]) : pf[j]; };
#pragma unroll
          for (int w = 8 * qh; w < 8 * qh + 8; ++w) {
            float a0, a1, a2, a3;
            unpack2(mul2(pack2(ds(4 * w), ds(4 * w + 1)), inv2), a0, a1);
            unpack2(mul2(pack2(ds(4 * w + 2), ds(4 * w + 3)), inv2), a2, a3);
            dsw[w] = cvt_e4m3x4(a0, a1, a2, a3);
          }
        }
        // the dQ^T product's MN-major B operand: row = key, 64 bytes = 4 chunks of 16 B, 64 B swizzle
        auto ds_rows = [&]() {
#pragma unroll
          for (int q4 = 0; q4 < 2 * NQ; ++q4)
            sts128(ds_row + (((2 * qb + q4) ^ ((r >> 1) & 3)) << 4), dsw[4 * q4], dsw[4 * q4 + 1], dsw[4 * q4 + 2], dsw[4 * q4 + 3]);
        };
        if constexpr (!RL) {
          // dQ's query-side scales: row = query; byte = this warp's key block
#pragma unroll
          for (int qh = 0; qh < NQ; ++qh) sts8(at_q + 4 * qh, ebyte[qh] + lq[qh]);
          ds_rows();
        }
        // the other half's scores must have left the region (long since, when the halves run half an iteration apart)
        if (x == 0 || it + 1 < n_it || n_it == 1) {
          if (!(ok = mbar_wait(&bars[BB_GRANT + x], cg & 1, p.ctl, abortp, 36))) break;
          ++cg;
          tc_fence_after();
        }
        {
          // dV: A = 1 (token-local: the issuer's copy of P-hat's atom follows), B = dO's exponent per 32 queries (bytes = the
          // half's two K steps); dK: B = Q's exponents; dQ^T: A[head-dim lane] = K's exponents per key block with the power-of-two
          // f16 pre-scale of the query tile folded in
          uint32_t sf[16] = {0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, edo2, edo2, edo2, edo2,
                             eq2, eq2, eq2, eq2, ekb_word, ekb_word, ekb_word, ekb_word};
          if constexpr (NQ == 2) {
            FL_TMEM_ST_16(t_ox + TO_P, pw);
            FL_TMEM_ST_16(t_ox + TO_DS, dsw);
            FL_TMEM_ST_16(t_ox + TO_SFA_P, sf);
          } else {
            FL_TMEM_ST_8(t_ox + TO_P + 8 * qb, pw);
            FL_TMEM_ST_8(t_ox + TO_DS + 8 * qb, dsw);
            if (qb == 0) FL_TMEM_ST_8(t_ox + TO_SFA_P, sf);
            else FL_TMEM_ST_8(t_ox + TO_SFB_Q, (sf + 8));
          }
        }
        if constexpr (RL) {
          static_assert(!RL || QW == 32, "one query block per warpgroup");
          // the dQ side's own codes: one exponent per (query, this warp's 32 keys); token-local: they carry f_K(key). Per column:
          // s = the bits of 2^-7 amax rounded up to the next 448 2^k, floored so that the UE8M0 byte is at least 1; the bits of
          // 2^(127 - e) are its exponent field inverted. (Integer and min / max instructions issue at half rate: the fewer per
          // column the better.) The columns' values are the same in all lanes; lane = query keeps its own by a selection tree
          // over the lane's bits (one select per column instead of a comparison and a select).
          uint32_t tree[4];
#pragma unroll
          for (int w = 0; w < 8; ++w) {
            float v[4];
            uint32_t iv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = pf[4 * w + e];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int sb = __viaddmax_s32((int)warp_max_abs_f32(v[e]), 0x00200000 - 0x03800000, 2 << 23);
              iv[e] = ~(uint32_t)sb & 0x7F800000u;
            }
            unpack2(mul2(pack2(v[0], v[1]), pack2(__uint_as_float(iv[0]), __uint_as_float(iv[1]))), v[0], v[1]);
            unpack2(mul2(pack2(v[2], v[3]), pack2(__uint_as_float(iv[2]), __uint_as_float(iv[3]))), v[2], v[3]);
            dsw[w] = cvt_e4m3x4(v[0], v[1], v[2], v[3]);
            uint32_t n = (lane & 2) ? ((lane & 1) ? iv[3] : iv[2]) : ((lane & 1) ? iv[1] : iv[0]);
            if (w & 1) {
              n = (lane & 4) ? n : tree[0];
              if ((w & 3) == 3) {
                n = (lane & 8) ? n : tree[1];
                if (w == 7) tree[3] = (lane & 16) ? n : tree[2];
                else tree[2] = n;
              } else {
                tree[1] = n;
              }
            } else {
              tree[0] = n;
            }
          }
          sts8(at_q, 254u - (tree[3] >> 23) + lq[0]);   // UE8M0 byte e: 2^(127 - e) has the exponent field 254 - e
          ds_rows();
        }
        tc_wait_st();
        fence_proxy_async();             // the dS-hat tile and the atoms in shared memory are read by the tensor core (async proxy)
        tc_fence_before();
        mbar_arrive_warp(&bars[BB_DS + x]);
      }
      if (!ok) break;
      gi += n_it;

      // ---- item epilogue: the warpgroups of half 0 write dV, those of half 1 dK (four warpgroups: half of the columns each)
      if (!(ok = mbar_wait(&bars[BB_ACC], k & 1, p.ctl, abortp, 33))) break;
      tc_fence_after();
      {
        const uint32_t t_acc = lane_base + (x == 0 ? TC_DV : TC_DK);
        // dV carries 2^8 (P'), dK the softmax scale (and the mantissa of a Q factor that is no power of two)
        const float mult = (x == 0) ? 0.00390625f : p.softmax_scale * ((FULL && p.dk_mult) ? p.dk_mult[bh_k] : 1.0f);
        const float mk = key_valid ? mult : 0.f;       // rows past the end of the document store zeros
        // dK of rotated operands: (y H / sqrt(128)) * signs. Levels 1 .. 16 of the butterfly inside the warpgroup's blocks of 32
        // columns, in place in tensor memory, then (all blocks done) levels 32 and 64 across the blocks on the way out, eight
        // columns at a time. Small loops: unrolled over a row of registers it was 900 instructions, which pushed the main loops
        // out of the instruction cache at every item.
        const bool rot = D == 128 && x == 1 && p.had_dk && n_it > 0;
        if (rot) {
#pragma unroll 1
          for (int cc = 0; cc < 8 / NWG; ++cc) {
            uint32_t v[32];
            FL_TMEM_LD_32(t_acc + 64 * qb + 32 * cc, v);
            tc_wait_ld();
            uint64_t Y[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {            // level 1: the two halves of a pair
              const float a = __uint_as_float(v[2 * i]), b2 = __uint_as_float(v[2 * i + 1]);
              Y[i] = pack2(a + b2, a - b2);
            }
#pragma unroll
            for (int hs = 1; hs < 16; hs <<= 1) {     // levels 2 .. 16: whole pairs
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                if ((i & hs) == 0) {
                  const uint64_t a = Y[i], b2 = Y[i + hs];
                  Y[i] = add2(a, b2);
                  Y[i + hs] = sub2(a, b2);
                }
              }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              float a, b2;
              unpack2(Y[i], a, b2);
              v[2 * i] = __float_as_uint(a);
              v[2 * i + 1] = __float_as_uint(b2);
            }
            FL_TMEM_ST_32(t_acc + 64 * qb + 32 * cc, v);
          }
          tc_wait_st();
          if constexpr (NWG == 4) {
            tc_fence_before();
            mbar_arrive_warp(&bars[BB_ROT]);
            if (!(ok = mbar_wait(&bars[BB_ROT], n_rot & 1, p.ctl, abortp, 37))) break;
            ++n_rot;
            tc_fence_after();
          }
        }
        // rows -> shared memory (boxes of 64 elements, 128 B swizzle) -> one TMA store per box: a thread's own row
        // written straight to global memory costs 32 separate 128-byte lines per warp instruction. At d = 128 the first
        // box goes through the finished item's K (dV) / V (dK) buffer: every product that read it has completed. The second box
        // has a buffer of its own where shared memory allows (the plain 8-bit route); otherwise it follows in the first one's.
        // Nobody waits for the stores here: the thread that issued one confirms that it has read its source, and only then
        // hands the K / V buffer back to the producer, one query tile into the next item.
        if (pending_kve >= 0) {          // (an item with fewer than two query tiles came in between)
          free_kv(pending_kve);
          pending_kve = -1;
          mbar_arrive_warp(bar_epi);
          if (!(ok = mbar_wait(bar_epi, epi & 1, p.ctl, abortp, 38))) break;
          ++epi;
        }
        const CUtensorMap* tm_out = (x == 0) ? &tm_dv : &tm_dk;
        // packed output: the key tile is slot T.k0 / 128 of the aligned buffer; its rows go to the packed rows out_row ..
        // + out_n of the caller's tensor: a full slot as TMA stores, a document's last rows row by row
        int out_row = T.k0, out_n = T.nk > 0 ? 128 : 0;
        if (FULL && p.slot_src) {
          out_row = T.nk > 0 ? p.slot_src[T.k0 / 128] : -1;
          out_n = (T.nk > 0 && out_row >= 0) ? min(p.slot_rows[T.k0 / 128], 128) : 0;
        }
        const bool by_rows = FULL && p.slot_src && out_n < 128;   // (CTA-uniform)
        uint16_t* out_base = reinterpret_cast<uint16_t*>(x == 0 ? p.dv : p.dk);
        const float cs = rot ? 0.08838834764831845f * mk : mk;
        // eight columns of both 32-column blocks of a box, finished, as words of two 16-bit values
        auto octets = [&](int bx, int c8, uint32_t (&w)[2][4]) {
          uint32_t v[2][8];
#pragma unroll
          for (int b2 = 0; b2 < 2; ++b2) {
            if (n_it > 0) FL_TMEM_LD_8(t_acc + (rot ? 0 : 64 * bx) + 32 * b2 + 8 * c8, v[b2]);   // (CTA-uniform: warp-collective loads)
            else {
#pragma unroll
              for (int e = 0; e < 8; ++e) v[b2][e] = 0;              // no query tile saw this key tile
            }
          }
          uint64_t Y[2][4];
          if (D == 128 && rot) {
            uint32_t u[2][8];
            FL_TMEM_LD_8(t_acc + 64 + 8 * c8, u[0]);
            FL_TMEM_LD_8(t_acc + 96 + 8 * c8, u[1]);
            tc_wait_ld();
            const float sg = bx == 0 ? 1.0f : -1.0f;
            const uint64_t sg2 = pack2(sg, sg);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const uint64_t l0 = pack2(__uint_as_float(v[0][2 * e]), __uint_as_float(v[0][2 * e + 1])),
                             l1 = pack2(__uint_as_float(v[1][2 * e]), __uint_as_float(v[1][2 * e + 1])),
                             h0 = pack2(__uint_as_float(u[0][2 * e]), __uint_as_float(u[0][2 * e + 1])),
                             h1 = pack2(__uint_as_float(u[1][2 * e]), __uint_as_float(u[1][2 * e + 1]));
              Y[0][e] = fma2(add2(h0, h1), sg2, add2(l0, l1));       // (the products are exact)
              Y[1][e] = fma2(sub2(h0, h1), sg2, sub2(l0, l1));
            }
          } else {
            tc_wait_ld();
#pragma unroll
            for (int b2 = 0; b2 < 2; ++b2)
#pragma unroll
              for (int e = 0; e < 4; ++e) Y[b2][e] = pack2(__uint_as_float(v[b2][2 * e]), __uint_as_float(v[b2][2 * e + 1]));
          }
#pragma unroll
          for (int b2 = 0; b2 < 2; ++b2) {
            const uint32_t neg = !rot ? 0u : (bx == 0 ? (b2 == 0 ? 0x10D2E03Eu : 0xE0D9F0E2u) : (b2 == 0 ? 0x45809F07u : 0x75954FEDu)) >> (8 * c8);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float c0 = __uint_as_float(__float_as_uint(cs) ^ ((neg << (31 - 2 * e)) & 0x80000000u)),
                          c1 = __uint_as_float(__float_as_uint(cs) ^ ((neg << (30 - 2 * e)) & 0x80000000u));
              float f0, f1;
              unpack2(mul2(Y[b2][e], pack2(c0, c1)), f0, f1);
              if (p.out_f16) {
                __half2 hh = __floats2half2_rn(f0, f1);
                w[b2][e] = *reinterpret_cast<uint32_t*>(&hh);
              } else {
                w[b2][e] = pack_bf16x2(f0, f1);
              }
            }
          }
        };
        auto stage_of = [&](int bx) -> uint8_t* {
          return smem + (D == 64 || (EPI2 && bx == 1) ? SM::OUT + x * 16384 : (x == 0 ? SM::K : SM::V) + kb * TILE_BYTES);
        };
        auto put = [&](int bx, int c8, const uint32_t (&w)[2][4]) {
#pragma unroll
          for (int b2 = 0; b2 < 2; ++b2) {
            const int ch = 8 * bx + 4 * b2 + c8;     // 16-byte chunk of the row
            if (by_rows) {
              if (r < out_n && 8 * ch < p.d_out)
                *reinterpret_cast<uint4*>(out_base + ((size_t)(out_row + r) * p.h_kv + hkv) * p.d_out + 8 * ch) =
                    make_uint4(w[b2][0], w[b2][1], w[b2][2], w[b2][3]);
            } else {
              sts128(smem_u32(stage_of(bx)) + r * 128 + (((ch & 7) ^ (r & 7)) << 4), w[b2][0], w[b2][1], w[b2][2], w[b2][3]);
            }
          }
        };
        auto announce = [&](int bx) -> bool {        // the warpgroup's four warps have written their rows: out with them
          if (by_rows) return true;
          fence_proxy_async();
          mbar_arrive_warp(bar_epi);
          if (!mbar_wait(bar_epi, epi & 1, p.ctl, abortp, 38)) return false;
          ++epi;
          if (r == 0 && out_n == 128) {
            tma_store_4d(tm_out, stage_of(bx), 64 * bx, hkv, out_row, T.bat);
            tma_store_commit();
          }
          return true;
        };
        auto free_acc = [&]() {                      // the accumulators are in registers: the next item's products may overwrite them
          tc_fence_before();
          mbar_arrive_warp(&bars[BB_ACCFREE]);
        };
        // One buffer for both boxes: two warpgroups take turns (four), or the second box's words wait in registers (two).
        constexpr bool IN_TURN = D == 128 && !EPI2, HOLD = IN_TURN && NWG == 2;
        constexpr int N_BOX = NWG == 4 || HOLD ? 1 : D / 64;
#pragma unroll 1
        for (int bx = qb; bx < qb + N_BOX; ++bx) {
          if (IN_TURN && NWG == 4 && bx == 1 && !by_rows) {      // the first box has been read
            if (!(ok = mbar_wait(&bars[BB_EPX + x], epx & 1, p.ctl, abortp, 38))) break;
            ++epx;
          }
#pragma unroll 1
          for (int c8 = 0; c8 < 4; ++c8) {
            uint32_t w[2][4];
            octets(bx, c8, w);
            if (!HOLD && c8 == 3 && bx + 1 == qb + N_BOX) free_acc();
            put(bx, c8, w);
          }
          [[maybe_unused]] uint32_t held[HOLD ? 4 : 1][2][4];
          if constexpr (HOLD) {
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8) octets(1, c8, held[c8]);
            free_acc();
          }
          if (!(ok = announce(bx))) break;
          if constexpr (HOLD) {
            if (!by_rows) {
              if (r == 0) tma_store_wait_read<0>();
              mbar_arrive_warp(bar_epi);
              if (!(ok = mbar_wait(bar_epi, epi & 1, p.ctl, abortp, 38))) break;
              ++epi;
            }
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8) put(1, c8, held[c8]);
            if (!(ok = announce(1))) break;
          } else if (IN_TURN && bx == 0 && r == 0 && !by_rows) {
            tma_store_wait_read<0>();
            mbar_arrive(&bars[BB_EPX + x]);
          }
        }
        if (!ok) break;
        pending_kve = kb;
      }
    }
    // the shared-memory sources of the last stores must outlive the copies (the writes complete with the grid)
    if (r == 0) tma_store_wait_read<0>();
  }
  if (misc.abort) {
    for (int it = 0; it < 200; ++it) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0) report_abort(p.ctl, abortp);
  if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace fl

static int bwd_launch(const fl_attn_args* a, const void* work, void* stream) {
  using namespace fl;
  if (!a || !a->q_codes || !a->k_codes || !a->v_codes || !a->do_codes || !a->status) return FL_ERR_BAD_ARG;
  if (!a->fac_q || !a->fac_k || !a->fac_v || !a->fac_do || !a->lse_log2 || !a->d_rows || !a->dq_acc || (!a->dq_scale && !a->dq_scale_rows) ||
      !a->dk || !a->dv)
    return FL_ERR_BAD_ARG;
  if (a->d != 128 && a->d != 64) return FL_ERR_UNSUPPORTED;
  if (a->mode != FL_MODE_FP8 && a->mode != FL_MODE_FP4) return FL_ERR_UNSUPPORTED;
  const bool fp4 = a->mode == FL_MODE_FP4;
  if (fp4 && (!a->q4 || !a->k4 || !a->sfq4 || !a->sfk4)) return FL_ERR_BAD_ARG;
  const bool tl = (a->flags & FL_A_TOKEN_LOCAL) != 0, rl = (a->flags & FL_A_DQ_ROWLOCAL) != 0, fold = (a->flags & FL_A_D_PER_FACTOR) != 0;
  if (fold && !tl) return FL_ERR_BAD_ARG;
  if (tl && (!rl || fp4 || a->doc_start)) return FL_ERR_UNSUPPORTED;   // token-local needs the dQ side's own codes
  if (a->d == 64 && (fp4 || rl || tl)) return FL_ERR_UNSUPPORTED;       // d = 64: the default 8-bit route only
  if (a->h <= 0 || a->h_kv <= 0 || a->h % a->h_kv) return FL_ERR_BAD_ARG;
  if ((a->s_q % 128) || (a->s_k % 128) || a->s_q <= 0 || a->s_k <= 0 || a->b <= 0) return FL_ERR_BAD_ARG;
  if (a->doc_start && (a->b != 1 || a->n_docs <= 0 || !a->doc_len || a->s_q != a->s_k)) return FL_ERR_BAD_ARG;
  if (a->seqused_k && a->doc_start) return FL_ERR_UNSUPPORTED;      // documents carry their own lengths
  // batch rows of fewer rows than the whole tiles of the intermediates
  const bool trim = (a->flags & FL_A_ROWS) && !a->doc_start;
  if (trim && (a->s_q != a->s_k || a->out_rows <= 0 || a->out_rows > a->s_q || a->out_rows <= a->s_q - 128)) return FL_ERR_BAD_ARG;
  const int k_len = trim ? a->out_rows : a->s_k;
  CUtensorMap mq, mk, mv, mdo, macc, mq4, mk4, mdk, mdv;
  int rc;
  // (boxes of 64 query rows where a half tile is loaded at a time)
  if ((rc = make_rows_map(&mq, a->q_codes, a->b, a->s_q, a->h, a->d, fp4 ? 64 : 128))) return rc;
  if ((rc = make_rows_map(&mk, a->k_codes, a->b, a->s_k, a->h_kv, a->d, 128))) return rc;
  if ((rc = make_rows_map(&mv, a->v_codes, a->b, a->s_k, a->h_kv, a->d, 128))) return rc;
  if ((rc = make_rows_map(&mdo, a->do_codes, a->b, a->s_q, a->h, a->d, 64))) return rc;
  if (a->d == 128) rc = make_acc_t_map_16(&macc, a->dq_acc, a->b, a->h, a->d, a->s_q);
  else rc = make_acc_map_16(&macc, a->dq_acc, a->b, a->h, a->s_q, a->d, 64);       // (b, h, s, d): boxes of 64 query rows
  if (rc) return rc;
  // the NVFP4 copies (64-byte rows); the 8-bit route passes the E4M3 maps again, which the kernel never touches
  if ((rc = make_rows_map(&mq4, fp4 ? (const void*)a->q4 : (const void*)a->q_codes, a->b, a->s_q, a->h, fp4 ? 64 : a->d, 128)))
    return rc;
  if ((rc = make_rows_map(&mk4, fp4 ? (const void*)a->k4 : (const void*)a->k_codes, a->b, a->s_k, a->h_kv, fp4 ? 64 : a->d,
                          128)))
    return rc;
  // a box that reaches past a row's last column (zero-padded head dims) stores the columns inside only
  const int d_out = (a->flags >> 16) > 0 ? (a->flags >> 16) : a->d;
  if (d_out > a->d || d_out % 8) return FL_ERR_BAD_ARG;
  if ((rc = make_rows_map_16(&mdk, a->dk, a->b, a->slot_src ? a->out_rows : k_len, a->h_kv, d_out, 128))) return rc;
  if ((rc = make_rows_map_16(&mdv, a->dv, a->b, a->slot_src ? a->out_rows : k_len, a->h_kv, d_out, 128))) return rc;
  BwdParams p;
  p.fac_q = a->fac_q; p.fac_k = a->fac_k; p.fac_v = a->fac_v; p.fac_do = a->fac_do; p.lse_log2 = a->lse_log2;
  p.d_rows = a->d_rows; p.dq_scale = a->dq_scale; p.dq_scale_rows = a->dq_scale_rows; p.dk = a->dk; p.dv = a->dv;
  p.dk_mult = a->dk_mult;
  if (a->dk_mult && a->doc_start) return FL_ERR_UNSUPPORTED;            // per-(batch row, head) factors: the batched form
  p.slot_src = a->slot_src; p.slot_rows = a->slot_rows;
  if (a->slot_src && (!a->doc_start || !a->slot_rows || a->out_rows <= 0)) return FL_ERR_BAD_ARG;
  if (a->dq_scale_rows && a->doc_start) return FL_ERR_UNSUPPORTED;      // per-row pre-scale: the batched form
  p.sfq4 = a->sfq4; p.sfk4 = a->sfk4;
  p.doc_start = a->doc_start; p.doc_len = a->doc_len; p.n_docs = a->n_docs;
  p.seqused_k = a->seqused_k;
  p.dq_order = a->dq_order;
  p.b = a->b; p.s_q = a->s_q; p.s_k = a->s_k; p.h = a->h; p.h_kv = a->h_kv; p.d_out = d_out;
  p.q_len = trim ? k_len : a->s_q; p.k_len = k_len;
  p.softmax_scale = a->softmax_scale;
  p.scale_log2 = a->softmax_scale * 1.4426950408889634f;
  const bool sc = a->softcap > 0.f;
  if (sc && (tl || rl)) return FL_ERR_UNSUPPORTED;     // soft cap: the default dS-hat route only
  p.cap_a = sc ? a->softcap * 1.4426950408889634f : 0.f;
  p.cap_b = sc ? 1.0f / p.cap_a : 0.f;
  p.causal = (a->flags & FL_A_CAUSAL) ? 1 : 0;
  p.win_l = window_side(a->window_left_p1);
  p.win_r = p.causal ? 0 : window_side(a->window_right_p1);
  p.out_f16 = (a->flags & FL_A_OUT_F16) ? 1 : 0;
  p.had_dk = (a->flags & FL_A_HAD_DK) ? 1 : 0;
  p.ctl = dev_ctl(a->status, a->wait_cycles > 0 ? a->wait_cycles : kDefaultWaitCycles);
  const int ntile = a->doc_start && !work ? (a->s_k / 128 + a->n_docs) : a->s_k / 128;
  const int nb = a->doc_start ? 1 : a->b;
  p.n_tile = ntile;
  const long long n_items = (long long)ntile * a->h_kv * nb;
  if (n_items > 0x3FFFFFFF) return FL_ERR_TOO_LARGE;
  p.n_items = (int)n_items;
  p.zigzag = ((p.causal && !a->doc_start) || work) ? 1 : 0;
  if (work && !a->doc_start) return FL_ERR_BAD_ARG;
  p.work_head = (const int4*)work;
  p.work = work ? p.work_head + 1 + a->s_k / 128 : nullptr;
  p.div_item = FastDiv(a->doc_start ? 1 : p.causal ? a->h_kv * a->b : ntile);
  p.div_h = FastDiv(a->h_kv);
  p.grp = a->h / a->h_kv;
  const int grid = (int)(n_items < sm_count() ? n_items : sm_count());     // one persistent CTA per SM
  const int smem = a->d == 64 ? BwdSmem<64, false, false>::BYTES : fp4 ? BwdSmem<128, true, false>::BYTES
                   : tl ? BwdSmem<128, false, true>::BYTES : BwdSmem<128, false, false>::BYTES;
  auto launch = [&](auto kern) -> int {
    if (int e = set_smem(kern, smem, "fl_bwd: cudaFuncSetAttribute")) return e;
    launch_after(kern, grid, bwd_threads(rl || tl ? 1 : 0), smem, (cudaStream_t)stream, mq, mk, mv, mdo, macc, mq4, mk4, mdk, mdv, p);
    return FL_OK;
  };
  const bool det = a->dq_order != nullptr;
  if (det && (sc || rl || tl)) return FL_ERR_UNSUPPORTED;     // ordered dQ: the default dS-hat route only
  // the lean kernels serve the plain calls; any of the rarer forms takes the full variant of the same kernel
  const bool full = det || a->dq_scale_rows || a->doc_start || a->dk_mult;
#define FL_BWD_LAUNCH(D_, FP4_, VAR_, SC_) \
  (full ? launch(bwd_kernel_pipelined<D_, FP4_, VAR_, SC_, true>) : launch(bwd_kernel_pipelined<D_, FP4_, VAR_, SC_, false>))
  if (sc) {
    if (a->d == 64) rc = FL_BWD_LAUNCH(64, false, 0, true);
    else rc = fp4 ? FL_BWD_LAUNCH(128, true, 0, true) : FL_BWD_LAUNCH(128, false, 0, true);
  } else if (a->d == 64) {
    rc = FL_BWD_LAUNCH(64, false, 0, false);
  } else if (fp4) {
    rc = rl ? FL_BWD_LAUNCH(128, true, 1, false) : FL_BWD_LAUNCH(128, true, 0, false);
  } else if (tl) {
    rc = fold ? FL_BWD_LAUNCH(128, false, 3, false) : FL_BWD_LAUNCH(128, false, 2, false);
  } else {
    rc = rl ? FL_BWD_LAUNCH(128, false, 1, false) : FL_BWD_LAUNCH(128, false, 0, false);
  }
#undef FL_BWD_LAUNCH
  if (rc) return rc;
  return launch_result("fl_bwd: kernel launch");
}

extern "C" int fl_bwd(const fl_attn_args* a, void* stream) { return bwd_launch(a, nullptr, stream); }

extern "C" int fl_bwd_work(const fl_attn_args* a, const int32_t* work, void* stream) {
  return work ? bwd_launch(a, work, stream) : fl::FL_ERR_BAD_ARG;
}
