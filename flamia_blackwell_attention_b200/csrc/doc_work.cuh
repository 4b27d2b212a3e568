// Work lists of packed documents, built by one block.
#pragma once
#include "sm100.cuh"

namespace fl {

// Work lists of packed documents: the (document, block) pairs that exist, longest first, for the forward (256-row blocks) and the
// backward (128-key tiles). Entry = {document start, document length, block of it, 0}; header {forward entries, backward entries};
// capacity / 128 places per list, then capacity / 128 ints of scratch. Without them the attention kernels search the document
// table once per item, one document after the other (a packed batch of thousands of short documents spent its time there), and
// walk the documents in their order: a long document at the end left most of the chip idle.
// One CTA; thread = 128-row tile of the buffer: documents leave their number at their first tile, a prefix maximum spreads it, a
// counting sort over the cost (key / query tiles visited; 1023 = that or more) places the pairs. ordered: the pairs keep their
// order (the ordered dQ reduction waits for earlier entries).
// The block that runs it is a launch of its own (fl_doc_work) or one of the quantiser's (fl_quant_qkv_work, which says when): nothing
// reads the lists before the forward, and on its own it stood 7 us in the stream. 6000 packed tokens h16/4, fp4 step 191.7 -> 184.5
// us, 8 x 1000 x 12 heads at d = 64 200.3 -> 195.5.
struct DocWork {
  const int32_t* doc_start;
  const int32_t* doc_len;
  int n_docs, capacity, win_l, win_r, ordered;
  int4* work;              // null: no lists
};
static constexpr int DW_BINS = 1024, DOC_WORK_INTS = 2 * DW_BINS + 3 * 32;      // shared memory, ints

// the whole block of THREADS threads; what is read has to be complete (grid_dependency)
template <int THREADS>
__device__ __forceinline__ void doc_work(const DocWork& w, int* sm, int* status) {
  static_assert(THREADS % 32 == 0 && DW_BINS % THREADS == 0);
  int (*s_bin)[DW_BINS] = reinterpret_cast<int (*)[DW_BINS]>(sm);
  int (*s_warp)[32] = reinterpret_cast<int (*)[32]>(sm + 2 * DW_BINS);
  int* s_mark = sm + 2 * DW_BINS + 2 * 32;
  const int32_t *doc_start = w.doc_start, *doc_len = w.doc_len;
  const int n_docs = w.n_docs, capacity = w.capacity, win_l = w.win_l, win_r = w.win_r, ordered = w.ordered;
  int4* const work = w.work;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int T = capacity / 128;
  int* mark = reinterpret_cast<int*>(work + 1 + 2 * T);
  for (int t = tid; t < T; t += THREADS) mark[t] = -1;
  for (int i = tid; i < DW_BINS; i += THREADS) { s_bin[0][i] = 0; s_bin[1][i] = 0; }
  __syncthreads();
  for (int i = tid; i < n_docs; i += THREADS) {
    int st, len;
    doc_entry(doc_start, doc_len, i, capacity, status, st, len);
    if (len > 0) mark[st / 128] = i;
  }
  __syncthreads();
  auto block_exclusive = [&](int v, int (*sums)[32], int which, int& total) {   // exclusive sum over the block (two barriers)
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) sums[which][warp] = inc;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int w = 0; w < THREADS / 32; ++w) { before += w < warp ? sums[which][w] : 0; total += sums[which][w]; }
    __syncthreads();
    return before + inc - v;
  };
  // a tile's document (from the last mark at or before it), its pairs and their costs
  struct Pair { int st, len, rel, cf, cb; };
  auto pair_of = [&](int t, int doc, Pair& q) -> bool {
    if (t >= T || doc < 0) return false;
    int st, len;
    doc_entry(doc_start, doc_len, doc, capacity, nullptr, st, len);
    const int rel = t * 128 - st;
    if (rel < 0 || rel >= len) return false;
    q.st = st; q.len = len; q.rel = rel; q.cf = 0;
    if (!(rel & 255)) {                             // a forward block starts here
      const int nq = min(256, len - rel), k_lo = win_l >= 0 ? max(0, rel - win_l) / 128 * 128 : 0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int rows = min(128, nq - 128 * i);
        const int k_hi = win_r >= 0 ? min(len, rel + 128 * i + rows + win_r) : len;
        if (rows > 0) q.cf += (k_hi - k_lo + 127) / 128;
      }
    }
    int m_hi = (len + 127) / 128, m_lo = 0;
    if (win_r >= 0 && rel > win_r) m_lo = (rel - win_r) / 128;
    if (win_l >= 0) m_hi = min(m_hi, (rel + min(128, len - rel) - 1 + win_l) / 128 + 1);
    q.cb = max(1, m_hi - m_lo);
    return true;
  };
  auto bin_of = [](int cost) { return DW_BINS - 1 - min(cost, DW_BINS - 1); };
  int carry = -1;                                   // the last mark of the tiles before this chunk
  for (int t0 = 0; t0 < T; t0 += THREADS) {
    const int t = t0 + tid;
    int m = (t < T && mark[t] >= 0) ? t : -1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xFFFFFFFFu, m, o);
      if (lane >= o) m = max(m, u);
    }
    if (lane == 31) s_mark[warp] = m;
    __syncthreads();
    int all = carry;
    for (int w = 0; w < THREADS / 32; ++w) { if (w < warp) m = max(m, s_mark[w]); all = max(all, s_mark[w]); }
    m = max(m, carry);
    const int doc = m >= 0 ? mark[m] : -1;
    __syncthreads();                                // (a tile with a mark keeps it; the others take the document's number)
    if (t < T) mark[t] = doc;
    carry = all;
    Pair q;
    if (!ordered && pair_of(t, doc, q)) {
      if (q.cf) atomicAdd(&s_bin[0][bin_of(q.cf)], 1);
      atomicAdd(&s_bin[1][bin_of(q.cb)], 1);
    }
    __syncthreads();
  }
  int n[2] = {0, 0};
  if (!ordered) {
#pragma unroll
    for (int l = 0; l < 2; ++l) {                   // a run of bins per thread
      constexpr int RUN = DW_BINS / THREADS;
      int v = 0;
      for (int i = 0; i < RUN; ++i) v += s_bin[l][tid * RUN + i];
      int at = block_exclusive(v, s_warp, l, n[l]);
      for (int i = 0; i < RUN; ++i) { const int c = s_bin[l][tid * RUN + i]; s_bin[l][tid * RUN + i] = at; at += c; }
    }
    __syncthreads();
  }
  for (int t0 = 0; t0 < T; t0 += THREADS) {
    const int t = t0 + tid;
    Pair q;
    const bool live = pair_of(t, t < T ? mark[t] : -1, q);
    int at[2];
    if (ordered) {
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        int total;
        at[l] = n[l] + block_exclusive(live && (l || q.cf), s_warp, l, total);
        n[l] += total;
      }
    } else if (live) {
      at[0] = q.cf ? atomicAdd(&s_bin[0][bin_of(q.cf)], 1) : 0;
      at[1] = atomicAdd(&s_bin[1][bin_of(q.cb)], 1);
    }
    if (live) {
      if (q.cf) work[1 + at[0]] = make_int4(q.st, q.len, q.rel / 256, 0);
      work[1 + T + at[1]] = make_int4(q.st, q.len, q.rel / 128, 0);
    }
  }
  if (tid == 0) work[0] = make_int4(n[0], n[1], 0, 0);
}

}  // namespace fl
