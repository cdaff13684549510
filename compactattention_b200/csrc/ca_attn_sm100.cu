// Block-table-indexed dense causal attention for sm_100a: tcgen05 MMA with TMEM accumulators,
// TMA loads whose page coordinate comes from the per-KV-head block table.
//
// Work unit = one KV-head row (b, hkv) and a pair of 128-row query tiles ("A" and "B").  A query
// tile stacks the G query heads of the KV head along M: tile row i is (token i / G, head i % G),
// so one K/V stage feeds G heads.  K/V are consumed in 128-token steps = two 64-token sub-blocks,
// each fetched by its own TMA box at (page, token offset) resolved from the block table and the
// optional page table.  Selected past blocks are fully visible; the chunk's own blocks follow in
// order and are causally masked (bottom-right aligned), which is what
// compact_attn/kernels/varlen/indexed_dense_prefill_direct_triton.py:155-241 computes.
//
// Scheduling (ca_attn_plan.cuh): a persistent grid of one CTA per SM.  All units are laid end to end, each as
// long as its KV steps and what it costs beside them, and the kernel decides from the rows' counts whether this
// line is cut into equal spans ("stream-K": the SMs stay balanced whatever the per-row block counts are and
// however few rows a tensor-parallel rank owns) or units stay whole: one per CTA where there are enough CTAs,
// else those that start inside an equal share of the line.  A unit that falls entirely inside one span is written
// straight to the output; a unit cut by a span boundary leaves per-segment partials (unnormalised O, running
// max, running sum) in the workspace and a small combine kernel merges them; it is launched where units may be
// cut.  Without a workspace units stay whole.
//
// Warp roles (384 threads): warps 0-3 softmax of tile A, warps 4-7 softmax of tile B (thread =
// TMEM lane = tile row), warp 8 issues every tcgen05.mma, warp 9 issues every TMA, warps
// 10-11 idle.  The third warpgroup gives its registers to the softmax warpgroups (setmaxnreg),
// which hold a whole 128-column S row per thread.
// TMEM (512 columns): S | P_A | P_B | O_A | O_B, of 128, 64, 64, 128 and 128 columns.  S is one buffer that the tiles
// take in turn: a softmax warpgroup moves its S into registers at once and gives the buffer back; P (16-bit) has a place
// of its own and feeds the P.V MMA straight from TMEM.  So S(j+1) does not wait for P.V(j), as it did when each tile had
// its own S and P lay over it (S -> softmax -> P -> P.V -> next S was one chain of about 3300 cycles a step).
// MMA order S_A0 S_B0 { S_A(j+1) PV_A(j) S_B(j+1) PV_B(j) }.  With the chain / without, us, single launches and at the
// power cap: 1024 x 106K keys, 32/8 heads 458 / 435, 528 / 511; 8192 x 8192, f16 512 / 490, 562 / 549; 8192 x 40K,
// 28/4 heads 3305 / 3191, 3823 / 3684.  Every wait is bounded; on expiry the CTA raises CA_STATUS_TIMEOUT, drains
// what it issued, frees TMEM and returns.
#include "ca_attn_plan.cuh"
#include "ca_attn_shared.cuh"

#include <mutex>

namespace ca {
namespace attn {

constexpr int kThreads = 384;  // three warpgroups: softmax A, softmax B, {MMA, TMA, 2 idle warps}
constexpr int kTileM = 128;
constexpr int kTileN = 128;
constexpr int kHeadDim = 128;
constexpr int kHalfBytes = 128 * 128;  // one [128 rows][64 x 16-bit] swizzled half tile
constexpr int kTileBytes = 2 * kHalfBytes;
constexpr int kBoxBytes = kSub * 128;  // one [64 tokens][64 x 16-bit] box
constexpr int kStages = 4;
constexpr int kTmemCols = 512;
constexpr int kMaxRows = 1024;  // (batch x kv heads) rows per launch
constexpr int kMaxSegs = 64;    // segments planned per batch
constexpr float kRescaleThreshold = 8.0f;  // log2 units; lazy accumulator rescale
// Measured with the earlier form (one issuing lane in a branch, P over S; 300 launches, 128K context, 20 % density): handing P
// to the MMA warp in two halves 434 us, in one piece 450 us; packed fp32 pairs for the scale and the row sum 421 us; a polynomial
// exp2 on the FMA pipe for 2 / 4 / 6 of every 16 pairs 486 / 499 / 518 us, without it 485.  The issuing lane was the pace then, so the
// last says nothing of this form, where MUFU is about as busy as the tensor pipe; it has not been measured here.
#ifndef CA_ATTN_PROFILE
#define CA_ATTN_PROFILE 0
#endif
#ifndef CA_ATTN_MERGE_DEPENDENT
// The merge kernel is enqueued as a programmatic dependent of the attention kernel (it waits with
// griddepcontrol.wait before reading anything): its CTAs are resident when the last attention CTA
// leaves.  Measured: 90.8 -> 88.2 us (one KV head), 134.4 -> 131.1 us (two), 32.9 -> 30.8 us (a small
// shape whose units stay whole); 0 restores a plain launch.
#define CA_ATTN_MERGE_DEPENDENT 1
#endif
constexpr int kPParts = 2;  // P is handed to the MMA warp in this many pieces (of 4 MMAs each) so P.V overlaps the softmax

// Optional cycle accounting (development builds only, -DCA_ATTN_PROFILE=1): one thread of each role
// adds the clock cycles between consecutive marks to per-CTA counters.
#if CA_ATTN_PROFILE
__device__ long long g_prof[160][32];
#define CA_PROF_DECL unsigned prof_t = clock(); unsigned prof_acc[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
#define CA_PROF(i) { const unsigned prof_n = clock(); prof_acc[i] += prof_n - prof_t; prof_t = prof_n; }
#define CA_PROF_FLUSH(base) { for (int prof_i = 0; prof_i < 10; ++prof_i) g_prof[blockIdx.x][(base) + prof_i] = prof_acc[prof_i]; }
#else
#define CA_PROF_DECL
#define CA_PROF(i) {}
#define CA_PROF_FLUSH(base) {}
#endif

// Partial results of one segment of a split unit.
constexpr int kPartialOFloats = 2 * kTileM * kHeadDim;  // [tile][col/4][row][4]
constexpr int kPartialMLFloats = 2 * kTileM * 2;        // [tile][row][m, l]

struct SegDesc {  // one per workspace slot
  int unit;       // row * n_pairs + pair, or -1 when the slot is unused
  int j0, j1;     // KV-step range of the segment inside the unit
  int n_iter;     // KV steps of the whole unit
};

struct Segment {
  int row, pair;
  int j0, j1;
  int n_sub, n_past_sub;
  int slot;  // workspace slot of a partial segment (the unit's first: odd, others: even), -1: whole unit, written to the output
  int pad;   // to 32 bytes: with 28, 8192 x 8192 (32/8 heads) took 566 us instead of 556
};

struct KernelArgs : Units {  // q_off: 0 unless a dense launch has an unaligned past
  int G, Hkv, B;
  int past_blocks;  // Pb
  int block_size;
  int past_tokens;  // tokens before the chunk region (a multiple of block_size)
  int page_size, pages_per_seq, num_pages;
  const int32_t* block_idx;
  int block_idx_stride;
  const int32_t* counts;
  const int32_t* page_table;
  void* out;
  long long o_stride_b, o_stride_t, o_stride_h;
  float* lse;
  float scale_log2;
  int32_t* status;
  uint32_t idesc_qk, idesc_pv;
  unsigned long long wait_limit_ns;
  unsigned int wait_limit_us;
  // K/V tensor-map dimensions 1..3 are ordered by ascending stride at encode time; these give the
  // coordinate slot (0..2) of the token, page and head coordinates.
  int slot_tok, slot_page, slot_head;
  int kv_head_div;     // block-table rows per KV head (1 unless per-query-head / sub-group tables)
  int split;           // 1: spans may cut units (needs the workspace)
  SegDesc* descs;      // [2 * gridDim.x]
  float* part_ml;      // [2 * gridDim.x][kPartialMLFloats]
  float* part_o;       // [2 * gridDim.x][kPartialOFloats]
};

struct TileBars {
  uint64_t s_full, p_part[2], o_free;  // the last piece of P in use completes it
};

struct Shared {
  uint64_t q_full[2];
  uint64_t q_free;
  uint64_t ring_full[kStages];
  uint64_t ring_empty[kStages];
  uint64_t s_free;      // the warpgroup whose turn it was has S in registers
  TileBars tile[2];
  uint64_t pv_done[2];  // P has been read, O is up to date
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
  int n_segs;
  int more;            // another batch of segments follows
  int cut;             // spans may end inside a unit
  int cur_row, cur_pair;        // the unit the next segment comes from ...
  long long cur_acc;            // ... and where that starts on the line of all units
  int row_count[kMaxRows];
  long long row_prefix[kMaxRows + 1];
  Segment segs[kMaxSegs];
};

constexpr int kSmemBytes = 2 * kTileBytes + kStages * kTileBytes + 1024 /*align*/ + static_cast<int>(sizeof(Shared));

template <typename T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Number of visible columns (0..64) of 64-token sub-block u for chunk token t.
__device__ __forceinline__ int visible_cols(int u, int n_sub, int n_past_sub, int t) {
  // t counts from the start of the chunk region (query token index + q_off)
  if (u >= n_sub) return 0;
  if (u < n_past_sub) return kSub;
  int lim = t - (u - n_past_sub) * kSub + 1;
  return lim < 0 ? 0 : (lim > kSub ? kSub : lim);
}

// Finds the unit that holds position x of the line (one warp, all lanes): its row and pair, where it starts.
__device__ void locate_unit(const KernelArgs& a, const Shared* sh, long long x, int R, int lane, int* row, int* pair, long long* acc) {
  int lo = 0, hi = R;  // largest row with row_prefix[row] <= x
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (sh->row_prefix[mid] <= x) lo = mid; else hi = mid;
  }
  long long base = sh->row_prefix[lo];
  const int count = sh->row_count[lo];
  *row = lo, *pair = 0, *acc = base;
  for (int p0 = 0; p0 < a.n_pairs; p0 += 32) {
    const int p = p0 + lane;
    const int ni = p < a.n_pairs ? unit_cost(a, count, p) : 0;
    int inc = ni;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += n;
    }
    const uint32_t hit = __ballot_sync(0xffffffffu, p < a.n_pairs && base + inc > x);
    if (hit) {
      const int l = __ffs(hit) - 1;
      *pair = p0 + l;
      *acc = base + __shfl_sync(0xffffffffu, inc - ni, l);
      return;
    }
    base += __shfl_sync(0xffffffffu, inc, 31);
  }
}

// Plans up to kMaxSegs further segments of this CTA's span (thread 0 only).
__device__ void plan_segments(const KernelArgs& a, Shared* sh, long long span_begin, long long span_end, int R) {
  int n = 0;
  int row = sh->cur_row, pair = sh->cur_pair;
  long long acc = sh->cur_acc;
  const bool cut = sh->cut != 0;
#pragma unroll 1
  while (acc < span_end && n < kMaxSegs && row < R) {
    const int count = sh->row_count[row];
    const int ni = unit_iters(a, count, pair);
    int j0 = 0, j1 = ni;
    if (cut) {  // a boundary within the unit's first kUnitSteps cuts nothing off
      const long long before = span_begin - acc - kUnitSteps;
      if (before > 0) j0 = static_cast<int>(before);
      const long long left = span_end - acc - kUnitSteps;
      if (left < ni) j1 = static_cast<int>(left);
    }
    if (j1 > j0) {
      Segment& s = sh->segs[n++];
      s.row = row, s.pair = pair, s.j0 = j0, s.j1 = j1;
      s.n_past_sub = count * a.spb;
      s.n_sub = s.n_past_sub + chunk_subs(a, pair);
      s.slot = -1;
      if (j0 > 0 || j1 < ni) {
        const int slot = static_cast<int>(2 * blockIdx.x + (j0 > 0 ? 0 : 1));
        s.slot = slot;
        SegDesc d;
        d.unit = row * a.n_pairs + pair, d.j0 = j0, d.j1 = j1, d.n_iter = ni;
        a.descs[slot] = d;
      }
    }
    acc += ni + kUnitSteps;
    if (++pair == a.n_pairs) pair = 0, ++row;
  }
  sh->n_segs = n;
  sh->cur_row = row, sh->cur_pair = pair, sh->cur_acc = acc;
  sh->more = (acc < span_end && row < R) ? 1 : 0;
}

// P = exp2(S*sc + neg_m) for one 128-column row held in registers: packs to 16 bit, calls p_free, which blocks until P's own TMEM
// columns may be overwritten (before the first store), stores the four 32-column chunks there, signals the MMA warp after each of
// the kPParts pieces.  The scale and the row sum use packed fp32 pairs.  Returns the row sum of P.
template <typename T, typename Free>
__device__ __forceinline__ float exp_pack_store(const uint32_t (&sv)[128], float sc, float neg_m, uint32_t tP,
                                                uint32_t p_part_bar, Free p_free) {
  float2 l2 = make_float2(0.f, 0.f);
  const float2 sc2 = make_float2(sc, sc);
  const float2 nm2 = make_float2(neg_m, neg_m);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t pk[16];
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[c * 32 + i]), __uint_as_float(sv[c * 32 + i + 1])), sc2, nm2);
      float2 pr;
      pr.x = ptx::ex2(x.x);
      pr.y = ptx::ex2(x.y);
      l2 = __fadd2_rn(l2, pr);
      pk[i >> 1] = pack2<T>(pr.x, pr.y);
    }
    if (c == 0) p_free();
    ptx::tmem_st16(tP + c * 16, pk);
    if ((c + 1) % (4 / kPParts) == 0) {
      // a piece of P is in TMEM: let the MMA warp run P.V on it (the last piece completes P)
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      ptx::mbar_arrive(p_part_bar + static_cast<uint32_t>(((c + 1) / (4 / kPParts) - 1) * sizeof(uint64_t)));
    }
  }
  return l2.x + l2.y;
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
    attn_compact_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                        const __grid_constant__ CUtensorMap v_map, const KernelArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_aligned = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const uint32_t q_smem = smem_base;                      // Q_A, Q_B
  const uint32_t ring_smem = smem_base + 2 * kTileBytes;  // kStages slots
  Shared* sh = reinterpret_cast<Shared*>(smem_aligned + 2 * kTileBytes + kStages * kTileBytes);

  const uint32_t sh_addr = ring_smem + kStages * kTileBytes;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int R = a.B * a.Hkv;
  volatile int* abort_flag = &sh->abort_flag;
  const uint64_t limit = a.wait_limit_ns;
  bool bad_index = false;

#if CA_ATTN_PROFILE
  const long long prof_kernel_t0 = clock64();
#endif
  // ---- on-chip set-up first: it needs nothing from global memory, so under a programmatic
  // dependent launch it overlaps the tail of the previous kernel (the table builder) ----
  ptx::grid_launch_dependents();
  if (tid == 0) {
    sh->row_prefix[0] = 0;
    sh->abort_flag = 0;
    ptx::mbar_init(ptx::smem_u32(&sh->q_full[0]), 1);
    ptx::mbar_init(ptx::smem_u32(&sh->q_full[1]), 1);
    ptx::mbar_init(ptx::smem_u32(&sh->q_free), 1);
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(ptx::smem_u32(&sh->ring_full[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&sh->ring_empty[s]), 1);
    }
    ptx::mbar_init(ptx::smem_u32(&sh->tile[0].s_full), 1);
    ptx::mbar_init(ptx::smem_u32(&sh->tile[1].s_full), 1);
    ptx::mbar_init(ptx::smem_u32(&sh->s_free), 128);
    ptx::mbar_init(ptx::smem_u32(&sh->pv_done[0]), 1);
    ptx::mbar_init(ptx::smem_u32(&sh->pv_done[1]), 1);
    for (int q = 0; q < 2; ++q) {
      ptx::mbar_init(ptx::smem_u32(&sh->tile[0].p_part[q]), 128);
      ptx::mbar_init(ptx::smem_u32(&sh->tile[1].p_part[q]), 128);
    }
    ptx::mbar_init(ptx::smem_u32(&sh->tile[0].o_free), 128);
    ptx::mbar_init(ptx::smem_u32(&sh->tile[1].o_free), 128);
    ptx::mbar_init(ptx::smem_u32(&sh->drain), 1);
    ptx::mbar_fence_init();
    ptx::fence_proxy_async_smem();
  }
  if (warp == 8) {
    ptx::tmem_alloc(ptx::smem_u32(&sh->tmem_base), kTmemCols);
    ptx::tmem_relinquish();
  }
  if (warp == 9 && lane == 0) {
    ptx::tma_prefetch_desc(&q_map);
    ptx::tma_prefetch_desc(&k_map);
    ptx::tma_prefetch_desc(&v_map);
  }
  ptx::grid_dependency_wait();  // nothing in global memory is touched before this

  // ---- per-row totals (KV steps and what units cost beside them) and their prefix (every CTA; a warp per row) ----
  for (int r = warp; r < R; r += kThreads / 32) {
    int count = a.past_blocks;
    if (a.block_idx != nullptr) {
      count = a.counts[r];
      const int cap = a.block_idx_stride < a.past_blocks ? a.block_idx_stride : a.past_blocks;
      if (count < 0 || count > cap) {
        bad_index = true;
        count = count < 0 ? 0 : cap;
      }
    }
    const unsigned part = lane_cost(a, count, lane);  // their sum may need more than 32 bits
    const unsigned lo = __reduce_add_sync(0xffffffffu, part & 0xffffu), hi = __reduce_add_sync(0xffffffffu, part >> 16);
    if (lane == 0) {
      sh->row_count[r] = count;
      sh->row_prefix[r + 1] = (static_cast<long long>(hi) << 16) + lo;  // turned into a prefix below
    }
  }
  if (tid == 0 && a.descs) {
    SegDesc none;
    none.unit = -1, none.j0 = 0, none.j1 = 0, none.n_iter = 0;
    a.descs[2 * blockIdx.x] = none;
    a.descs[2 * blockIdx.x + 1] = none;
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = sh->tmem_base;
  long long span_begin = 0, span_end = 0;
  if (warp == 0) {
    if (lane == 0) {
      for (int r = 0; r < R; ++r) sh->row_prefix[r + 1] += sh->row_prefix[r];
    }
    // shortest and longest unit: the first pair of the shortest row, the last pair of the longest
    int c_lo = 0x7fffffff, c_hi = 0;
    for (int r = lane; r < R; r += 32) c_lo = min(c_lo, sh->row_count[r]), c_hi = max(c_hi, sh->row_count[r]);
    const int l_min = unit_cost(a, __reduce_min_sync(0xffffffffu, c_lo), 0);
    const int l_max = unit_cost(a, __reduce_max_sync(0xffffffffu, c_hi), a.n_pairs - 1);
    __syncwarp();
    const long long total = sh->row_prefix[R];
    const long long c = blockIdx.x;
    const long long n_units = static_cast<long long>(R) * a.n_pairs;
    const long long g = gridDim.x;
    int nc = 1;
    const bool cut = a.split && units_are_cut(total, n_units, l_min, l_max, gridDim.x, &nc);
    int row = 0, pair = 0;
    long long acc = 0;
    if (cut) {
      if (c < nc) {
        span_begin = total * c / nc;
        span_end = total * (c + 1) / nc;
      }
    } else if (n_units <= g) {
      // a unit of its own; its steps need no place among the others'
      row = static_cast<int>(c / a.n_pairs), pair = static_cast<int>(c % a.n_pairs);
      if (c < n_units) span_end = 1;
    } else {
      // the units that start inside an equal share of the steps
      span_begin = total * c / g;
      span_end = total * (c + 1) / g;
    }
    if (span_end > span_begin && (cut || n_units > g)) {
      locate_unit(a, sh, span_begin, R, lane, &row, &pair, &acc);
      if (!cut && acc < span_begin) {
        acc += unit_cost(a, sh->row_count[row], pair);
        if (++pair == a.n_pairs) pair = 0, ++row;
        span_begin = acc;
      }
    }
    if (lane == 0) {
      sh->cut = cut ? 1 : 0;
      sh->cur_row = row, sh->cur_pair = pair, sh->cur_acc = acc;
      sh->more = span_end > span_begin && row < R ? 1 : 0;
      sh->n_segs = 0;
    }
  }
  __syncthreads();

#if CA_ATTN_PROFILE
  if (tid == 0) g_prof[blockIdx.x][30] = clock64() - prof_kernel_t0;  // prologue
#endif
  // role state that lives across segments
  int ring_n = 0;        // ring entries issued (loader) / consumed (MMA)
  uint32_t it = 0;       // KV steps processed so far: parity of s_full / p_part / pv_done, and, two to a step, of s_free
  uint32_t seg_seq = 0;  // segments processed so far: parity of q_full / q_free / o_free
  uint32_t q_issued = 0; // Q loads issued (loader)
  bool ok = true;

  // The producer warpgroup hands registers to the softmax warpgroups.  The pool is what the CTA got
  // at launch, 384 threads x 168 registers = 64512, so 2 x 128 x 208 + 128 x 88 = 64512 fits it
  // exactly; asking for more would block the second setmaxnreg.inc forever.  Each side keeps its
  // own copy of the batch loop so the raised budget applies to the softmax code; both sides
  // execute the same sequence of CTA-wide barriers.
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    while (true) {
      __syncthreads();
      const int n_segs = sh->n_segs;
      if (n_segs == 0) break;
      if (warp == 9) {
        // =============================== TMA producer ===============================
        for (int si = 0; si < n_segs && ok; ++si) {
          const Segment sg = sh->segs[si];
          const int b = sg.row / a.Hkv, hkv = sg.row % a.Hkv;
          int vp0 = 0, vo0 = 0, vp1 = 0, vo1 = 0;
          bool v_two = true;
          // one ring entry: the two (or one) 64-token sub-blocks of a K or V tile
          auto load_tile = [&](const CUtensorMap& map, int p0, int o0, int p1, int o1, bool two) {
            const int slot = ring_n % kStages;
            const uint32_t phase = (ring_n / kStages) & 1;
            if (ok) ok = ptx::mbar_wait_bounded(ptx::smem_u32(&sh->ring_empty[slot]), phase ^ 1u, abort_flag, limit);
            if (!ok) return;
            const uint32_t bar = ptx::smem_u32(&sh->ring_full[slot]);
            const uint32_t dst = ring_smem + slot * kTileBytes;
            ptx::mbar_expect_tx(bar, two ? 4u * kBoxBytes : 2u * kBoxBytes);
            int c0[3], c1[3];
            c0[a.slot_tok] = o0, c0[a.slot_page] = p0, c0[a.slot_head] = hkv / a.kv_head_div;
            c1[a.slot_tok] = o1, c1[a.slot_page] = p1, c1[a.slot_head] = hkv / a.kv_head_div;
            for (int h = 0; h < 2; ++h) {
              ptx::tma_load_4d(dst + h * kHalfBytes, &map, bar, h * 64, c0[0], c0[1], c0[2]);
              if (two) ptx::tma_load_4d(dst + h * kHalfBytes + kBoxBytes, &map, bar, h * 64, c1[0], c1[1], c1[2]);
            }
            ++ring_n;
          };
          for (int base = 2 * sg.j0; base < 2 * sg.j1 && ok; base += 32) {
            // every lane resolves one sub-block of this batch of 32
            const int u = base + lane;
            int page = 0, off = 0;
            if (u < sg.n_sub) {
              int tok;
              if (u < sg.n_past_sub) {
                const int bi = u / a.spb;
                int blk = a.block_idx ? a.block_idx[static_cast<long long>(sg.row) * a.block_idx_stride + bi] : bi;
                if (blk < 0 || blk >= a.past_blocks) {
                  bad_index = true;
                  blk = blk < 0 ? 0 : a.past_blocks - 1;
                }
                tok = blk * a.block_size + (u - bi * a.spb) * kSub;
              } else {
                tok = a.past_tokens + (u - sg.n_past_sub) * kSub;
              }
              const int lp = tok / a.page_size;
              off = tok - lp * a.page_size;
              if (a.page_table) {
                page = (lp < a.pages_per_seq) ? a.page_table[static_cast<long long>(b) * a.pages_per_seq + lp] : -1;
                if (page < 0 || page >= a.num_pages) {
                  bad_index = true;
                  page = 0;
                }
              } else {
                page = b * a.pages_per_seq + lp;  // beyond the tensor: TMA zero-fills
              }
            }
            for (int i = 0; i < 16 && ok; ++i) {
              const int j = (base >> 1) + i;
              if (j >= sg.j1) break;
              const int p0 = __shfl_sync(0xffffffffu, page, 2 * i);
              const int o0 = __shfl_sync(0xffffffffu, off, 2 * i);
              const int p1 = __shfl_sync(0xffffffffu, page, 2 * i + 1);
              const int o1 = __shfl_sync(0xffffffffu, off, 2 * i + 1);
              const bool two = (2 * j + 1) < sg.n_sub;
              if (lane == 0) {
                // in the order in which the issuer takes them: K of this step, V of the one before
                load_tile(k_map, p0, o0, p1, o1, two);
                if (j == sg.j0) {
                  // Q follows the segment's first K tile: its memory is free once the last Q.K^T of the previous
                  // segment has completed, while that segment's last softmax, P.V and epilogue still run
                  if (ok && seg_seq > 0) ok = ptx::mbar_wait_bounded(ptx::smem_u32(&sh->q_free), (seg_seq - 1) & 1, abort_flag, limit);
                  if (ok) {
                    const uint32_t q_bytes = 2u * 128u * static_cast<uint32_t>(a.G * a.tpt);
                    for (int tile = 0; tile < 2; ++tile) {
                      const uint32_t q_bar = ptx::smem_u32(&sh->q_full[tile]);
                      ptx::mbar_expect_tx(q_bar, q_bytes);
                      for (int h = 0; h < 2; ++h) {
                        ptx::tma_load_5d(q_smem + tile * kTileBytes + h * kHalfBytes, &q_map, q_bar, h * 64, 0, hkv,
                                         (2 * sg.pair + tile) * a.tpt, b);
                      }
                    }
                    ++q_issued;
                  }
                } else {
                  load_tile(v_map, vp0, vo0, vp1, vo1, true);  // only a unit's last step can have one sub-block
                }
                vp0 = p0, vo0 = o0, vp1 = p1, vo1 = o1, v_two = two;
              }
              ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            }
          }
          if (ok && lane == 0) load_tile(v_map, vp0, vo0, vp1, vo1, v_two);
          ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
          ++seg_seq;
        }
      } else if (warp == 8) {
        // =============================== MMA issuer ===============================
        {
          // The warp stays converged and one elected lane issues.  From a branch that one lane takes, the MMAs and commits of a
          // KV step took that lane 2850 cycles, 78 % of the step (1024 x 106K keys, 32/8 heads); from the converged warp 1790.
          // us before / after, single launches and at the power cap: that shape 472 / 458, 535 / 528; 8192 x 8192, f16 538 / 512,
          // 580 / 562; 8192 x 40K, 28/4 heads 3379 / 3305, 3914 / 3823.
          const uint32_t lead = ptx::elect_one();
          const uint32_t tS = tmem;
          const uint32_t tP[2] = {tmem + 128u, tmem + 192u};
          const uint32_t tO[2] = {tmem + 256u, tmem + 384u};
          // Descriptors: one base per operand buffer; within a product's block of instructions a constant is added per MMA (the
          // start address sits in the low 14 bits in 16-byte units and never carries).
          const uint64_t q_desc[2] = {ptx::make_smem_desc_sw128(q_smem, 0, 1024),
                                      ptx::make_smem_desc_sw128(q_smem + kTileBytes, 0, 1024)};
          const uint64_t k_desc0 = ptx::make_smem_desc_sw128(ring_smem, 0, 1024);
          const uint64_t v_desc0 = ptx::make_smem_desc_sw128(ring_smem, kHalfBytes, 1024);
          const uint32_t idesc_qk = a.idesc_qk, idesc_pv = a.idesc_pv;
          auto issue_s = [&](int tile, int slot) {
            ptx::mma_ss_128x128x128(lead, tS, q_desc[tile], k_desc0 + static_cast<uint64_t>(slot * (kTileBytes >> 4)), idesc_qk);
          };
          // a half (4 k-steps) of O += P.V
          auto issue_pv = [&](int tile, int slot, int half, bool first) {
            ptx::mma_ts_128x128x64(lead, tO[tile], tP[tile] + half * 32, v_desc0 + static_cast<uint64_t>(slot * (kTileBytes >> 4) + half * (8192 >> 4)),
                                   idesc_pv, (first && half == 0) ? 0u : 1u);
          };
          auto wait = [&](uint64_t* bar, uint32_t parity) {
            if (ok) {
              ok = ptx::mbar_wait_bounded(ptx::smem_u32(bar), parity, abort_flag, limit);
              ok = __all_sync(0xffffffffu, ok);
            }
            return ok;
          };
          CA_PROF_DECL
          // S is one buffer for both tiles: the next one may go there once the other tile's warpgroup has taken its own
          auto wait_s_free = [&](uint32_t n) { return n == 0 || wait(&sh->s_free, (n - 1) & 1); };
          for (int si = 0; si < n_segs && ok; ++si) {
            const Segment sg = sh->segs[si];
            const uint32_t qpar = seg_seq & 1;
            {
              const int slot = ring_n % kStages;
              const uint32_t phase = (ring_n / kStages) & 1;
              if (!(wait(&sh->q_full[0], qpar) && wait(&sh->q_full[1], qpar) && wait(&sh->ring_full[slot], phase))) break;
              if (!wait_s_free(2 * it)) break;
              ptx::tc_fence_after();
              issue_s(0, slot);
              ptx::tc_commit_if(lead, ptx::smem_u32(&sh->tile[0].s_full));
              if (!wait_s_free(2 * it + 1)) break;
              ptx::tc_fence_after();
              issue_s(1, slot);
              ptx::tc_commit_if(lead, ptx::smem_u32(&sh->tile[1].s_full));
              ptx::tc_commit_if(lead, ptx::smem_u32(&sh->ring_empty[slot]));
              if (sg.j0 + 1 == sg.j1) ptx::tc_commit_if(lead, ptx::smem_u32(&sh->q_free));
              ++ring_n;
            }
            for (int j = sg.j0; j < sg.j1 && ok; ++j, ++it) {
              const bool more = (j + 1) < sg.j1;
              const int k_slot = ring_n % kStages;
              const uint32_t k_phase = (ring_n / kStages) & 1;
              if (more) ++ring_n;
              const int v_slot = ring_n % kStages;
              const uint32_t v_phase = (ring_n / kStages) & 1;
              ++ring_n;
              const bool two = (2 * j + 1) < sg.n_sub;
              const bool first = j == sg.j0;
#pragma unroll
              for (int tile = 0; tile < 2; ++tile) {
                CA_PROF(0)
                if (more) {
                  if (tile == 0 && !wait(&sh->ring_full[k_slot], k_phase)) break;
                  CA_PROF(4)
                  if (!wait_s_free(2 * it + 2 + tile)) break;
                  CA_PROF(6)
                  ptx::tc_fence_after();
                  issue_s(tile, k_slot);
                  ptx::tc_commit_if(lead, ptx::smem_u32(&sh->tile[tile].s_full));
                  if (tile == 1) {
                    ptx::tc_commit_if(lead, ptx::smem_u32(&sh->ring_empty[k_slot]));
                    if (j + 2 == sg.j1) ptx::tc_commit_if(lead, ptx::smem_u32(&sh->q_free));
                  }
                }
                CA_PROF(0)
                if (tile == 0 && !wait(&sh->ring_full[v_slot], v_phase)) break;
                CA_PROF(1)
                // P arrives in pieces so P.V starts while the softmax still works
#pragma unroll
                for (int q = 0; q < kPParts && ok; ++q) {
                  if (q > 0) CA_PROF(0)
                  if (!wait(&sh->tile[tile].p_part[q], it & 1)) break;
                  if (tile == 0) { CA_PROF(2) } else { CA_PROF(5) }
                  // the accumulator is free once the previous segment's epilogue has read it
                  if (q == 0 && first && seg_seq > 0 && !wait(&sh->tile[tile].o_free, (seg_seq - 1) & 1)) break;
                  ptx::tc_fence_after();
                  if (q == 0 || two) issue_pv(tile, v_slot, q, first);
                }
                if (!ok) break;
                ptx::tc_commit_if(lead, ptx::smem_u32(&sh->pv_done[tile]));
              }
              if (!ok) break;
              ptx::tc_commit_if(lead, ptx::smem_u32(&sh->ring_empty[v_slot]));
            }
            ++seg_seq;
            CA_PROF(7)
          }
          if (lane == 0) CA_PROF_FLUSH(0)
        }
      }
      ok = __syncthreads_and(ok ? 1 : 0) != 0;  // all roles finished this batch (or aborted)
      if (!ok) break;
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    while (true) {
      if (tid == 0 && sh->more) plan_segments(a, sh, span_begin, span_end, R);
      else if (tid == 0) sh->n_segs = 0;
      __syncthreads();
      const int n_segs = sh->n_segs;
      if (n_segs == 0) break;
      {
        // =============================== softmax + epilogue ===============================
        const int tile = warp >> 2;  // 0: A, 1: B
        const int r = tid & 127;     // tile row = TMEM lane
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t tS = tmem + lane_base;
        const uint32_t tP = tmem + lane_base + 128u + tile * 64u;
        const uint32_t tO = tmem + lane_base + 256u + tile * 128u;
        const uint32_t tile_bars = sh_addr + offsetof(Shared, tile) + tile * sizeof(TileBars);
        const uint32_t abort_addr = sh_addr + offsetof(Shared, abort_flag);
        const float sc = a.scale_log2;
        uint32_t v[32];
        CA_PROF_DECL
        for (int si = 0; si < n_segs && ok; ++si) {
          const Segment sg = sh->segs[si];
          const int b = sg.row / a.Hkv, hkv = sg.row % a.Hkv;
          const int t = (2 * sg.pair + tile) * a.tpt + r / a.G;  // chunk token of this row
          const int g = r % a.G;
          float m_run = -INFINITY;
          float l_run = 0.f;
          for (int j = sg.j0; j < sg.j1; ++j, ++it) {
            CA_PROF(0)
            ok = ptx::mbar_wait_lean(tile_bars + offsetof(TileBars, s_full), it & 1, abort_addr, a.wait_limit_us);
            ok = __all_sync(0xffffffffu, ok);  // keep the warp converged for the collective TMEM ops
            if (!ok) break;
            CA_PROF(1)
            ptx::tc_fence_after();
            bool masked = (2 * j + 1) >= sg.n_past_sub;  // a chunk or tail sub-block is in this step
            int lim0 = kSub, lim1 = kSub;
            if (masked) {
              lim0 = visible_cols(2 * j, sg.n_sub, sg.n_past_sub, t + a.q_off);
              lim1 = visible_cols(2 * j + 1, sg.n_sub, sg.n_past_sub, t + a.q_off);
              // in a long chunk most of these steps lie wholly before the warp's rows (8192 x 8192: 667 -> 604 us)
              masked = __any_sync(0xffffffffu, lim0 < kSub || lim1 < kSub);
            }
            // the whole S row (128 fp32) comes into registers with one wait
            uint32_t sv[128];
            ptx::tmem_ld32_row<0>(tS + 0, sv);
            ptx::tmem_ld32_row<32>(tS + 32, sv);
            ptx::tmem_ld32_row<64>(tS + 64, sv);
            ptx::tmem_ld32_row<96>(tS + 96, sv);
            ptx::tc_wait_ld();
            ptx::tc_fence_before();
            ptx::mbar_arrive(sh_addr + offsetof(Shared, s_free));
            CA_PROF(2)
            if (masked) {
  #pragma unroll
              for (int i = 0; i < 128; ++i) {
                const int lim = i < 64 ? lim0 : lim1;
                if ((i & 63) >= lim) sv[i] = 0xff800000u;  // -inf
              }
            }
            float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
  #pragma unroll
            for (int i = 0; i < 128; i += 4) {
              mx0 = fmaxf(mx0, __uint_as_float(sv[i]));
              mx1 = fmaxf(mx1, __uint_as_float(sv[i + 1]));
              mx2 = fmaxf(mx2, __uint_as_float(sv[i + 2]));
              mx3 = fmaxf(mx3, __uint_as_float(sv[i + 3]));
            }
            const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
            // lazy rescale of the running accumulator
            const float m_new = fmaxf(m_run, mx);
            const bool need = m_new > m_run && (m_run == -INFINITY || (m_new - m_run) * sc > kRescaleThreshold);
            if (__any_sync(0xffffffffu, need)) {
              const float alpha = need ? (m_run == -INFINITY ? 0.f : ptx::ex2((m_run - m_new) * sc)) : 1.0f;
              if (j > sg.j0) {
                ok = ptx::mbar_wait_lean(sh_addr + static_cast<uint32_t>(offsetof(Shared, pv_done)) + tile * 8, (it - 1) & 1, abort_addr, a.wait_limit_us);
                ok = __ballot_sync(0xffffffffu, ok) == 0xffffffffu;
                if (!ok) break;  // a P.V may still be writing the accumulator
                ptx::tc_fence_after();
                // Two rounds of 16 columns are in flight.  us where the maximum rises by 9 in every step, and normal scores, for rounds
                // one at a time with a wait for each store / this: 16 units of 256 steps 561 / 543, 418 / 420; 2048 x 4096, 32/8 heads
                // 126.2 / 122.5, 103.2 / 103.1.  32 columns at a time: 538, 430; after P, in the registers of S, told to the MMA warp
                // only then: 490, 421 and 116, 106: what rescales in every step is rarer than what hardly ever does.  The pair makes the
                // kernel spill 92 bytes; one round at a time, still with one wait at the end, spills none and is no faster: 564 / 549 where
                // the maximum rises, 425.7 / 426.1 for normal scores.
  #pragma unroll 2
                for (int c = 0; c < 8; ++c) {
                  uint32_t w[16];
                  ptx::tmem_ld16(tO + c * 16, w);
                  ptx::tc_wait_ld();
  #pragma unroll
                  for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * alpha);
                  ptx::tmem_st16(tO + c * 16, w);
                }
                ptx::tc_wait_st();
              }
              l_run *= alpha;
              if (need) m_run = m_new;
            }
            // P = exp2(S*sc - m*sc) -> 16-bit, where the P before it was.  Masked entries are -inf -> 0; a row
            // that has seen nothing yet (m = -inf) produces zeros.
            const float neg_m = m_run == -INFINITY ? 0.f : -m_run * sc;
            const uint32_t half_bar = tile_bars + offsetof(TileBars, p_part);
            CA_PROF(3)
            auto p_free = [&] {  // a fresh barrier counts its phase -1 as complete
              ok = ptx::mbar_wait_lean(sh_addr + static_cast<uint32_t>(offsetof(Shared, pv_done)) + tile * 8, (it - 1) & 1, abort_addr, a.wait_limit_us);
              __syncwarp();
              ptx::tc_fence_after();
            };
            l_run += exp_pack_store<T>(sv, sc, neg_m, tP, half_bar, p_free);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            CA_PROF(4)

          }
          if (ok) ok = ptx::mbar_wait_lean(sh_addr + static_cast<uint32_t>(offsetof(Shared, pv_done)) + tile * 8, (it - 1) & 1, abort_addr, a.wait_limit_us);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          ptx::tc_fence_after();
          const bool live = (r < a.tpt * a.G) && (t < a.Q);
          if (sg.slot < 0) {
            // whole unit: normalise and write the output rows
            const float inv_l = 1.0f / l_run;
            T* orow = reinterpret_cast<T*>(a.out) + b * a.o_stride_b + static_cast<long long>(t) * a.o_stride_t +
                      static_cast<long long>(hkv * a.G + g) * a.o_stride_h;
  #pragma unroll
            for (int c = 0; c < 4; ++c) {
              ptx::tmem_ld32(tO + c * 32, v);
              ptx::tc_wait_ld();
              if (live) {
  #pragma unroll
                for (int i = 0; i < 32; i += 8) {
                  uint4 w;
                  w.x = pack2<T>(__uint_as_float(v[i + 0]) * inv_l, __uint_as_float(v[i + 1]) * inv_l);
                  w.y = pack2<T>(__uint_as_float(v[i + 2]) * inv_l, __uint_as_float(v[i + 3]) * inv_l);
                  w.z = pack2<T>(__uint_as_float(v[i + 4]) * inv_l, __uint_as_float(v[i + 5]) * inv_l);
                  w.w = pack2<T>(__uint_as_float(v[i + 6]) * inv_l, __uint_as_float(v[i + 7]) * inv_l);
                  *reinterpret_cast<uint4*>(orow + c * 32 + i) = w;
                }
              }
            }
            if (live && a.lse) {
              a.lse[(static_cast<long long>(b) * (a.Hkv * a.G) + hkv * a.G + g) * a.Q + t] =
                  0.6931471805599453f * (m_run * sc + log2f(l_run));
            }
          } else {
            // segment of a split unit: unnormalised accumulator, running max and sum to the workspace
            float* po = a.part_o + static_cast<long long>(sg.slot) * kPartialOFloats + tile * (kTileM * kHeadDim);
            float* pml = a.part_ml + static_cast<long long>(sg.slot) * kPartialMLFloats + (tile * kTileM + r) * 2;
  #pragma unroll
            for (int c = 0; c < 4; ++c) {
              ptx::tmem_ld32(tO + c * 32, v);
              ptx::tc_wait_ld();
  #pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const int c4 = (c * 32 + i) >> 2;
                *reinterpret_cast<uint4*>(po + (static_cast<long long>(c4) * kTileM + r) * 4) =
                    make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
              }
            }
            pml[0] = m_run;
            pml[1] = l_run;
          }
          // the accumulator may be overwritten by the next segment
          ptx::tc_fence_before();
          ptx::mbar_arrive(tile_bars + offsetof(TileBars, o_free));
          ++seg_seq;
          CA_PROF(5)
        }
        if ((tid & 127) == 0) CA_PROF_FLUSH(10 + 10 * tile)
      }
      ok = __syncthreads_and(ok ? 1 : 0) != 0;  // all roles finished this batch (or aborted)
      if (!ok) break;
    }
  }

  // ---- teardown: every thread arrives here on every path ----
  if (sh->abort_flag) {
    if (warp == 9 && lane == 0) {
      // drain: give copies already issued a bounded chance to land before the CTA exits
      for (int e = (ring_n > kStages ? ring_n - kStages : 0); e < ring_n; ++e) {
        int dummy = 0;
        ptx::mbar_wait_bounded(ptx::smem_u32(&sh->ring_full[e % kStages]), (e / kStages) & 1, &dummy, 100000000ull);
      }
      for (int tile = 0; tile < 2 && q_issued > 0; ++tile) {
        int dummy = 0;
        ptx::mbar_wait_bounded(ptx::smem_u32(&sh->q_full[tile]), (q_issued - 1) & 1, &dummy, 100000000ull);
      }
    }
    if (warp == 8) {
      // drain the tensor pipe (bounded) before TMEM is released
      ptx::tc_commit_if(ptx::elect_one(), ptx::smem_u32(&sh->drain));
      int dummy = 0;
      ptx::mbar_wait_bounded(ptx::smem_u32(&sh->drain), 0, &dummy, 100000000ull);
    }
  }
  if (bad_index && a.status) atomicOr(a.status, CA_STATUS_BAD_INDEX);
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
  if (tid == 0 && sh->abort_flag && a.status) atomicOr(a.status, CA_STATUS_TIMEOUT);
#if CA_ATTN_PROFILE
  if (tid == 0) g_prof[blockIdx.x][31] = clock64() - prof_kernel_t0;  // whole kernel
#endif
}

// Merges the segments of every split unit.  One CTA per (attention CTA, tile, column part); the CTAs whose odd slot
// holds the first segment of a unit (j0 == 0) find the unit's others in the even slots of the CTAs that follow.  Thread =
// tile row.  A chain of memory latencies (descriptors, maxima and sums, accumulators), so all that can be asked for at once is:
// the descriptors by all threads together, and the accumulators of kBatch segments while the maxima are still on their way.
// Against one thread walking the descriptors and weights kept in shared memory before any accumulator was loaded, us of attention and
// merge in a loop: 256 x 8K, 8 KV heads, 27.1 -> 24.9; 1024 x 128K, one KV head 71.4 -> 69.0; 1024 x 32K 227.0 -> 225.9.  Batches of 8
// in 16 parts where a unit has five pieces or more: 28.5, 70.2.
constexpr int kMergeAhead = 2 * kTileM;  // following CTAs looked at
constexpr int kBatch = 4;                // segments in flight
constexpr int kParts = 8;                // column parts per tile

template <typename T>
__global__ void __launch_bounds__(kTileM) attn_combine_kernel(const KernelArgs a, int n_slots) {
  constexpr int kC8 = kHeadDim / 8 / kParts;  // 8-column groups per part
  ptx::grid_launch_dependents();
  ptx::grid_dependency_wait();  // nothing in global memory is touched before this
  __shared__ int chain_sh[1 + kMergeAhead];
  __shared__ uint32_t hit_sh[kMergeAhead / 32];
  __shared__ int steps_sh[kMergeAhead / 32];
  // blockIdx.x = attention CTA; the first segment of a unit that it cut is in its odd slot
  const int tile = blockIdx.y, part = blockIdx.z, r = threadIdx.x;
  const int slot = 2 * blockIdx.x + 1;
  const SegDesc first = a.descs[slot];
  if (first.unit < 0) return;
#pragma unroll
  for (int i = r; i < kMergeAhead; i += kTileM) {
    const int s = (slot / 2 + 1 + i) * 2;
    SegDesc d;
    d.unit = -1, d.j0 = 0, d.j1 = 0, d.n_iter = 0;
    if (s < n_slots) d = a.descs[s];
    const bool mine = d.unit == first.unit;  // unused slots hold -1
    const uint32_t hits = __ballot_sync(0xffffffffu, mine);
    const int steps = __reduce_add_sync(0xffffffffu, mine ? d.j1 - d.j0 : 0);
    if ((r & 31) == 0) hit_sh[i >> 5] = hits, steps_sh[i >> 5] = steps;
  }
  __syncthreads();
  int n = 1, steps = first.j1 - first.j0;
#pragma unroll
  for (int w = 0; w < kMergeAhead / 32; ++w) {
    const uint32_t hits = hit_sh[w];
    if ((r >> 5) == (w & (kTileM / 32 - 1)) && ((hits >> (r & 31)) & 1u)) {
      chain_sh[n + __popc(hits & ((1u << (r & 31)) - 1u))] = (slot / 2 + 1 + w * 32 + (r & 31)) * 2;
    }
    n += __popc(hits);
    steps += steps_sh[w];
  }
  if (r == 0) chain_sh[0] = slot;
  __syncthreads();
  if (first.j0 != 0 || steps != first.n_iter) {
    if (r == 0 && part == 0 && a.status) atomicOr(a.status, CA_STATUS_BAD_INDEX);
    return;
  }
  const int row = first.unit / a.n_pairs, pair = first.unit % a.n_pairs;
  const int b = row / a.Hkv, hkv = row % a.Hkv;
  const int t = (2 * pair + tile) * a.tpt + r / a.G;
  const int g = r % a.G;
  const bool live = (r < a.tpt * a.G) && (t < a.Q);
  const float sc = a.scale_log2;
  float4 x[kBatch][2];
  auto load_o = [&](int i0, int cc) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      if (i0 + k >= n) break;
      const float* po = a.part_o + static_cast<long long>(chain_sh[i0 + k]) * kPartialOFloats + tile * (kTileM * kHeadDim);
      const int c4 = 2 * (part * kC8 + cc);
      x[k][0] = *reinterpret_cast<const float4*>(po + (static_cast<long long>(c4) * kTileM + r) * 4);
      x[k][1] = *reinterpret_cast<const float4*>(po + (static_cast<long long>(c4 + 1) * kTileM + r) * 4);
    }
  };
  auto ml_of = [&](int i) {
    return *reinterpret_cast<const float2*>(a.part_ml + static_cast<long long>(chain_sh[i]) * kPartialMLFloats + (tile * kTileM + r) * 2);
  };
  load_o(0, 0);
  float m = -INFINITY;
#pragma unroll kBatch
  for (int i = 0; i < n; ++i) m = fmaxf(m, ml_of(i).x);
  float l = 0.f;
  float acc[kC8][8] = {};
  for (int i0 = 0; i0 < n; i0 += kBatch) {
    float w[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      if (i0 + k >= n) break;
      const float2 ml = ml_of(i0 + k);
      w[k] = ml.x == -INFINITY ? 0.f : ptx::ex2((ml.x - m) * sc);
      l += ml.y * w[k];
    }
#pragma unroll
    for (int cc = 0; cc < kC8; ++cc) {
      if (i0 > 0 || cc > 0) load_o(i0, cc);
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (i0 + k >= n) break;
        acc[cc][0] += w[k] * x[k][0].x, acc[cc][1] += w[k] * x[k][0].y, acc[cc][2] += w[k] * x[k][0].z, acc[cc][3] += w[k] * x[k][0].w;
        acc[cc][4] += w[k] * x[k][1].x, acc[cc][5] += w[k] * x[k][1].y, acc[cc][6] += w[k] * x[k][1].z, acc[cc][7] += w[k] * x[k][1].w;
      }
    }
  }
  const float inv_l = 1.0f / l;
  T* orow = reinterpret_cast<T*>(a.out) + b * a.o_stride_b + static_cast<long long>(t) * a.o_stride_t +
            static_cast<long long>(hkv * a.G + g) * a.o_stride_h;
  if (live) {
#pragma unroll
    for (int cc = 0; cc < kC8; ++cc) {
      uint4 w;
      w.x = pack2<T>(acc[cc][0] * inv_l, acc[cc][1] * inv_l);
      w.y = pack2<T>(acc[cc][2] * inv_l, acc[cc][3] * inv_l);
      w.z = pack2<T>(acc[cc][4] * inv_l, acc[cc][5] * inv_l);
      w.w = pack2<T>(acc[cc][6] * inv_l, acc[cc][7] * inv_l);
      *reinterpret_cast<uint4*>(orow + (part * kC8 + cc) * 8) = w;
    }
    if (part == 0 && a.lse) {
      a.lse[(static_cast<long long>(b) * (a.Hkv * a.G) + hkv * a.G + g) * a.Q + t] = 0.6931471805599453f * (m * sc + log2f(l));
    }
  }
}

static int encode_map(CUtensorMap* map, CUtensorMapDataType dt, int rank, const void* base, const cuuint64_t* dims,
                      const cuuint64_t* strides_bytes, const cuuint32_t* box, const char* what) {
  tensor_map_encode_fn enc = get_tensor_map_encoder();
  if (!enc) return fail(CA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint32_t elem_strides[5] = {1, 1, 1, 1, 1};
  CUresult res = enc(map, dt, static_cast<cuuint32_t>(rank), const_cast<void*>(base), dims, strides_bytes, box,
                     elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (res != CUDA_SUCCESS) return fail(CA_ERR_CUDA, "cuTensorMapEncodeTiled(%s) failed with CUresult %d", what, (int)res);
  return CA_OK;
}

int encode_kv_maps(const ca_attn_params* p, CUtensorMap* k_map, CUtensorMap* v_map, int (&slot_of_role)[3]) {
  const CUtensorMapDataType dt = p->dtype == CA_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  // roles: 0 token-in-page, 1 page, 2 head; outer dimensions sorted by ascending stride
  const cuuint64_t role_dim[3] = {(cuuint64_t)p->kv.page_size, (cuuint64_t)p->kv.num_pages,
                                  (cuuint64_t)(p->Hkv / (p->kv.head_div > 1 ? p->kv.head_div : 1))};
  const cuuint64_t role_stride[3] = {(cuuint64_t)p->kv.token_stride * 2, (cuuint64_t)p->kv.page_stride * 2,
                                     (cuuint64_t)p->kv.head_stride * 2};
  const cuuint32_t role_box[3] = {64, 1, 1};
  int order[3] = {0, 1, 2};
  for (int i = 0; i < 3; ++i)
    for (int j = i + 1; j < 3; ++j)
      if (role_stride[order[j]] < role_stride[order[i]]) { int t = order[i]; order[i] = order[j]; order[j] = t; }
  cuuint64_t dims[4] = {(cuuint64_t)kHeadDim, 0, 0, 0};
  cuuint64_t strides[3];
  cuuint32_t box[4] = {64, 0, 0, 0};
  for (int i = 0; i < 3; ++i) {
    dims[i + 1] = role_dim[order[i]];
    strides[i] = role_stride[order[i]];
    box[i + 1] = role_box[order[i]];
    slot_of_role[order[i]] = i;
  }
  const int rc = encode_map(k_map, dt, 4, p->kv.k, dims, strides, box, "k");
  return rc != CA_OK ? rc : encode_map(v_map, dt, 4, p->kv.v, dims, strides, box, "v");
}

std::mutex& pair_mutex(cudaStream_t stream) {
  static std::mutex mu[64];  // more streams than this share; a collision costs a wait, no more
  return mu[(reinterpret_cast<uintptr_t>(stream) * 0x9E3779B97F4A7C15ull) >> 58];
}

static int validate(const ca_attn_params* p) {
  CA_REQUIRE(p != nullptr, "params is null");
  CA_REQUIRE(p->q && p->out && p->kv.k && p->kv.v, "q, out, kv.k and kv.v must be non-null");
  CA_REQUIRE(p->D == kHeadDim, "head dim must be 128, got %d", p->D);
  CA_REQUIRE(p->dtype == CA_DTYPE_BF16 || p->dtype == CA_DTYPE_F16, "dtype must be bf16 or f16");
  CA_REQUIRE(p->B > 0 && p->Q > 0 && p->Hq > 0 && p->Hkv > 0, "B, Q, Hq, Hkv must be positive");
  CA_REQUIRE(p->Hq % p->Hkv == 0, "Hq (%d) must be a multiple of Hkv (%d)", p->Hq, p->Hkv);
  CA_REQUIRE(p->kv.head_div >= 0 && (p->kv.head_div <= 1 || p->Hkv % p->kv.head_div == 0),
             "kv.head_div (%d) must divide the number of block-table rows per batch entry (Hkv = %d)", p->kv.head_div, p->Hkv);
  CA_REQUIRE(p->Hq / p->Hkv <= 128, "GQA group larger than 128 is not supported");
  CA_REQUIRE(static_cast<long long>(p->B) * p->Hkv <= kMaxRows, "more than %d (batch x kv head) rows are not supported", kMaxRows);
  CA_REQUIRE(p->block_size > 0 && p->block_size % kSub == 0, "block_size must be a positive multiple of 64");
  CA_REQUIRE(p->kv_len >= p->Q, "kv_len (%d) must be >= Q (%d)", p->kv_len, p->Q);
  CA_REQUIRE((p->kv_len - p->Q) % p->block_size == 0 || p->block_idx == nullptr,
             "with a block table the past length (kv_len - Q = %d) must be a multiple of block_size (%d)", p->kv_len - p->Q,
             p->block_size);
  CA_REQUIRE(p->kv.page_size > 0 && (p->kv.page_size % kSub == 0 || p->kv.pages_per_seq == 1),
             "page_size must be a positive multiple of 64 (any length when a sequence is one page)");
  CA_REQUIRE(p->kv.num_pages > 0 && p->kv.pages_per_seq > 0, "num_pages and pages_per_seq must be positive");
  CA_REQUIRE((long long)p->kv.pages_per_seq * p->kv.page_size >= p->kv_len,
             "pages_per_seq*page_size (%lld) does not cover kv_len (%d)",
             (long long)p->kv.pages_per_seq * p->kv.page_size, p->kv_len);
  CA_REQUIRE(p->kv.page_stride % 8 == 0 && p->kv.token_stride % 8 == 0 && p->kv.head_stride % 8 == 0,
             "kv strides must be multiples of 8 elements (16 bytes)");
  CA_REQUIRE(p->q_stride_b % 8 == 0 && p->q_stride_t % 8 == 0 && p->q_stride_h % 8 == 0,
             "q strides must be multiples of 8 elements (16 bytes)");
  CA_REQUIRE(p->o_stride_b % 8 == 0 && p->o_stride_t % 8 == 0 && p->o_stride_h % 8 == 0,
             "out strides must be multiples of 8 elements (16 bytes)");
  CA_REQUIRE((reinterpret_cast<uintptr_t>(p->q) | reinterpret_cast<uintptr_t>(p->out) |
              reinterpret_cast<uintptr_t>(p->kv.k) | reinterpret_cast<uintptr_t>(p->kv.v)) % 16 == 0,
             "q, out, k, v must be 16-byte aligned");
  if (p->block_idx) {
    CA_REQUIRE(p->counts != nullptr, "counts is required with block_idx");
    CA_REQUIRE(p->block_idx_stride > 0 || p->kv_len == p->Q, "block_idx_stride must be positive");
  }
  CA_REQUIRE(p->workspace == nullptr || reinterpret_cast<uintptr_t>(p->workspace) % 256 == 0,
             "workspace must be 256-byte aligned");
  return CA_OK;
}

// Workspace layout for a grid of nc CTAs: descriptors, then (max, sum) pairs, then accumulators.
static size_t desc_bytes(int nc) { return ((static_cast<size_t>(2) * nc * sizeof(SegDesc) + 255) / 256) * 256; }
static size_t ml_bytes(int nc) { return static_cast<size_t>(2) * nc * kPartialMLFloats * sizeof(float); }
static size_t o_bytes(int nc) { return static_cast<size_t>(2) * nc * kPartialOFloats * sizeof(float); }
static size_t workspace_bytes_for(int nc) { return desc_bytes(nc) + ml_bytes(nc) + o_bytes(nc); }


// ---- scratch for callers that cannot allocate -------------------------------------------------
// Room for the split-unit partials of a grid of up to kStaticMaxCtas CTAs (a B200 has 148 SMs):
// 160 * 2 slots * (128 KiB accumulator + 2 KiB max/sum) + descriptors = 41.6 MiB, resident on every
// GPU that loads the library until the process exits.
constexpr int kStaticMaxCtas = 160;
constexpr size_t kStaticScratchBytes =
    ((2 * kStaticMaxCtas * sizeof(SegDesc) + 255) / 256) * 256 +
    static_cast<size_t>(2) * kStaticMaxCtas * (kPartialMLFloats + kPartialOFloats) * sizeof(float);
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// Device address of g_static_scratch on the current device.  In host code the array's name is only
// a stand-in for the symbol, not a pointer a kernel can use, so the address is asked from the
// runtime once per device (with that device current) and remembered.
static int static_scratch_address(void** out) {
  static std::mutex mu;
  static void* cached[64] = {nullptr};
  int dev = 0;
  CA_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(CA_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == nullptr) {
    void* ptr = nullptr;
    cudaError_t err = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (err != cudaSuccess || ptr == nullptr) {
      return fail(CA_ERR_CUDA, "cudaGetSymbolAddress(static attention scratch) failed: %s", cudaGetErrorString(err));
    }
    cached[dev] = ptr;
  }
  *out = cached[dev];
  return CA_OK;
}

}  // namespace attn
}  // namespace ca

extern "C" {

int ca_attn_workspace_bytes(const ca_attn_params* p, size_t* bytes_out) {
  using namespace ca;
  CA_REQUIRE(bytes_out != nullptr, "bytes_out is null");
  int rc = attn::validate(p);
  if (rc != CA_OK) return rc;
  DeviceInfo dev;
  rc = get_device_info(&dev);
  if (rc != CA_OK) return rc;
  *bytes_out = attn::workspace_bytes_for(dev.sm_count);
  return CA_OK;
}

int ca_attn_compact(const ca_attn_params* p, ca_stream_t stream_) {
  using namespace ca;
  using namespace ca::attn;
  int rc = validate(p);
  if (rc != CA_OK) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  DeviceInfo dev;
  rc = get_device_info(&dev);
  if (rc != CA_OK) return rc;
  if (dev.cc_major != 10) return fail(CA_ERR_UNSUPPORTED, "this library targets sm_100a; device is sm_%d%d", dev.cc_major, dev.cc_minor);
  if (decode_applies(p)) return launch_decode(p, dev, stream);

  const int G = p->Hq / p->Hkv;
  const int tpt = kTileM / G;
  const int n_mtiles = ceil_div(p->Q, tpt);
  const int n_pairs = ceil_div(n_mtiles, 2);
  const CUtensorMapDataType dt = p->dtype == CA_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;

  CUtensorMap q_map, k_map, v_map;
  int slots[3];
  {
    // (d, g, hkv, token, batch): the box walks g fastest, then tokens, so tile row = token*G + g
    cuuint64_t dims[5] = {(cuuint64_t)kHeadDim, (cuuint64_t)G, (cuuint64_t)p->Hkv, (cuuint64_t)p->Q, (cuuint64_t)p->B};
    cuuint64_t strides[4] = {(cuuint64_t)p->q_stride_h * 2, (cuuint64_t)p->q_stride_h * G * 2,
                             (cuuint64_t)p->q_stride_t * 2, (cuuint64_t)p->q_stride_b * 2};
    cuuint32_t box[5] = {64, (cuuint32_t)G, 1, (cuuint32_t)tpt, 1};
    rc = encode_map(&q_map, dt, 5, p->q, dims, strides, box, "q");
    if (rc != CA_OK) return rc;
  }
  rc = encode_kv_maps(p, &k_map, &v_map, slots);
  if (rc != CA_OK) return rc;

  KernelArgs a;
  a.Q = p->Q;
  a.G = G;
  a.Hkv = p->Hkv;
  a.B = p->B;
  a.tpt = tpt;
  a.n_pairs = n_pairs;
  a.block_size = p->block_size;
  // a dense launch whose past is not a block multiple treats the remainder as the head of the chunk region
  a.q_off = (p->kv_len - p->Q) % p->block_size;
  a.past_tokens = p->kv_len - p->Q - a.q_off;
  a.past_blocks = a.past_tokens / p->block_size;
  a.spb = p->block_size / kSub;
  a.page_size = p->kv.page_size;
  a.pages_per_seq = p->kv.pages_per_seq;
  a.num_pages = p->kv.num_pages;
  a.block_idx = p->block_idx;
  a.block_idx_stride = p->block_idx_stride;
  a.counts = p->counts;
  a.page_table = p->kv.page_table;
  a.out = p->out;
  a.o_stride_b = p->o_stride_b;
  a.o_stride_t = p->o_stride_t;
  a.o_stride_h = p->o_stride_h;
  a.lse = p->lse;
  a.scale_log2 = p->softmax_scale * 1.4426950408889634f;
  a.status = p->status;
  const uint32_t fmt = p->dtype == CA_DTYPE_BF16 ? 1u : 0u;
  a.idesc_qk = ptx::make_idesc_f16(fmt, kTileM, kTileN, 0, 0);
  a.idesc_pv = ptx::make_idesc_f16(fmt, kTileM, kHeadDim, 0, 1);
  a.wait_limit_ns = 2000000000ull;
  a.wait_limit_us = 2000000u;
  a.kv_head_div = p->kv.head_div > 1 ? p->kv.head_div : 1;
  a.slot_tok = slots[0];
  a.slot_page = slots[1];
  a.slot_head = slots[2];

  // persistent grid: one CTA per SM, never more CTAs than units when units cannot be cut
  const long long n_units = static_cast<long long>(p->B) * p->Hkv * n_pairs;
  int grid = dev.sm_count;
  const int cap_blocks = p->block_idx && p->block_idx_stride < a.past_blocks ? p->block_idx_stride : a.past_blocks;
  const bool can_split = p->workspace != nullptr && p->workspace_bytes >= workspace_bytes_for(grid);
  a.split = can_split && may_be_cut(a, p->B * p->Hkv, cap_blocks, p->block_idx == nullptr, grid) ? 1 : 0;
  if (!a.split && n_units < grid) grid = static_cast<int>(n_units);
  a.descs = nullptr, a.part_ml = nullptr, a.part_o = nullptr;
  if (a.split) {
    uint8_t* ws = static_cast<uint8_t*>(p->workspace);
    a.descs = reinterpret_cast<SegDesc*>(ws);
    a.part_ml = reinterpret_cast<float*>(ws + desc_bytes(grid));
    a.part_o = reinterpret_cast<float*>(ws + desc_bytes(grid) + ml_bytes(grid));
  }

  // the opt-in shared-memory size is a per-device function attribute: set once per device and type
  // (the call costs a few microseconds of host time, which short contexts notice)
  {
    static std::mutex mu;
    static bool done[2][64] = {};
    const int ti = p->dtype == CA_DTYPE_BF16 ? 0 : 1;
    std::lock_guard<std::mutex> lock(mu);
    if (!done[ti][dev.ordinal]) {
      if (ti == 0) {
        CA_CUDA(cudaFuncSetAttribute(attn_compact_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
      } else {
        CA_CUDA(cudaFuncSetAttribute(attn_compact_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
      }
      done[ti][dev.ordinal] = true;
    }
  }
  std::unique_lock<std::mutex> pair(pair_mutex(stream), std::defer_lock);
  if (a.split) pair.lock();
  if (p->dtype == CA_DTYPE_BF16) {
    // a programmatic dependent launch: barrier set-up, TMEM allocation and descriptor prefetch overlap the tail of
    // the table builder; the kernel waits (griddepcontrol.wait) before it reads anything from global memory
    launch_kernel_as(true, attn_compact_kernel<__nv_bfloat16>, dim3(grid), dim3(kThreads), kSmemBytes, stream, q_map, k_map, v_map, a);
  } else {
    launch_kernel_as(true, attn_compact_kernel<__half>, dim3(grid), dim3(kThreads), kSmemBytes, stream, q_map, k_map, v_map, a);
  }
  CA_LAUNCH_CHECK("attn_compact_kernel");
  if (a.split) {
    if (p->dtype == CA_DTYPE_BF16) {
      launch_kernel_as(CA_ATTN_MERGE_DEPENDENT != 0, attn_combine_kernel<__nv_bfloat16>, dim3(grid, 2, kParts), dim3(kTileM), 0, stream, a, 2 * grid);
    } else {
      launch_kernel_as(CA_ATTN_MERGE_DEPENDENT != 0, attn_combine_kernel<__half>, dim3(grid, 2, kParts), dim3(kTileM), 0, stream, a, 2 * grid);
    }
    CA_LAUNCH_CHECK("attn_combine_kernel");
  }
  return CA_OK;
}

int ca_attn_compact_static_scratch(const ca_attn_params* p, ca_stream_t stream) {
  using namespace ca;
  using namespace ca::attn;
  int rc = validate(p);
  if (rc != CA_OK) return rc;
  DeviceInfo dev;
  rc = get_device_info(&dev);
  if (rc != CA_OK) return rc;
  const size_t need = workspace_bytes_for(dev.sm_count);
  if (need > kStaticScratchBytes) {
    return fail(CA_ERR_CAPACITY,
                "this device has %d SMs and needs %zu bytes of attention scratch; the built-in scratch holds %zu bytes "
                "(up to %d SMs): use ca_attn_compact with a caller-provided workspace",
                dev.sm_count, need, kStaticScratchBytes, kStaticMaxCtas);
  }
  void* scratch = nullptr;
  rc = static_scratch_address(&scratch);  // first call on a device looks the address up
  if (rc != CA_OK) return rc;
  ca_attn_params q = *p;
  q.workspace = scratch;
  q.workspace_bytes = kStaticScratchBytes;
  return ca_attn_compact(&q, stream);
}

}  // extern "C"

#if CA_ATTN_PROFILE
// Development builds only: copies the cycle counters of the last launch to the host.
extern "C" int ca_debug_attn_profile(long long* dst) {
  return cudaMemcpyFromSymbol(dst, ca::attn::g_prof, sizeof(long long) * 160 * 32) == cudaSuccess ? 0 : -3;
}
#endif
