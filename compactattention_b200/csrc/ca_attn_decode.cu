// Block-table attention for few query rows (decode): Q * G <= 16 rows per KV head.
//
// Bound by the bytes of K and V, so the design is about keeping copies in flight and the result on chip:
// * the KV of one (batch, KV head) row is cut over the CTAs of a cluster (1..8) and, when rows are too few to
//   fill the GPU even so, over several clusters;
// * a CTA streams 64-token sub-blocks (K and V, 32 KB) through a three-stage TMA ring; two CTAs share an SM, so
//   192 KB are in flight per SM;
// * each of four warps owns 16 of a sub-block's tokens with running max / sum / accumulator of its own
//   (mma.sync m16n8k16: a 16-row tile has no use for a 128-row tcgen05 tile, whose softmax would run on 124 dead
//   rows), so there is no hand-off between warps inside the loop;
// * the warps merge in shared memory, the CTAs of a cluster through distributed shared memory: one launch and no
//   scratch in global memory.  Only rows cut over several clusters leave partials in the workspace and are
//   merged by a dependent launch.
//
// Measured on B200 (32/8 heads, bf16; through the 256-row kernel -> here): 8 sequences of 32768 tokens 267 -> 162 us
// (1.07 GB, 6.64 TB/s), one of 131072 145 -> 85 us, one of 4001 31 -> 8.3 us; one KV head, 131072 tokens 184 -> 19 us;
// 16 x 8192, 28/4 heads 81 -> 45 us.
#include "ca_attn_plan.cuh"
#include "ca_attn_shared.cuh"
#include "ca_ring.cuh"

#include <cooperative_groups.h>
#include <mutex>

namespace ca {
namespace attn {
namespace decode {

namespace cg = cooperative_groups;

constexpr int kHeadDim = 128;
constexpr int kRows = 16;  // query rows of one mma tile
constexpr int kWarps = 4;  // consumer warps; one producer warp follows
constexpr int kThreads = (kWarps + 1) * 32;
constexpr int kStages = 3;
constexpr int kBoxBytes = kSub * 128;       // [64 tokens][64 channels]
constexpr int kStageBytes = 4 * kBoxBytes;  // K low / high channels, V low / high channels
constexpr int kMinSubsPart = 8;    // sub-blocks a CTA should have of a row that is cut over several clusters (the merge launch)

struct Args {
  const void* q;
  long long q_stride_b, q_stride_t, q_stride_h;
  void* out;
  long long o_stride_b, o_stride_t, o_stride_h;
  int Q, G, Hkv, rows;  // rows = Q * G
  int past_blocks, spb, block_size, past_tokens, q_off;
  int page_size, pages_per_seq, num_pages;
  const int32_t* block_idx;
  int block_idx_stride;
  const int32_t* counts;
  const int32_t* page_table;
  float* lse;
  float scale_log2;
  int32_t* status;
  unsigned long long wait_limit_ns;
  int slot_tok, slot_page, slot_head, kv_head_div;
  int parts;       // clusters per row
  float* part_o;   // [R][parts][kRows][kHeadDim], parts > 1 only
  float2* part_ml; // [R][parts][kRows]
};

struct Shared {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  int abort_flag;
  float2 warp_ml[kWarps][kRows];
  float2 cta_ml[kRows];                    // read by the cluster
  __align__(16) float cta_o[kRows][kHeadDim];  // read by the cluster
};
constexpr int kSmemBytes = kStages * kStageBytes + 1024 + static_cast<int>(sizeof(Shared));
static_assert(kWarps * kRows * kHeadDim * 4 <= kStages * kStageBytes, "the warps' partials reuse the ring");
static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs share an SM");

template <typename T>
struct Half2;
template <>
struct Half2<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
};
template <>
struct Half2<__half> {
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
};

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// Byte offset of 16-byte piece `piece` (0..15) of token `tok` inside a [64][128]-channel stage half
// (two 64-channel boxes, 128-byte swizzle).
__device__ __forceinline__ uint32_t piece_offset(int tok, int piece) {
  return static_cast<uint32_t>((piece >> 3) * kBoxBytes + tok * 128 + (((piece & 7) ^ (tok & 7)) << 4));
}
__device__ __forceinline__ float quad_max(float x) {
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
  return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
}
__device__ __forceinline__ float quad_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  return x + __shfl_xor_sync(0xffffffffu, x, 2);
}
__device__ __forceinline__ float weight(float m_part, float m, float sc) {
  return m_part == -INFINITY ? 0.f : ptx::ex2((m_part - m) * sc);
}

template <typename T>
__device__ __forceinline__ void store_row4(const Args& a, int row, int i, int d, float4 o, float l) {
  const int b = row / a.Hkv, hkv = row % a.Hkv, t = i / a.G, g = i % a.G;
  const float inv_l = 1.0f / l;
  T* p = reinterpret_cast<T*>(a.out) + b * a.o_stride_b + static_cast<long long>(t) * a.o_stride_t +
         static_cast<long long>(hkv * a.G + g) * a.o_stride_h + d;
  *reinterpret_cast<uint2*>(p) = make_uint2(Half2<T>::pack(o.x * inv_l, o.y * inv_l), Half2<T>::pack(o.z * inv_l, o.w * inv_l));
}
__device__ __forceinline__ void store_lse(const Args& a, int row, int i, float m, float l) {
  const int b = row / a.Hkv, hkv = row % a.Hkv, t = i / a.G, g = i % a.G;
  a.lse[(static_cast<long long>(b) * (a.Hkv * a.G) + hkv * a.G + g) * a.Q + t] = 0.6931471805599453f * (m * a.scale_log2 + log2f(l));
}

// Some wait of this CTA expired, maybe a consumer's after the producer had issued everything: copies already issued get a
// bounded chance to land before the CTA exits (all threads; `issued` is the producer lane's).  Out of line: between the
// cluster's last barrier and the exit the code itself is not in the instruction cache (inline: 18.9 -> 21.0 us for
// 131072 tokens of one KV head, 87.4 -> 91.4 for eight).
__device__ __noinline__ void give_up(int32_t* status, Shared* sh, int issued) {
  if (threadIdx.x == kWarps * 32) {
    drain_ring(issued, kStages, [&](int s, uint32_t parity) {
      int dummy = 0;
      ptx::mbar_wait_bounded(ptx::smem_u32(&sh->full[s]), parity, &dummy, 100000000ull);
    });
  }
  if (threadIdx.x == 0 && status) atomicOr(status, CA_STATUS_TIMEOUT);
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 2)
    attn_decode_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, const Args a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t ring = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* ring_ptr = smem_raw + (ring - ptx::smem_u32(smem_raw));
  Shared* sh = reinterpret_cast<Shared*>(ring_ptr + kStages * kStageBytes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const int cluster_id = blockIdx.x / cs;
  const int row = cluster_id / a.parts, part = cluster_id % a.parts;
  volatile int* abort_flag = &sh->abort_flag;
  const uint64_t limit = a.wait_limit_ns;

  ptx::grid_launch_dependents();
  if (tid == 0) {
    sh->abort_flag = 0;
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(ptx::smem_u32(&sh->full[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&sh->empty[s]), kWarps);
    }
    ptx::mbar_fence_init();
    ptx::fence_proxy_async_smem();
    ptx::tma_prefetch_desc(&k_map);
    ptx::tma_prefetch_desc(&v_map);
  }
  __syncthreads();
  ptx::grid_dependency_wait();  // nothing in global memory is touched before this

  // this CTA's sub-blocks of the row
  bool bad_index = false;
  int count = a.past_blocks;
  if (a.block_idx != nullptr) {
    count = a.counts[row];
    const int cap = a.block_idx_stride < a.past_blocks ? a.block_idx_stride : a.past_blocks;
    if (count < 0 || count > cap) {
      bad_index = true;
      count = count < 0 ? 0 : cap;
    }
  }
  const int n_past_sub = count * a.spb;
  const int n_sub = n_past_sub + (a.Q - 1 + a.q_off) / kSub + 1;
  const long long slices = static_cast<long long>(a.parts) * cs, slice = static_cast<long long>(part) * cs + rank;
  const int u0 = static_cast<int>(n_sub * slice / slices), u1 = static_cast<int>(n_sub * (slice + 1) / slices);
  int issued = 0;  // ring entries whose copies have been issued (producer lane)

  if (warp == kWarps) {
    // =============================== TMA producer ===============================
    const int b = row / a.Hkv, head = (row % a.Hkv) / a.kv_head_div;
    bool ok = true;
    for (int base = u0; base < u1 && ok; base += 32) {
      // every lane resolves one sub-block of this batch of 32
      const int u = base + lane;
      int page = 0, off = 0;
      if (u < u1) {
        int tok;
        if (u < n_past_sub) {
          const int bi = u / a.spb;
          int blk = a.block_idx ? a.block_idx[static_cast<long long>(row) * a.block_idx_stride + bi] : bi;
          if (blk < 0 || blk >= a.past_blocks) {
            bad_index = true;
            blk = blk < 0 ? 0 : a.past_blocks - 1;
          }
          tok = blk * a.block_size + (u - bi * a.spb) * kSub;
        } else {
          tok = a.past_tokens + (u - n_past_sub) * kSub;
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
      const int m = u1 - base < 32 ? u1 - base : 32;
      for (int i = 0; i < m && ok; ++i) {
        const int p0 = __shfl_sync(0xffffffffu, page, i), o0 = __shfl_sync(0xffffffffu, off, i);
        if (lane == 0) {
          const int s = issued % kStages;
          ok = ptx::mbar_wait_bounded(ptx::smem_u32(&sh->empty[s]), ((issued / kStages) & 1) ^ 1u, abort_flag, limit);
          if (ok) {
            const uint32_t bar = ptx::smem_u32(&sh->full[s]), dst = ring + s * kStageBytes;
            ptx::mbar_expect_tx(bar, kStageBytes);
            int c[3];
            c[a.slot_tok] = o0, c[a.slot_page] = p0, c[a.slot_head] = head;
            for (int h = 0; h < 2; ++h) ptx::tma_load_4d(dst + h * kBoxBytes, &k_map, bar, h * 64, c[0], c[1], c[2]);
            for (int h = 0; h < 2; ++h) ptx::tma_load_4d(dst + (2 + h) * kBoxBytes, &v_map, bar, h * 64, c[0], c[1], c[2]);
            ++issued;
          }
        }
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      }
    }
  } else {
    // =============================== attention ===============================
    const int r0 = lane >> 2, r1 = r0 + 8;  // the two query rows of this thread
    const int b = row / a.Hkv, hkv = row % a.Hkv;
    uint32_t qf[8][4];
    {
      auto load_row = [&](int i, int half) {
        const bool live = i < a.rows;
        const int t = live ? i / a.G : 0, g = live ? i % a.G : 0;
        const uint16_t* p = reinterpret_cast<const uint16_t*>(a.q) + b * a.q_stride_b + static_cast<long long>(t) * a.q_stride_t +
                            static_cast<long long>(hkv * a.G + g) * a.q_stride_h + (lane & 3) * 2;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          qf[k][half] = live ? *reinterpret_cast<const uint32_t*>(p + k * 16) : 0u;
          qf[k][half + 2] = live ? *reinterpret_cast<const uint32_t*>(p + k * 16 + 8) : 0u;
        }
      };
      load_row(r0, 0);
      load_row(r1, 1);
    }
    float o[16][4];
#pragma unroll
    for (int d = 0; d < 16; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[d][e] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    const float sc = a.scale_log2;
    const int k_tok = warp * 16 + ((lane >> 4) << 3) + (lane & 7), k_piece = (lane >> 3) & 1;
    const int v_tok = warp * 16 + (((lane >> 3) & 1) << 3) + (lane & 7), v_piece = lane >> 4;
    bool ok = true;
    int n = 0;
    for (int u = u0; u < u1; ++u, ++n) {
      const int s = n % kStages;
      ok = ptx::mbar_wait_bounded(ptx::smem_u32(&sh->full[s]), (n / kStages) & 1, abort_flag, limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const uint32_t ks = ring + s * kStageBytes, vs = ks + 2 * kBoxBytes;
      float sv[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        uint32_t kf[4];
        ldsm4(ks + piece_offset(k_tok, 2 * k + k_piece), kf);
        Half2<T>::mma(sv[0], qf[k], kf[0], kf[1]);
        Half2<T>::mma(sv[1], qf[k], kf[2], kf[3]);
      }
      if (u >= n_past_sub) {
        // the chunk's own tokens: causal, counted from the start of the chunk region
        const int col = (u - n_past_sub) * kSub + warp * 16 + (lane & 3) * 2;
        const int lim0 = r0 / a.G + a.q_off, lim1 = r1 / a.G + a.q_off;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (col + nt * 8 + e > lim0) sv[nt][e] = -INFINITY;
            if (col + nt * 8 + e > lim1) sv[nt][2 + e] = -INFINITY;
          }
      }
      const float n0 = fmaxf(m0, quad_max(fmaxf(fmaxf(sv[0][0], sv[0][1]), fmaxf(sv[1][0], sv[1][1]))));
      const float n1 = fmaxf(m1, quad_max(fmaxf(fmaxf(sv[0][2], sv[0][3]), fmaxf(sv[1][2], sv[1][3]))));
      if (__any_sync(0xffffffffu, n0 > m0 || n1 > m1)) {
        const float c0 = weight(m0, n0, sc), c1 = weight(m1, n1, sc);
        l0 *= c0, l1 *= c1;
#pragma unroll
        for (int d = 0; d < 16; ++d) o[d][0] *= c0, o[d][1] *= c0, o[d][2] *= c1, o[d][3] *= c1;
        m0 = n0, m1 = n1;
      }
      // masked entries are -inf -> 0; a row that has seen nothing yet (m = -inf) produces zeros
      const float s0 = m0 == -INFINITY ? 0.f : -m0 * sc, s1 = m1 == -INFINITY ? 0.f : -m1 * sc;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        sv[nt][0] = ptx::ex2(fmaf(sv[nt][0], sc, s0)), sv[nt][1] = ptx::ex2(fmaf(sv[nt][1], sc, s0));
        sv[nt][2] = ptx::ex2(fmaf(sv[nt][2], sc, s1)), sv[nt][3] = ptx::ex2(fmaf(sv[nt][3], sc, s1));
        l0 += sv[nt][0] + sv[nt][1], l1 += sv[nt][2] + sv[nt][3];
      }
      const uint32_t pf[4] = {Half2<T>::pack(sv[0][0], sv[0][1]), Half2<T>::pack(sv[0][2], sv[0][3]),
                              Half2<T>::pack(sv[1][0], sv[1][1]), Half2<T>::pack(sv[1][2], sv[1][3])};
#pragma unroll
      for (int d = 0; d < 8; ++d) {
        uint32_t vf[4];
        ldsm4_t(vs + piece_offset(v_tok, 2 * d + v_piece), vf);
        Half2<T>::mma(o[2 * d], pf, vf[0], vf[1]);
        Half2<T>::mma(o[2 * d + 1], pf, vf[2], vf[3]);
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&sh->empty[s]));
    }
    // every warp has consumed the whole ring (or the launch is void): its memory takes the warps' partials
    asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory");
    if (sh->abort_flag == 0) {
      float* po = reinterpret_cast<float*>(ring_ptr);
      l0 = quad_sum(l0), l1 = quad_sum(l1);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = h ? r1 : r0;
        if (r < a.rows) {
          if ((lane & 3) == 0) sh->warp_ml[warp][r] = make_float2(h ? m1 : m0, h ? l1 : l0);
#pragma unroll
          for (int d = 0; d < 16; ++d) {
            *reinterpret_cast<float2*>(po + (warp * kRows + r) * kHeadDim + d * 8 + (lane & 3) * 2) = make_float2(o[d][2 * h], o[d][2 * h + 1]);
          }
        }
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory");
    if (sh->abort_flag == 0) {
      const float* po = reinterpret_cast<const float*>(ring_ptr);
      for (int i = warp; i < a.rows; i += kWarps) {
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) m = fmaxf(m, sh->warp_ml[w][i].x);
        float l = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          const float c = weight(sh->warp_ml[w][i].x, m, sc);
          const float4 x = *reinterpret_cast<const float4*>(po + (w * kRows + i) * kHeadDim + lane * 4);
          l += sh->warp_ml[w][i].y * c;
          acc.x += x.x * c, acc.y += x.y * c, acc.z += x.z * c, acc.w += x.w * c;
        }
        if (slices == 1) {
          store_row4<T>(a, row, i, lane * 4, acc, l);
          if (a.lse && lane == 0) store_lse(a, row, i, m, l);
        } else {
          *reinterpret_cast<float4*>(&sh->cta_o[i][lane * 4]) = acc;
          if (lane == 0) sh->cta_ml[i] = make_float2(m, l);
        }
      }
    }
  }
  if (bad_index && a.status) atomicOr(a.status, CA_STATUS_BAD_INDEX);
  if (slices > 1) {
    cluster.sync();
    // the cluster's threads share the rows' columns, four at a time
    for (int e = rank * kThreads + tid; e < a.rows * (kHeadDim / 4); e += cs * kThreads) {
      const int i = e / (kHeadDim / 4), d = (e % (kHeadDim / 4)) * 4;
      float m = -INFINITY;
      for (int c = 0; c < cs; ++c) m = fmaxf(m, cluster.map_shared_rank(&sh->cta_ml[i], c)->x);
      float l = 0.f;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int c = 0; c < cs; ++c) {
        const float2 ml = *cluster.map_shared_rank(&sh->cta_ml[i], c);
        const float4 x = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&sh->cta_o[i][d], c));
        const float w = weight(ml.x, m, a.scale_log2);
        l += ml.y * w;
        acc.x += x.x * w, acc.y += x.y * w, acc.z += x.z * w, acc.w += x.w * w;
      }
      if (a.parts == 1) {
        store_row4<T>(a, row, i, d, acc, l);
        if (a.lse && d == 0) store_lse(a, row, i, m, l);
      } else {
        const long long p = (static_cast<long long>(row) * a.parts + part) * kRows + i;
        *reinterpret_cast<float4*>(a.part_o + p * kHeadDim + d) = acc;
        if (d == 0) a.part_ml[p] = make_float2(m, l);
      }
    }
    cluster.sync();  // no CTA leaves while its shared memory is read
  }
  __syncthreads();
  if (sh->abort_flag) give_up(a.status, sh, issued);
}

// Merges the partials of rows that were cut over several clusters: one CTA per row, a warp per query row.
template <typename T>
__global__ void __launch_bounds__(128) attn_decode_merge_kernel(const Args a) {
  ptx::grid_launch_dependents();
  ptx::grid_dependency_wait();  // nothing in global memory is touched before this
  const int row = blockIdx.x, lane = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i < a.rows; i += 4) {
    const long long p0 = static_cast<long long>(row) * a.parts * kRows + i;
    float m = -INFINITY;
    for (int p = 0; p < a.parts; ++p) m = fmaxf(m, a.part_ml[p0 + p * kRows].x);
    float l = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int p = 0; p < a.parts; ++p) {
      const float2 ml = a.part_ml[p0 + p * kRows];
      const float4 x = *reinterpret_cast<const float4*>(a.part_o + (p0 + p * kRows) * kHeadDim + lane * 4);
      const float w = weight(ml.x, m, a.scale_log2);
      l += ml.y * w;
      acc.x += x.x * w, acc.y += x.y * w, acc.z += x.z * w, acc.w += x.w * w;
    }
    store_row4<T>(a, row, i, lane * 4, acc, l);
    if (a.lse && lane == 0) store_lse(a, row, i, m, l);
  }
}

template <typename T>
static int launch(const Args& a, const CUtensorMap& k_map, const CUtensorMap& v_map, int R, int cs, int ordinal, cudaStream_t stream) {
  {
    // function attributes are per device: set once per device and type
    static std::mutex mu;
    static bool done[64] = {};
    std::lock_guard<std::mutex> lock(mu);
    if (!done[ordinal]) {
      CA_CUDA(cudaFuncSetAttribute(attn_decode_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
      done[ordinal] = true;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(R) * a.parts * cs), cfg.blockDim = dim3(kThreads), cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cs, attr[1].val.clusterDim.y = 1, attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr, cfg.numAttrs = 2;
  std::unique_lock<std::mutex> pair(pair_mutex(stream), std::defer_lock);
  if (a.parts > 1) pair.lock();
  cudaLaunchKernelEx(&cfg, attn_decode_kernel<T>, k_map, v_map, a);
  CA_LAUNCH_CHECK("attn_decode_kernel");
  if (a.parts > 1) {
    launch_kernel_as(true, attn_decode_merge_kernel<T>, dim3(R), dim3(128), 0, stream, a);
    CA_LAUNCH_CHECK("attn_decode_merge_kernel");
  }
  return CA_OK;
}

}  // namespace decode

// Up to 16 query rows per KV head.  Beyond one mma tile the rows would be read by several tiles and the 256-row
// kernel's tensor-core rate starts to count; at 16 rows (one tile, whatever part of it is live) the bytes decide.
bool decode_applies(const ca_attn_params* p) { return static_cast<long long>(p->Q) * (p->Hq / p->Hkv) <= decode::kRows; }

int launch_decode(const ca_attn_params* p, const DeviceInfo& dev, cudaStream_t stream) {
  using namespace decode;
  CUtensorMap k_map, v_map;
  int slots[3];
  int rc = encode_kv_maps(p, &k_map, &v_map, slots);
  if (rc != CA_OK) return rc;
  Args a;
  a.q = p->q, a.q_stride_b = p->q_stride_b, a.q_stride_t = p->q_stride_t, a.q_stride_h = p->q_stride_h;
  a.out = p->out, a.o_stride_b = p->o_stride_b, a.o_stride_t = p->o_stride_t, a.o_stride_h = p->o_stride_h;
  a.Q = p->Q, a.G = p->Hq / p->Hkv, a.Hkv = p->Hkv, a.rows = a.Q * a.G;
  a.block_size = p->block_size, a.spb = p->block_size / kSub;
  a.q_off = (p->kv_len - p->Q) % p->block_size;
  a.past_tokens = p->kv_len - p->Q - a.q_off;
  a.past_blocks = a.past_tokens / p->block_size;
  a.page_size = p->kv.page_size, a.pages_per_seq = p->kv.pages_per_seq, a.num_pages = p->kv.num_pages;
  a.block_idx = p->block_idx, a.block_idx_stride = p->block_idx_stride, a.counts = p->counts;
  a.page_table = p->kv.page_table;
  a.lse = p->lse, a.scale_log2 = p->softmax_scale * 1.4426950408889634f, a.status = p->status;
  a.wait_limit_ns = 2000000000ull;
  a.slot_tok = slots[0], a.slot_page = slots[1], a.slot_head = slots[2];
  a.kv_head_div = p->kv.head_div > 1 ? p->kv.head_div : 1;

  const int R = p->B * p->Hkv;
  const int blocks = a.block_idx ? (a.block_idx_stride < a.past_blocks ? a.block_idx_stride : a.past_blocks) : a.past_blocks;
  const long long most = static_cast<long long>(blocks) * a.spb + (a.Q - 1 + a.q_off) / kSub + 1;  // sub-blocks of a row
  // Rows too few for the GPU even in clusters of 8 (one KV head of a tensor-parallel rank) are cut over several clusters,
  // which costs the merge launch (131072 tokens of one head: 19 us).
  const int cs = decode_cluster_size(R, most, dev.sm_count);
  a.parts = 1;
  if (cs == kMaxCluster) {
    long long parts = decode_places(cs, dev.sm_count) / (R * cs);
    const long long by_work = most / (cs * kMinSubsPart);
    if (parts > by_work) parts = by_work;
    const size_t per_part = static_cast<size_t>(R) * kRows * (kHeadDim * sizeof(float) + sizeof(float2));
    if (p->workspace != nullptr && parts > 1 && parts * per_part <= p->workspace_bytes) a.parts = static_cast<int>(parts);
  }
  a.part_o = static_cast<float*>(p->workspace);
  a.part_ml = a.parts > 1 ? reinterpret_cast<float2*>(a.part_o + static_cast<size_t>(R) * a.parts * kRows * kHeadDim) : nullptr;
  return p->dtype == CA_DTYPE_BF16 ? launch<__nv_bfloat16>(a, k_map, v_map, R, cs, dev.ordinal, stream)
                                   : launch<__half>(a, k_map, v_map, R, cs, dev.ordinal, stream);
}

}  // namespace attn
}  // namespace ca
