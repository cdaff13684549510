// Harness for the per-tile dependency chain of an earlier form of the attention kernel, whose P lay over its S: S = Q.K^T (8 MMAs) -> softmax -> P -> O += P.V (8 MMAs)
// -> next S ...  One tile, so the period is exactly 1024 cycles of MMA work + hand-off latencies + softmax time.
// Timing only (operands are zeros).  argv: variant iters
//   0: softmax as in that kernel (one thread per row, 128 columns, P in two pieces)
//   1: S loaded in chunks, row max of a chunk computed while the next chunks are in flight
//   2: two warpgroups per tile, each thread owns 64 columns of a row (row max exchanged through shared memory)
//   3: variant 2 + polynomial exp2 for POLY of every 16 pairs (env POLY)
//   4: variant 0 + polynomial exp2 for POLY of every 16 pairs
#include "../csrc/ca_common.cuh"
#include <cstdio>
#include <cstdlib>
using namespace ca;
__device__ long long g_cycles[160];
__device__ int g_status;
struct P { int variant; int iters; int poly; };

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 ex2_poly2(float2 x) {
  x.x = fmaxf(x.x, -126.0f); x.y = fmaxf(x.y, -126.0f);
  const float2 magic = make_float2(12582912.0f, 12582912.0f);
  const float2 t = __fadd2_rn(x, magic);
  const float2 u = __fadd2_rn(t, make_float2(-12582912.0f, -12582912.0f));
  const float2 f = __ffma2_rn(u, make_float2(-1.0f, -1.0f), x);
  float2 p = __ffma2_rn(make_float2(0.0558755025267601f, 0.0558755025267601f), f, make_float2(0.24229444563388824f, 0.24229444563388824f));
  p = __ffma2_rn(p, f, make_float2(0.6931272745132446f, 0.6931272745132446f));
  p = __ffma2_rn(p, f, make_float2(0.999948263168335f, 0.999948263168335f));
  p.x = __uint_as_float(__float_as_uint(p.x) + (__float_as_uint(t.x) << 23));
  p.y = __uint_as_float(__float_as_uint(p.y) + (__float_as_uint(t.y) << 23));
  return p;
}

template <int POLY>
__device__ __forceinline__ float exp_chunk(const uint32_t* sv, float sc, float neg_m, uint32_t taddr) {
  // 32 columns -> 16 packed words -> one tcgen05.st.x16
  float2 l2 = make_float2(0.f, 0.f);
  const float2 sc2 = make_float2(sc, sc), nm2 = make_float2(neg_m, neg_m);
  uint32_t pk[16];
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sc2, nm2);
    float2 pr;
    const int pi = i >> 1;
    const bool poly = POLY > 0 && ((pi * POLY) / 16 != ((pi + 1) * POLY) / 16);
    if (poly) pr = ex2_poly2(x);
    else { pr.x = ptx::ex2(x.x); pr.y = ptx::ex2(x.y); }
    l2 = __fadd2_rn(l2, pr);
    pk[pi] = pack_bf16(pr.x, pr.y);
  }
  ptx::tmem_st16(taddr, pk);
  return l2.x + l2.y;
}

template <int POLY>
__device__ __forceinline__ float exp_chunk_dispatch(int poly, const uint32_t* sv, float sc, float neg_m, uint32_t taddr) {
  return exp_chunk<POLY>(sv, sc, neg_m, taddr);
}

#define EXP_CHUNK(sv, taddr) (p.poly == 0 ? exp_chunk<0>(sv, sc, neg_m, taddr) : p.poly == 2 ? exp_chunk<2>(sv, sc, neg_m, taddr) : \
                              p.poly == 4 ? exp_chunk<4>(sv, sc, neg_m, taddr) : p.poly == 6 ? exp_chunk<6>(sv, sc, neg_m, taddr) : exp_chunk<8>(sv, sc, neg_m, taddr))

__global__ void __launch_bounds__(384, 1) chain_kernel(P p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ uint64_t s_full, p_part[2];
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  __shared__ float mx_sh[2][128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const bool two_wg = p.variant == 2 || p.variant == 3;
  if (tid == 0) {
    abort_flag = 0;
    ptx::mbar_init(ptx::smem_u32(&s_full), 1);
    ptx::mbar_init(ptx::smem_u32(&p_part[0]), 128);
    ptx::mbar_init(ptx::smem_u32(&p_part[1]), 128);
    ptx::mbar_fence_init();
    ptx::fence_proxy_async_smem();
  }
  for (int i = tid; i < 96 * 1024 / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(smem_raw + (base - ptx::smem_u32(smem_raw)))[i] = make_uint4(0, 0, 0, 0);
  ptx::fence_proxy_async_smem();
  if (warp == 8) { ptx::tmem_alloc(ptx::smem_u32(&tmem_base), 512); ptx::tmem_relinquish(); }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = tmem_base;
  volatile int* af = &abort_flag;
  const uint64_t lim = 1000000000ull;
  if (warp < 8) {
    const int wg = warp >> 2;
    if (wg == 1 && !two_wg) {
      // idle
    } else {
      const int r = tid & 127;
      const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
      const uint32_t tS = tmem + lane_base;
      const float sc = 0.125f * 1.4426950408889634f;
      float m_run = -INFINITY, l_run = 0.f;
      for (int it = 0; it < p.iters; ++it) {
        bool ok = ptx::mbar_wait_bounded(ptx::smem_u32(&s_full), it & 1, af, lim);
        if (!__all_sync(0xffffffffu, ok)) break;
        ptx::tc_fence_after();
        if (!two_wg) {
          uint32_t sv[128];
          float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
          if (p.variant == 1) {
            ptx::tmem_ld32_row<0>(tS + 0, sv);
            ptx::tc_wait_ld();
            ptx::tmem_ld32_row<32>(tS + 32, sv);
            ptx::tmem_ld32_row<64>(tS + 64, sv);
            ptx::tmem_ld32_row<96>(tS + 96, sv);
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              mx0 = fmaxf(mx0, __uint_as_float(sv[i])); mx1 = fmaxf(mx1, __uint_as_float(sv[i + 1]));
              mx2 = fmaxf(mx2, __uint_as_float(sv[i + 2])); mx3 = fmaxf(mx3, __uint_as_float(sv[i + 3]));
            }
            ptx::tc_wait_ld();
#pragma unroll
            for (int i = 32; i < 128; i += 4) {
              mx0 = fmaxf(mx0, __uint_as_float(sv[i])); mx1 = fmaxf(mx1, __uint_as_float(sv[i + 1]));
              mx2 = fmaxf(mx2, __uint_as_float(sv[i + 2])); mx3 = fmaxf(mx3, __uint_as_float(sv[i + 3]));
            }
          } else {
            ptx::tmem_ld32_row<0>(tS + 0, sv);
            ptx::tmem_ld32_row<32>(tS + 32, sv);
            ptx::tmem_ld32_row<64>(tS + 64, sv);
            ptx::tmem_ld32_row<96>(tS + 96, sv);
            ptx::tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 128; i += 4) {
              mx0 = fmaxf(mx0, __uint_as_float(sv[i])); mx1 = fmaxf(mx1, __uint_as_float(sv[i + 1]));
              mx2 = fmaxf(mx2, __uint_as_float(sv[i + 2])); mx3 = fmaxf(mx3, __uint_as_float(sv[i + 3]));
            }
          }
          const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
          const float m_new = fmaxf(m_run, mx);
          const bool need = m_new > m_run && (m_run == -INFINITY || (m_new - m_run) * sc > 8.0f);
          if (__any_sync(0xffffffffu, need)) { if (need) { l_run *= 0.5f; m_run = m_new; } }
          const float neg_m = m_run == -INFINITY ? 0.f : -m_run * sc;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            l_run += EXP_CHUNK(&sv[c * 32], tS + c * 16);
            if (c & 1) {
              ptx::tc_wait_st();
              ptx::tc_fence_before();
              ptx::mbar_arrive(ptx::smem_u32(&p_part[c >> 1]));
            }
          }
        } else {
          // this thread owns columns [64*wg, 64*wg + 64) of row r
          uint32_t sv[64];
          uint32_t lo[32], hi[32];
          ptx::tmem_ld32(tS + wg * 64, lo);
          ptx::tmem_ld32(tS + wg * 64 + 32, hi);
          ptx::tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) sv[i] = lo[i], sv[32 + i] = hi[i];
          float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            mx0 = fmaxf(mx0, __uint_as_float(sv[i])); mx1 = fmaxf(mx1, __uint_as_float(sv[i + 1]));
            mx2 = fmaxf(mx2, __uint_as_float(sv[i + 2])); mx3 = fmaxf(mx3, __uint_as_float(sv[i + 3]));
          }
          float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
          mx_sh[wg][r] = mx;
          asm volatile("bar.sync 1, 256;" ::: "memory");
          mx = fmaxf(mx, mx_sh[wg ^ 1][r]);
          const float m_new = fmaxf(m_run, mx);
          const bool need = m_new > m_run && (m_run == -INFINITY || (m_new - m_run) * sc > 8.0f);
          if (__any_sync(0xffffffffu, need)) { if (need) { l_run *= 0.5f; m_run = m_new; } }
          const float neg_m = m_run == -INFINITY ? 0.f : -m_run * sc;
          l_run += EXP_CHUNK(&sv[0], tS + wg * 32);
          l_run += EXP_CHUNK(&sv[32], tS + wg * 32 + 16);
          ptx::tc_wait_st();
          ptx::tc_fence_before();
          ptx::mbar_arrive(ptx::smem_u32(&p_part[wg]));
          asm volatile("bar.sync 2, 256;" ::: "memory");  // mx_sh may be rewritten only after both halves have read it
        }
      }
      if (l_run == 123.456f) g_status = 3;
    }
  } else if (warp == 8 && lane == 0) {
    const uint32_t idesc_ss = ptx::make_idesc_f16(1, 128, 128, 0, 0);
    const uint32_t idesc_pv = ptx::make_idesc_f16(1, 128, 128, 0, 1);
    const uint64_t a0 = ptx::make_smem_desc_sw128(base, 0, 1024);
    const uint64_t b0 = ptx::make_smem_desc_sw128(base + 32768, 0, 1024);
    const uint64_t v0 = ptx::make_smem_desc_sw128(base + 65536, 16384, 1024);
    bool ok = true;
    long long t0 = clock64();
    for (int it = 0; it < p.iters && ok; ++it) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint64_t o = static_cast<uint64_t>(((k >> 2) * 16384 + (k & 3) * 32) >> 4);
        ptx::mma_ss(tmem, a0 + o, b0 + o, idesc_ss, k > 0 ? 1u : 0u);
      }
      ptx::tc_commit(ptx::smem_u32(&s_full));
      for (int q = 0; q < 2 && ok; ++q) {
        ok = ptx::mbar_wait_bounded(ptx::smem_u32(&p_part[q]), it & 1, af, lim);
        ptx::tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ptx::mma_ts(tmem + 256u, tmem + (q * 4 + k) * 8, v0 + static_cast<uint64_t>((q * 4 + k) * (2048 >> 4)), idesc_pv, 1u);
      }
    }
    long long t1 = clock64();
    g_cycles[blockIdx.x] = t1 - t0;
    if (!ok) atomicOr(&g_status, 1);
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 8) { ptx::tc_fence_after(); ptx::tmem_dealloc(tmem, 512); }
}

int main(int argc, char** argv) {
  P p; p.variant = argc > 1 ? atoi(argv[1]) : 0; p.iters = argc > 2 ? atoi(argv[2]) : 2000;
  p.poly = getenv("POLY") ? atoi(getenv("POLY")) : 0;
  const int smem = 98 * 1024;
  cudaFuncSetAttribute(chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  for (int rep = 0; rep < 2; ++rep) {
    chain_kernel<<<148, 384, smem>>>(p);
    cudaError_t err = cudaDeviceSynchronize();
    if (err != cudaSuccess) { printf("error %s\n", cudaGetErrorString(err)); return 1; }
    long long cyc[160]; int st;
    cudaMemcpyFromSymbol(cyc, g_cycles, sizeof(cyc)); cudaMemcpyFromSymbol(&st, g_status, sizeof(int));
    printf("variant %d poly %d: %.0f cycles per step (1024 of MMA work + %.0f of hand-off and softmax), status %d\n", p.variant, p.poly,
           (double)cyc[0] / p.iters, (double)cyc[0] / p.iters - 1024.0, st);
  }
  return 0;
}
