// FlashAttention forward for sm_100a (tcgen05 + TMEM + TMA).
//
// One CTA owns 256 query rows of one (batch, head) as two tiles of 128.  K/V tiles of 128 rows stream through a
// 2-stage TMA ring and serve both.  S = Q K^T and O += P V run on tcgen05; S0, S1, O0 and O1 fill TMEM.
//
// A softmax warpgroup per query tile: a thread owns one whole query row (TMEM lane == row, all 128 key columns in
// registers), so the row maximum and sum never leave the thread.  P goes back, in 16 bits, over the columns of its S, from
// where the second product reads it as its left operand: nothing but Q, K and V passes through shared memory, whose port
// (128 bytes a clock) could not carry P's way out and in beside the operands.  While one warpgroup computes its softmax, the
// tensor core works on the other's tile: P V and then the next Q K^T, in that order, so S's columns are free by the time they
// are written.  O is rescaled in place by the softmax warps, only when the maximum moved by more than 2^8 (the S that
// a warpgroup waits for is committed after its last P V, so O is at rest then).  exp is exp2 with the softmax scale folded in.
// LSE is saved for the backward pass.
//
// Bound by the exponentials (16 a clock and SM: 1024 clocks for a tile of S, as long as its two products) and by what is left of each softmax's latency.
// Causal, 8 x 2048 rows, 16 heads of 128: 186 us (741 TFLOP/s of the masked half's work); 305 us with 128 query rows a CTA, two warpgroups on alternate key tiles
// and P through shared memory.  Not causal, 2 x 4096: 1043 TFLOP/s.
//
// Layout: q/k/v/o are [B, S, H, D] views with arbitrary batch/seq/head strides
// (so the fused qkv projection output is consumed in place); D in {64, 128}.
//
// The reference kernel (rumus/src/backend/gpu/shaders/flash_attn.wgsl:35) is a
// forward-only scalar loop: one thread per query row, K/V tiles of <= 16 rows in
// 16 KB of workgroup memory (rumus/src/backend/gpu/compute.rs:2079-2138).
#include "sm100_common.cuh"

namespace rb {

struct FaFwdParams {
  int B, H, Hkv, Sq, Sk;
  int causal;
  float scale_log2;  // softmax scale * log2(e)
  void* o;           // [B, Sq, H, D] contiguous
  float* lse;        // [B, H, Sq]
  int* status;
};

template <int HD>
struct FaFwdCfg {
  static constexpr int BM = 256, BN = 128;        // two query tiles of 128 rows
  static constexpr int SUB = HD / 64;             // 64-column sub-tiles per row
  static constexpr int TILE_BYTES = 128 * 128;    // one [128 x 64] 16-bit sub-tile
  static constexpr int Q_BYTES = SUB * TILE_BYTES;   // one query tile
  static constexpr int KV_BYTES = SUB * TILE_BYTES;  // per K or V tile
  static constexpr int STAGES = 2;
  static constexpr int SMEM_BYTES = 2 * Q_BYTES + STAGES * 2 * KV_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = 512;
  static constexpr int S_COL = 0;        // S of the two tiles at columns [0,128) and [128,256), P over the first half of each
  static constexpr int O_COL = 256;      // O at [256, 256+HD) and [384, 384+HD)
};

// two fp32 operations in one instruction
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f32x2_get(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

template <typename T, int HD>
__global__ void __launch_bounds__(320, 1)
    fa_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                  const __grid_constant__ CUtensorMap tv, const FaFwdParams p) {
  using C = FaFwdCfg<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;                                  // [2][Q_BYTES]
  uint8_t* sK = sQ + 2 * C::Q_BYTES;                   // [STAGES][KV_BYTES]
  uint8_t* sV = sK + C::STAGES * C::KV_BYTES;          // [STAGES][KV_BYTES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + C::STAGES * C::KV_BYTES);
  uint64_t* q_full = bars;         // [2]
  uint64_t* k_full = bars + 2;     // [2] K tile landed
  uint64_t* k_empty = bars + 4;    // [2] K slot free again (both S products that read it retired)
  uint64_t* v_full = bars + 6;     // [2]
  uint64_t* v_empty = bars + 8;    // [2]
  uint64_t* s_full = bars + 10;    // [2] per query tile: S written, and the P V before it retired
  uint64_t* p_ready = bars + 12;   // [2] per query tile
  uint64_t* o_full = bars + 14;    // [2] per query tile: last P V retired
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp_idx = uniform_warp_idx();
  const int lane = threadIdx.x & 31;
  const int q_tile = gridDim.x - 1 - blockIdx.x;  // heavy (late) causal tiles first
  const int h_idx = blockIdx.y, b = blockIdx.z;
  const int hkv = h_idx / (p.H / p.Hkv);
  const int q0 = q_tile * C::BM;
  const int off = p.Sk - p.Sq;
  // K/V tiles that query tile i looks at
  auto tiles_of = [&](int i) {
    const int r0 = q0 + i * 128;
    if (r0 >= p.Sq) return 0;
    if (!p.causal) return (p.Sk + C::BN - 1) / C::BN;
    const int last_kv = min(p.Sk - 1, r0 + 127 + off);
    return last_kv < 0 ? 0 : last_kv / C::BN + 1;
  };
  const int n_of[2] = {tiles_of(0), tiles_of(1)};
  const int n_tiles = max(n_of[0], n_of[1]);

  if (threadIdx.x == 0) {
    prefetch_tensormap(&tq);
    prefetch_tensormap(&tk);
    prefetch_tensormap(&tv);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&q_full[s]), 1);
      mbar_init(smem_u32(&k_full[s]), 1);
      mbar_init(smem_u32(&k_empty[s]), 1);
      mbar_init(smem_u32(&v_full[s]), 1);
      mbar_init(smem_u32(&v_empty[s]), 1);
      mbar_init(smem_u32(&s_full[s]), 1);
      mbar_init(smem_u32(&p_ready[s]), 128);     // the 128 threads of the warpgroup that owns the tile
      mbar_init(smem_u32(&o_full[s]), 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp_idx == 9) {
    tmem_alloc(smem_u32(tmem_ptr_smem), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp_idx == 8) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0 && n_tiles > 0) {
      auto load_q = [&](int i) {
        if (n_of[i] == 0) return;
        mbar_arrive_expect_tx(smem_u32(&q_full[i]), C::Q_BYTES);
#pragma unroll
        for (int s = 0; s < C::SUB; ++s)
          tma_load_4d(smem_u32(sQ + i * C::Q_BYTES + s * C::TILE_BYTES), &tq, smem_u32(&q_full[i]), s * 64, q0 + i * 128, h_idx, b);
      };
      auto load = [&](uint8_t* dst, const CUtensorMap* m, uint32_t bar, int j) {
        mbar_arrive_expect_tx(bar, C::KV_BYTES);
#pragma unroll
        for (int s = 0; s < C::SUB; ++s) tma_load_4d(smem_u32(dst + s * C::TILE_BYTES), m, bar, s * 64, j * C::BN, hkv, b);
      };
      load_q(0);
      bool ok = true;
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        ok = mbar_wait(smem_u32(&k_empty[st]), ph ^ 1, abort_flag, p.status, RB_ERR_TIMEOUT_EMPTY);
        if (!ok) break;
        load(sK + st * C::KV_BYTES, &tk, smem_u32(&k_full[st]), j);
        if (j == 0) load_q(1);
        ok = mbar_wait(smem_u32(&v_empty[st]), ph ^ 1, abort_flag, p.status, RB_ERR_TIMEOUT_EMPTY);
        if (!ok) break;
        load(sV + st * C::KV_BYTES, &tv, smem_u32(&v_full[st]), j);
      }
      if (!ok)
        for (int i = 0; i < 64; ++i) __nanosleep(10000);
    }
  } else if (warp_idx == 9) {
    // ------------------------------ MMA issuer --------------------------------
    if (n_tiles > 0) {   // whole warp; one elected lane issues each instruction
      constexpr uint32_t idesc_s = make_idesc(UmmaFormat<T>::value, 0, 0, 128, 128);
      constexpr uint32_t idesc_o = make_idesc(UmmaFormat<T>::value, 0, 1, 128, HD);
      auto issue_s = [&](int i, int j) {
        const uint64_t qd = make_smem_desc_sw128(smem_u32(sQ + i * C::Q_BYTES), 16, 1024);
        const uint64_t kd = make_smem_desc_sw128(smem_u32(sK + (j & 1) * C::KV_BYTES), 16, 1024);
#pragma unroll
        for (int s = 0; s < C::SUB; ++s)
          umma_f16_w4<2, 2>(tmem_base + C::S_COL + i * 128, qd + s * (C::TILE_BYTES >> 4), kd + s * (C::TILE_BYTES >> 4), idesc_s, s != 0);
        umma_commit_w(smem_u32(&s_full[i]));
      };
      auto issue_pv = [&](int i, int j) {
        const uint64_t vd = make_smem_desc_sw128(smem_u32(sV + (j & 1) * C::KV_BYTES), C::TILE_BYTES, 1024);
#pragma unroll
        for (int s = 0; s < 2; ++s)
          umma_f16_ts_w4<8, 128>(tmem_base + C::O_COL + i * 128, tmem_base + C::S_COL + i * 128 + s * 32, vd + s * 512, idesc_o,
                                 (j | s) != 0);
      };
      bool ok = mbar_wait(smem_u32(&k_full[0]), 0, abort_flag, p.status, RB_ERR_TIMEOUT_FULL);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (ok && n_of[i] > 0) {
          ok = mbar_wait(smem_u32(&q_full[i]), 0, abort_flag, p.status, RB_ERR_TIMEOUT_FULL);
          if (ok) {
            tc_fence_after();
            issue_s(i, 0);
          }
        }
      if (ok) umma_commit_w(smem_u32(&k_empty[0]));
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        const bool more = j + 1 < n_tiles;
        if (more) ok = mbar_wait(smem_u32(&k_full[st ^ 1]), ((j + 1) >> 1) & 1, abort_flag, p.status, RB_ERR_TIMEOUT_FULL);
        if (ok) ok = mbar_wait(smem_u32(&v_full[st]), ph, abort_flag, p.status, RB_ERR_TIMEOUT_FULL);
        if (!ok) break;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (j >= n_of[i]) continue;
          ok = mbar_wait(smem_u32(&p_ready[i]), j & 1, abort_flag, p.status, RB_ERR_TIMEOUT_FLAG);
          if (!ok) break;
          tc_fence_after();
          issue_pv(i, j);
          if (j + 1 < n_of[i]) issue_s(i, j + 1);
          else umma_commit_w(smem_u32(&o_full[i]));
        }
        if (!ok) break;
        umma_commit_w(smem_u32(&v_empty[st]));
        if (more) umma_commit_w(smem_u32(&k_empty[st ^ 1]));
      }
    }
  } else {
    // ------------------------------ softmax warps -----------------------------
    const int wg = warp_idx >> 2;                 // query tile
    const int t = (warp_idx & 3) * 32 + lane;     // row within the tile == TMEM lane
    const int row = q0 + wg * 128 + t;            // global query row
    const int n_mine = wg ? n_of[1] : n_of[0];
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp_idx & 3) * 32) << 16);
    const uint32_t s_addr = lane_addr + C::S_COL + wg * 128;
    const uint32_t o_addr = lane_addr + C::O_COL + wg * 128;
    const int kv_limit = p.causal ? min(p.Sk - 1, row + off) : p.Sk - 1;  // last valid kv index
    const int row_lo = q0 + wg * 128 + off;                               // the first row's own position
    float m_used = -INFINITY, l = 0.f;            // running maximum (log2 domain) and sum
    bool ok = true;
    for (int j = 0; j < n_mine; ++j) {
      ok = mbar_wait(smem_u32(&s_full[wg]), j & 1, abort_flag, p.status, RB_ERR_TIMEOUT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t s[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(s_addr + c * 32, s[c]);
      tmem_ld_wait();
      const int kv0 = j * C::BN;
      if ((kv0 + C::BN > p.Sk) || (p.causal && kv0 + C::BN - 1 > row_lo)) {
        const int last = kv_limit - kv0;          // last column that counts
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i > last) s[c][i] = 0xff800000u;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          mx4[(i >> 1) & 3] = fmaxf(fmaxf(mx4[(i >> 1) & 3], __uint_as_float(s[c][i])), __uint_as_float(s[c][i + 1]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const float m_new = fmaxf(m_used, mx * p.scale_log2);
      const bool need = m_new > m_used + 8.0f;  // also true on the first tile (m_used = -inf)
      if (__any_sync(0xffffffffu, need)) {       // the TMEM accesses below are warp-wide: uniform branch
        float alpha = 1.0f;
        if (need) {
          alpha = (m_used == -INFINITY) ? 0.0f : fast_exp2(m_used - m_new);
          m_used = m_new;
          l *= alpha;
        }
        if (j > 0) {
#pragma unroll 1
          for (int c = 0; c < HD / 16; ++c) {
            uint32_t r[16];
            tmem_ld_32x32b_x16(o_addr + c * 16, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st_32x32b_x16(o_addr + c * 16, r);
          }
        }
      }
      // P = exp2(S*scale - m) and the row sum; P over the first 64 columns of S
      const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
      const uint64_t scale2 = f32x2(p.scale_log2, p.scale_log2), neg2 = f32x2(neg_m, neg_m);
      uint64_t sum2[2] = {0, 0};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 x = f32x2_get(fma_f32x2(f32x2(__uint_as_float(s[c][2 * i]), __uint_as_float(s[c][2 * i + 1])), scale2, neg2));
          const float p0 = fast_exp2(x.x), p1 = fast_exp2(x.y);
          sum2[i & 1] = add_f32x2(sum2[i & 1], f32x2(p0, p1));
          packed[i] = pack2<T>(p0, p1);
        }
        tmem_st_32x32b_x16(s_addr + c * 16, packed);
      }
      const float2 sum = f32x2_get(add_f32x2(sum2[0], sum2[1]));
      l += sum.x + sum.y;
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(smem_u32(&p_ready[wg]));
    }
    if (ok && n_mine > 0) {
      ok = mbar_wait(smem_u32(&o_full[wg]), 0, abort_flag, p.status, RB_ERR_TIMEOUT_TMEM_EMPTY);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after();
      const float inv_l = l > 0.f ? 1.0f / l : 0.f;
      T* orow = reinterpret_cast<T*>(p.o) + ((static_cast<long long>(b) * p.Sq + row) * p.H + h_idx) * HD;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t r[32];
        if (n_mine > 0) {
          tmem_ld_32x32b_x32(o_addr + c * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0;
        }
        if (row < p.Sq) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              w[i] = pack2<T>(__uint_as_float(r[q * 8 + 2 * i]) * inv_l, __uint_as_float(r[q * 8 + 2 * i + 1]) * inv_l);
            *reinterpret_cast<uint4*>(orow + c * 32 + q * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      if (row < p.Sq)
        p.lse[(static_cast<long long>(b) * p.H + h_idx) * p.Sq + row] = (m_used + log2f(l)) * 0.6931471805599453f;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp_idx == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

template <typename T, int HD>
int launch_fa_fwd(int dtype, const void* q, const void* k, const void* v, const long long* qs,
                  const long long* ks, const long long* vs, const FaFwdParams& p, cudaStream_t st) {
  using C = FaFwdCfg<HD>;
  CUtensorMap tq, tk, tv;
  auto mk = [&](CUtensorMap* m, const void* base, const long long* s, int S, int heads) {
    uint64_t dims[4] = {(uint64_t)HD, (uint64_t)S, (uint64_t)heads, (uint64_t)p.B};
    uint64_t strides[4] = {2, (uint64_t)s[1] * 2, (uint64_t)s[2] * 2, (uint64_t)s[0] * 2};
    uint32_t box[4] = {64, 128, 1, 1};
    return rbh::encode_tensor_map(m, dtype, 4, const_cast<void*>(base), dims, strides, box, 1);
  };
  int rc = mk(&tq, q, qs, p.Sq, p.H);
  if (!rc) rc = mk(&tk, k, ks, p.Sk, p.Hkv);
  if (!rc) rc = mk(&tv, v, vs, p.Sk, p.Hkv);
  if (rc) return 1000 + rc;
  auto kern = fa_fwd_kernel<T, HD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
  if (e != cudaSuccess) return 2000 + (int)e;
  dim3 grid((p.Sq + C::BM - 1) / C::BM, p.H, p.B);
  kern<<<grid, 320, C::SMEM_BYTES, st>>>(tq, tk, tv, p);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 3000 + (int)e;
}

}  // namespace rb

extern "C" {
// q/k/v strides are {batch, seq, head} in elements (innermost dim contiguous).
// o is [B,Sq,H,D] contiguous, lse is [B,H,Sq] fp32.
int rb_flash_attn_fwd(int dtype, int head_dim, const void* q, const void* k, const void* v,
                      const long long* q_strides, const long long* k_strides,
                      const long long* v_strides, void* o, float* lse, int B, int H, int Hkv,
                      int Sq, int Sk, int causal, float scale, void* stream) {
  using namespace rb;
  if (B <= 0 || H <= 0 || Sq <= 0) return 0;
  FaFwdParams p;
  p.B = B; p.H = H; p.Hkv = Hkv; p.Sq = Sq; p.Sk = Sk; p.causal = causal;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.o = o; p.lse = lse;
  p.status = rbh::device_status_word();
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == rbh::DT_BF16) {
    if (head_dim == 128) return launch_fa_fwd<__nv_bfloat16, 128>(dtype, q, k, v, q_strides, k_strides, v_strides, p, st);
    if (head_dim == 64) return launch_fa_fwd<__nv_bfloat16, 64>(dtype, q, k, v, q_strides, k_strides, v_strides, p, st);
  } else if (dtype == rbh::DT_F16) {
    if (head_dim == 128) return launch_fa_fwd<__half, 128>(dtype, q, k, v, q_strides, k_strides, v_strides, p, st);
    if (head_dim == 64) return launch_fa_fwd<__half, 64>(dtype, q, k, v, q_strides, k_strides, v_strides, p, st);
  }
  return 20;  // unsupported dtype / head_dim
}
}
