// Serving kernels for sm_100a: paged-KV decode attention (split-KV, block-table gather),
// KV-cache append, greedy sampling (row argmax).
//
// The reference server keeps a dense zero-filled cache and a mock model
// (rumus-serve/src/model.rs:14-142) and scans the vocabulary on the CPU for the argmax
// (rumus-serve/src/scheduler.rs:101-135); none of these kernels has a counterpart there.
//
// Cache layout: k_cache / v_cache [num_blocks, block_size, Hkv, D] (token-major) or, with `head_major` and in
// rb_kv_append_hm, [num_blocks, Hkv, block_size, D] (head-major); a sequence's logical token t lives in
// physical block block_table[b][t / block_size] at offset t % block_size.
#include "warp_mma.cuh"

namespace rb {

constexpr int kPaWarps = 4;
constexpr int kPaStages = 3;       // pairs of tokens of every 8-lane group in shared memory or on their way

// grid (H, B, splits), 128 threads.  D = 128: eight lanes share one token (16 dims = two 16-byte
// loads of K and of V per lane), so a warp works on four tokens at once and every 8-lane group
// carries its own online-softmax state.  Bound by the cache's way from HBM: a lane copies its pieces
// of the next pairs of tokens (cp.async) into a ring that only the lane itself reads, so up to two pairs
// of every group are in flight while one is computed, without registers for them or barriers.  (Plain loads,
// used in the trip that asked for them: 225 us for 48 sequences of 1100 tokens, 32 heads, 865 MB.)
// partial_o [B,H,splits,D] fp32, partial_ml [B,H,splits,2] (running max in log2 domain, sum); with one split
// the result is written at once.
// A lane's sixteen numbers of a row are its pieces sub and sub + 8 of sixteen: eight lanes copy 128 bytes side by side (with pieces 2 sub and
// 2 sub + 1 each copy asked for half of every 32-byte sector, and each sector came twice: 240 us instead).
template <typename T>
__device__ __forceinline__ void pa_load16(const T* p, float* f) {
  const uint4 a = *reinterpret_cast<const uint4*>(p);
  const uint4 b = *reinterpret_cast<const uint4*>(p + 64);
  const T* ea = reinterpret_cast<const T*>(&a);
  const T* eb = reinterpret_cast<const T*>(&b);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    f[j] = to_f32<T>(ea[j]);
    f[8 + j] = to_f32<T>(eb[j]);
  }
}
// the sixteen numbers of a lane's two pieces in the ring, 512 bytes (one warp) apart
template <typename T>
__device__ __forceinline__ void pa_ring16(const uint8_t* p, float* f) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 a = *reinterpret_cast<const uint4*>(p + h * 512);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 v = unpack2<T>(w[j]);
      f[h * 8 + 2 * j] = v.x;
      f[h * 8 + 2 * j + 1] = v.y;
    }
  }
}

// HM = head-major cache [num_blocks, Hkv, block_size, D]: one head's tokens of a block are
// contiguous (block_size * 256 B), so the four tokens a warp reads per trip are one 1 KiB run
// instead of four 256-byte pieces a whole token row (Hkv * 256 B) apart.  block_shift: log2 of the block
// size, or -1 when it is no power of two.
template <typename T, bool HM = false>
__global__ void __launch_bounds__(kPaWarps * 32)
    paged_decode_attn_kernel(const T* __restrict__ q, long long ldq, const T* __restrict__ k_cache,
                             const T* __restrict__ v_cache, const int* __restrict__ block_tables,
                             const int* __restrict__ ctx_lens, float* __restrict__ partial_o,
                             float* __restrict__ partial_ml, T* __restrict__ out, int H, int Hkv, int block_size,
                             int block_shift, int max_blocks, int splits, float scale_log2) {
  constexpr int D = 128;
  constexpr int G = kPaWarps * 4;   // token groups per CTA
  constexpr int STAGE = 8 * 512;    // of a warp: two tokens of a group, K and V, two pieces each
  __shared__ __align__(16) uint8_t ring_all[kPaWarps * kPaStages * STAGE];
  const int h = blockIdx.x, b = blockIdx.y, sp = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = lane >> 3, sub = lane & 7;
  const int gid = warp * 4 + grp;
  const int hkv = h / (H / Hkv);
  const int ctx = ctx_lens[b];
  const int per = (ctx + splits - 1) / splits;
  const int t0 = sp * per, t1 = min(ctx, t0 + per);
  const int* table = block_tables + (long long)b * max_blocks;
  uint8_t* ring = ring_all + warp * kPaStages * STAGE + lane * 16;
  auto fetch = [&](int i) {
    const uint32_t dst = smem_u32(ring + (i % kPaStages) * STAGE);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = t0 + (2 * i + u) * G + gid;
      if (t < t1) {
        const int bi = block_shift >= 0 ? t >> block_shift : t / block_size;
        const int off = t - bi * block_size;
        const long long blk = table[bi];
        long long at;
        if constexpr (HM) at = ((blk * Hkv + hkv) * block_size + off) * D + sub * 8;
        else at = ((blk * block_size + off) * Hkv + hkv) * D + sub * 8;
        copy16(dst + (u * 4) * 512, k_cache + at, true);
        copy16(dst + (u * 4 + 1) * 512, k_cache + at + 64, true);
        copy16(dst + (u * 4 + 2) * 512, v_cache + at, true);
        copy16(dst + (u * 4 + 3) * 512, v_cache + at + 64, true);
      }
    }
    copy_commit();
  };
  const int trips = t1 > t0 ? (t1 - t0 + 2 * G - 1) / (2 * G) : 0;
#pragma unroll
  for (int i = 0; i < kPaStages - 1; ++i) fetch(i);
  float qv[16];
  pa_load16<T>(q + (long long)b * ldq + h * D + sub * 8, qv);
#pragma unroll
  for (int j = 0; j < 16; ++j) qv[j] *= scale_log2;
  float m = -INFINITY, l = 0.f, acc[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) acc[j] = 0.f;
  // every lane runs every trip (the shuffles are warp wide); out-of-range tokens are skipped
  for (int i = 0; i < trips; ++i) {
    copy_wait<kPaStages - 2>();
    fetch(i + kPaStages - 1);
    const uint8_t* st = ring + (i % kPaStages) * STAGE;
    const int ta = t0 + 2 * i * G + gid, tc = ta + G;
    const bool va = ta < t1, vc = tc < t1;
    float x[16];
    float sa = 0.f, sc = 0.f;
    if (va) {
      pa_ring16<T>(st, x);
#pragma unroll
      for (int j = 0; j < 16; ++j) sa = fmaf(qv[j], x[j], sa);
    }
    if (vc) {
      pa_ring16<T>(st + 4 * 512, x);
#pragma unroll
      for (int j = 0; j < 16; ++j) sc = fmaf(qv[j], x[j], sc);
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      sa += __shfl_xor_sync(0xffffffffu, sa, o);
      sc += __shfl_xor_sync(0xffffffffu, sc, o);
    }
    if (va) {
      const float mn = fmaxf(m, vc ? fmaxf(sa, sc) : sa);
      const float corr = fast_exp2(m - mn);   // m = -inf on the first token: exp2(-inf) = 0
      const float pa = fast_exp2(sa - mn);
      const float pc = vc ? fast_exp2(sc - mn) : 0.f;
      l = l * corr + pa + pc;
      pa_ring16<T>(st + 2 * 512, x);
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[j] = fmaf(pa, x[j], acc[j] * corr);
      if (vc) {
        pa_ring16<T>(st + 6 * 512, x);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] = fmaf(pc, x[j], acc[j]);
      }
      m = mn;
    }
  }
  // merge the 16 token groups of this CTA (their sums take the ring's place)
  copy_wait<0>();
  __syncthreads();
  float(*s_acc)[D] = reinterpret_cast<float(*)[D]>(ring_all);
  float *s_m = reinterpret_cast<float*>(ring_all) + G * D, *s_l = s_m + G;
  if (sub == 0) { s_m[gid] = m; s_l[gid] = l; }
#pragma unroll
  for (int j = 0; j < 16; ++j) s_acc[gid][(j >> 3) * 64 + sub * 8 + (j & 7)] = acc[j];
  __syncthreads();
  {
    const int d = threadIdx.x;   // 128 threads, one output dim each
    float gm = -INFINITY;
#pragma unroll
    for (int g = 0; g < G; ++g) gm = fmaxf(gm, s_m[g]);
    float gl = 0.f, o = 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float f = s_m[g] == -INFINITY ? 0.f : fast_exp2(s_m[g] - gm);
      gl += s_l[g] * f;
      o += s_acc[g][d] * f;
    }
    const long long pi = ((long long)b * H + h) * splits + sp;
    if (splits == 1) {
      out[pi * D + d] = from_f32<T>(gl > 0.f ? o / gl : 0.f);
    } else {
      partial_o[pi * D + d] = o;
      if (d == 0) { partial_ml[pi * 2] = gm; partial_ml[pi * 2 + 1] = gl; }
    }
  }
}

template <typename T>
__global__ void paged_decode_reduce_kernel(const float* __restrict__ partial_o,
                                           const float* __restrict__ partial_ml, T* __restrict__ out,
                                           int splits) {
  constexpr int D = 128;
  const long long bh = blockIdx.x;
  const int d = threadIdx.x;
  float gm = -INFINITY;
  for (int s = 0; s < splits; ++s) gm = fmaxf(gm, partial_ml[(bh * splits + s) * 2]);
  float gl = 0.f, o = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float ms = partial_ml[(bh * splits + s) * 2];
    const float f = ms == -INFINITY ? 0.f : fast_exp2(ms - gm);
    gl += partial_ml[(bh * splits + s) * 2 + 1] * f;
    o += partial_o[(bh * splits + s) * D + d] * f;
  }
  out[bh * D + d] = from_f32<T>(gl > 0.f ? o / gl : 0.f);
}

// cache[slot[t], hkv, :] = src[t, hkv, :]   (src rows may be strided: fused qkv buffer)
template <typename T>
__global__ void kv_append_kernel(const T* __restrict__ k_src, const T* __restrict__ v_src,
                                 long long src_stride, const long long* __restrict__ slots,
                                 T* __restrict__ k_cache, T* __restrict__ v_cache, int tokens,
                                 int row_elems) {
  const int vecs = row_elems / 8;
  const long long total = (long long)tokens * vecs;
  const long long gs = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gs) {
    const int t = (int)(i / vecs);
    const int c = (int)(i - (long long)t * vecs) * 8;
    const long long slot = slots[t];
    if (slot < 0) continue;
    *reinterpret_cast<uint4*>(k_cache + slot * row_elems + c) =
        *reinterpret_cast<const uint4*>(k_src + t * src_stride + c);
    *reinterpret_cast<uint4*>(v_cache + slot * row_elems + c) =
        *reinterpret_cast<const uint4*>(v_src + t * src_stride + c);
  }
}

// Head-major cache: cache[slot / bs, hkv, slot % bs, :] = src[t, hkv, :]
template <typename T>
__global__ void kv_append_hm_kernel(const T* __restrict__ k_src, const T* __restrict__ v_src,
                                    long long src_stride, const long long* __restrict__ slots,
                                    T* __restrict__ k_cache, T* __restrict__ v_cache, int tokens, int Hkv,
                                    int D, int block_size) {
  const int vecs_per_head = D / 8;
  const int vecs = Hkv * vecs_per_head;
  const long long total = (long long)tokens * vecs;
  const long long gs = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gs) {
    const int t = (int)(i / vecs);
    const int r = (int)(i - (long long)t * vecs);
    const int hkv = r / vecs_per_head;
    const int c = (r - hkv * vecs_per_head) * 8;
    const long long slot = slots[t];
    if (slot < 0) continue;
    const long long blk = slot / block_size, off = slot % block_size;
    const long long dst = ((blk * Hkv + hkv) * block_size + off) * D + c;
    const long long src = t * src_stride + (long long)hkv * D + c;
    *reinterpret_cast<uint4*>(k_cache + dst) = *reinterpret_cast<const uint4*>(k_src + src);
    *reinterpret_cast<uint4*>(v_cache + dst) = *reinterpret_cast<const uint4*>(v_src + src);
  }
}

// Rotary embedding of the query and key heads of packed rows [q | k | v] (pairs (i, i + hd/2)) in place, and the rotated keys and the values into the
// cache: one pass over the rows where two rotations and an append take three.  A CTA per token (gridDim.y of them
// share its heads): the angles are computed once per pair, not once per pair and head, and heads move in 16-byte pieces.
// 1555 tokens of 32 + 32 heads: 15 us; 21.5 us a rotation and 7.8 us an append before.
template <typename T, bool HM>
__global__ void __launch_bounds__(256)
    rope_append_kernel(T* __restrict__ qkv, long long ld, const long long* __restrict__ pos_ids, const long long* __restrict__ slots,
                       T* __restrict__ k_cache, T* __restrict__ v_cache, int H, int Hkv, int hd, int block_size, float theta) {
  extern __shared__ float s_angle[];                 // [hd/2] cosines, [hd/2] sines
  const int half = hd / 2;
  const long long t = blockIdx.x;
  const float posf = (float)pos_ids[t];
  for (int p = threadIdx.x; p < half; p += blockDim.x) {
    const float inv_freq = __powf(theta, -2.0f * (float)p / (float)hd);
    float sn, cs;
    sincosf(posf * inv_freq, &sn, &cs);
    s_angle[p] = cs;
    s_angle[half + p] = sn;
  }
  __syncthreads();
  T* row = qkv + t * ld;
  const long long slot = slots[t];
  auto place = [&](int hkv) -> long long {
    if constexpr (HM) return (((slot / block_size) * Hkv + hkv) * block_size + slot % block_size) * hd;
    else return (slot * Hkv + hkv) * hd;
  };
  const int first = blockIdx.y * blockDim.x + threadIdx.x, step = gridDim.y * blockDim.x;
  const int per = half / 8;
  for (int i = first; i < (H + Hkv) * per; i += step) {
    const int h = i / per, c = (i - h * per) * 8;
    T* base = row + (long long)h * hd + c;
    const uint4 lo = *reinterpret_cast<const uint4*>(base), hi = *reinterpret_cast<const uint4*>(base + half);
    const uint32_t l[4] = {lo.x, lo.y, lo.z, lo.w}, u[4] = {hi.x, hi.y, hi.z, hi.w};
    uint32_t a[4], b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = unpack2<T>(l[j]), y = unpack2<T>(u[j]);
      const float c0 = s_angle[c + 2 * j], c1 = s_angle[c + 2 * j + 1];
      const float s0 = s_angle[half + c + 2 * j], s1 = s_angle[half + c + 2 * j + 1];
      a[j] = pack2<T>(x.x * c0 - y.x * s0, x.y * c1 - y.y * s1);
      b[j] = pack2<T>(y.x * c0 + x.x * s0, y.y * c1 + x.y * s1);
    }
    const uint4 na = make_uint4(a[0], a[1], a[2], a[3]), nb = make_uint4(b[0], b[1], b[2], b[3]);
    *reinterpret_cast<uint4*>(base) = na;
    *reinterpret_cast<uint4*>(base + half) = nb;
    if (h >= H && slot >= 0) {
      T* dst = k_cache + place(h - H) + c;
      *reinterpret_cast<uint4*>(dst) = na;
      *reinterpret_cast<uint4*>(dst + half) = nb;
    }
  }
  if (slot < 0) return;
  const T* v = row + (long long)(H + Hkv) * hd;
  const int vper = hd / 8;
  for (int i = first; i < Hkv * vper; i += step) {
    const int h = i / vper, c = (i - h * vper) * 8;
    *reinterpret_cast<uint4*>(v_cache + place(h) + c) = *reinterpret_cast<const uint4*>(v + (long long)h * hd + c);
  }
}

// out_idx[r] = argmax_c x[r, c] (first maximum), out_val[r] = the maximum
template <typename T>
__global__ void __launch_bounds__(256)
    argmax_kernel(const T* __restrict__ x, long long ld, int n, long long* __restrict__ out_idx,
                  float* __restrict__ out_val) {
  __shared__ float sv[8];
  __shared__ int si[8];
  const T* row = x + (long long)blockIdx.x * ld;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    const float v = to_f32<T>(row[c]);
    if (v > best || (v == best && c < bi)) { best = v; bi = c; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; si[threadIdx.x >> 5] = bi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w)
      if (sv[w] > best || (sv[w] == best && si[w] < bi)) { best = sv[w]; bi = si[w]; }
    out_idx[blockIdx.x] = bi;
    if (out_val) out_val[blockIdx.x] = best;
  }
}

}  // namespace rb

extern "C" {

// CTAs that share the keys of one (row, head): parts of at most 512 tokens up to 8192 tokens (sixteen parts, longer ones beyond), shorter
// ones (down to 64 tokens) while the rows and heads alone leave less than four CTAs to an SM.  130 tokens of 48 rows of 8 heads:
// 6.2 us in one part, 10.4 in two; of 8 rows of 32 heads 5.4, 9.2 in three.
int rb_paged_decode_splits(int max_ctx, int rows_heads) {
  const int fill = (4 * rbh::sm_count() + rows_heads - 1) / (rows_heads > 0 ? rows_heads : 1);
  int s = fill < (max_ctx + 63) / 64 ? fill : (max_ctx + 63) / 64;
  if (fill < 4 && max_ctx <= 192) s = 1;       // two or three short parts save less than adding them up takes
  if (s < (max_ctx + 511) / 512) s = (max_ctx + 511) / 512;
  if (s > 16) s = 16;
  if (s < 1) s = 1;
  return s;
}

}

namespace rb {
template <typename T, bool HM>
static int paged_decode(const void* q, long long ldq, const void* k_cache, const void* v_cache, const int* block_tables,
                        const int* ctx_lens, void* out, float* scratch_o, float* scratch_ml, int B, int H, int Hkv,
                        int block_size, int max_blocks, int splits, float scale, cudaStream_t st) {
  int shift = -1;
  if ((block_size & (block_size - 1)) == 0)
    for (shift = 0; (1 << shift) < block_size; ++shift) {}
  paged_decode_attn_kernel<T, HM><<<dim3(H, B, splits), kPaWarps * 32, 0, st>>>(
      (const T*)q, ldq, (const T*)k_cache, (const T*)v_cache, block_tables, ctx_lens, scratch_o, scratch_ml, (T*)out, H, Hkv,
      block_size, shift, max_blocks, splits, scale * 1.4426950408889634f);
  if (splits > 1) paged_decode_reduce_kernel<T><<<B * H, 128, 0, st>>>(scratch_o, scratch_ml, (T*)out, splits);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 3000 + (int)e;
}
}  // namespace rb

extern "C" {

// q: rows of H * 128, ldq apart (a multiple of 8); out [B,H,128]; scratch_o: B*H*splits*128 floats; scratch_ml: B*H*splits*2 floats
// (neither is used with one split).  head_major: the cache is [num_blocks, Hkv, block_size, 128].
int rb_paged_decode_attn(int dtype, int head_major, const void* q, long long ldq, const void* k_cache, const void* v_cache,
                         const int* block_tables, const int* ctx_lens, void* out, float* scratch_o,
                         float* scratch_ml, int B, int H, int Hkv, int head_dim, int block_size,
                         int max_blocks, int splits, float scale, void* stream) {
  using namespace rb;
  if (head_dim != 128) return 20;
  if (B <= 0) return 0;
  if (ldq % 8) return 21;
  cudaStream_t st = (cudaStream_t)stream;
#define RB_PA(T)                                                                                                        \
  (head_major ? paged_decode<T, true>(q, ldq, k_cache, v_cache, block_tables, ctx_lens, out, scratch_o, scratch_ml, B, \
                                      H, Hkv, block_size, max_blocks, splits, scale, st)                                \
              : paged_decode<T, false>(q, ldq, k_cache, v_cache, block_tables, ctx_lens, out, scratch_o, scratch_ml, B, \
                                       H, Hkv, block_size, max_blocks, splits, scale, st))
  if (dtype == rbh::DT_BF16) return RB_PA(__nv_bfloat16);
  if (dtype == rbh::DT_F16) return RB_PA(__half);
#undef RB_PA
  return 20;
}

int rb_kv_append(int dtype, const void* k_src, const void* v_src, long long src_stride,
                 const long long* slots, void* k_cache, void* v_cache, int tokens, int row_elems,
                 void* stream) {
  using namespace rb;
  if (tokens <= 0) return 0;
  if (row_elems % 8 != 0 || src_stride % 8 != 0) return 21;
  cudaStream_t st = (cudaStream_t)stream;
  const long long total = (long long)tokens * (row_elems / 8);
  const unsigned blocks = (unsigned)((total + 255) / 256);
  if (dtype == rbh::DT_BF16)
    kv_append_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>((const __nv_bfloat16*)k_src, (const __nv_bfloat16*)v_src, src_stride, slots, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, tokens, row_elems);
  else if (dtype == rbh::DT_F16)
    kv_append_kernel<__half><<<blocks, 256, 0, st>>>((const __half*)k_src, (const __half*)v_src, src_stride, slots, (__half*)k_cache, (__half*)v_cache, tokens, row_elems);
  else
    return 20;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 3000 + (int)e;
}

// Head-major cache [num_blocks, Hkv, block_size, D].
int rb_kv_append_hm(int dtype, const void* k_src, const void* v_src, long long src_stride,
                    const long long* slots, void* k_cache, void* v_cache, int tokens, int Hkv, int D,
                    int block_size, void* stream) {
  using namespace rb;
  if (tokens <= 0) return 0;
  if (D % 8 != 0 || src_stride % 8 != 0) return 21;
  cudaStream_t st = (cudaStream_t)stream;
  const long long total = (long long)tokens * Hkv * (D / 8);
  const unsigned blocks = (unsigned)((total + 255) / 256);
  if (dtype == rbh::DT_BF16)
    kv_append_hm_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>((const __nv_bfloat16*)k_src, (const __nv_bfloat16*)v_src, src_stride, slots, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, tokens, Hkv, D, block_size);
  else if (dtype == rbh::DT_F16)
    kv_append_hm_kernel<__half><<<blocks, 256, 0, st>>>((const __half*)k_src, (const __half*)v_src, src_stride, slots, (__half*)k_cache, (__half*)v_cache, tokens, Hkv, D, block_size);
  else
    return 20;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 3000 + (int)e;
}

// qkv: rows [H heads | Hkv heads | Hkv heads] of hd numbers, ld apart; hd a multiple of 16, ld of 8.  slot < 0: not stored.
int rb_rope_append(int dtype, int head_major, void* qkv, long long ld, const long long* pos_ids, const long long* slots, void* k_cache,
                   void* v_cache, int tokens, int H, int Hkv, int hd, int block_size, float theta, void* stream) {
  using namespace rb;
  if (tokens <= 0) return 0;
  if (hd % 16 != 0 || hd > 1024 || ld % 8 != 0 || (reinterpret_cast<uintptr_t>(qkv) & 15)) return 21;
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid(tokens, tokens < rbh::sm_count() ? 4 : 1);
#define RB_ROPE_APPEND(T, HM) \
  rope_append_kernel<T, HM><<<grid, 256, hd * sizeof(float), st>>>((T*)qkv, ld, pos_ids, slots, (T*)k_cache, (T*)v_cache, H, Hkv, hd, block_size, theta)
  if (dtype == rbh::DT_BF16) { if (head_major) RB_ROPE_APPEND(__nv_bfloat16, true); else RB_ROPE_APPEND(__nv_bfloat16, false); }
  else if (dtype == rbh::DT_F16) { if (head_major) RB_ROPE_APPEND(__half, true); else RB_ROPE_APPEND(__half, false); }
  else return 20;
#undef RB_ROPE_APPEND
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 3000 + (int)e;
}

int rb_argmax(int dtype, const void* x, long long ld, int rows, int n, long long* out_idx,
              float* out_val, void* stream) {
  using namespace rb;
  if (rows <= 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == rbh::DT_BF16) argmax_kernel<__nv_bfloat16><<<rows, 256, 0, st>>>((const __nv_bfloat16*)x, ld, n, out_idx, out_val);
  else if (dtype == rbh::DT_F16) argmax_kernel<__half><<<rows, 256, 0, st>>>((const __half*)x, ld, n, out_idx, out_val);
  else argmax_kernel<float><<<rows, 256, 0, st>>>((const float*)x, ld, n, out_idx, out_val);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 3000 + (int)e;
}
}
