// Attention in 32 bits, forward and backward (the products stay on the FP32 pipes: no TF32 rounding): one launch each where the
// composition of batched products, scaling, mask and softmax takes some twenty forward and twice as many backward.  Meant for the
// small models that train in 32 bits: what bounds them is launches and latency, not arithmetic.
//
// A row (of queries; of keys for dK and dV) belongs to D / 16 neighbouring lanes with sixteen of its numbers each, in pieces of four
// that alternate between the lanes, so that the lanes read one row of a tile in shared memory without bank conflicts and the rows of a
// warp share the read.  Tiles of 32 rows pass through shared memory.  The forward pass keeps a running maximum per row and takes four
// keys at a time; the backward pass recomputes the weights from the log-sum-exp.  Its two halves, dQ by query rows and dK, dV by key rows,
// run side by side in one grid: nothing is added up in memory, so results do not depend on the order of CTAs.
//
// The reference composes this operation (rumus/src/nn/attention.rs:17-58).
#include "sm100_common.cuh"

namespace rb {

constexpr int AF_THREADS = 128, AF_TILE = 32;

struct AttnF32Params {
  const float *q, *k, *v, *o, *dout;
  float *out, *lse, *dq, *dk, *dv;      // out, o: [B, Sq, H, D]; lse: [B, H, Sq]
  long long qs[3], ks[3], vs[3], dos[3], dqs[3], dks[3], dvs[3];     // {batch, row, head}
  int B, H, Sq, Sk, causal;
  float scale;
};

template <int D>
struct AttnF32Row {
  static constexpr int LANES = D / 16, ROWS = AF_THREADS / LANES;
  static __device__ __forceinline__ void load(const float* p, int sub, float4 (&r)[4]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) r[c] = *reinterpret_cast<const float4*>(p + (c * LANES + sub) * 4);
  }
  static __device__ __forceinline__ void store(float* p, int sub, const float4 (&r)[4]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) *reinterpret_cast<float4*>(p + (c * LANES + sub) * 4) = r[c];
  }
  static __device__ __forceinline__ float dot(const float4 (&a)[4], const float4 (&b)[4]) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) s = fmaf(a[c].x, b[c].x, fmaf(a[c].y, b[c].y, fmaf(a[c].z, b[c].z, fmaf(a[c].w, b[c].w, s))));
    return s;
  }
  static __device__ __forceinline__ float all(float s) {
#pragma unroll
    for (int o = 1; o < LANES; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  }
};
__device__ __forceinline__ void af_axpy(float a, const float4 (&x)[4], float4 (&y)[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    y[c].x = fmaf(a, x[c].x, y[c].x);
    y[c].y = fmaf(a, x[c].y, y[c].y);
    y[c].z = fmaf(a, x[c].z, y[c].z);
    y[c].w = fmaf(a, x[c].w, y[c].w);
  }
}
__device__ __forceinline__ void af_zero(float4 (&y)[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) y[c] = make_float4(0.f, 0.f, 0.f, 0.f);
}
// rows [r0, r0 + AF_TILE) of a strided [rows, D] matrix into shared memory, zeros beyond n
template <int D>
__device__ __forceinline__ void af_tile(float* dst, const float* src, long long stride, int r0, int n) {
  for (int i = threadIdx.x; i < AF_TILE * D / 4; i += AF_THREADS) {
    const int r = i / (D / 4), c = i % (D / 4);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r0 + r < n) v = *reinterpret_cast<const float4*>(src + (long long)(r0 + r) * stride + c * 4);
    *reinterpret_cast<float4*>(dst + r * D + c * 4) = v;
  }
}

template <int D>
__global__ void __launch_bounds__(AF_THREADS) attn_f32_fwd_kernel(const AttnF32Params p) {
  using R = AttnF32Row<D>;
  __shared__ __align__(16) float sk[AF_TILE * D], sv[AF_TILE * D];
  const int sub = threadIdx.x % R::LANES, b = blockIdx.z, h = blockIdx.y;
  const int row0 = (gridDim.x - 1 - blockIdx.x) * R::ROWS, row = row0 + threadIdx.x / R::LANES;   // the longest first
  const int off = p.Sk - p.Sq;
  const float* k = p.k + b * p.ks[0] + h * p.ks[2];
  const float* v = p.v + b * p.vs[0] + h * p.vs[2];
  float4 q[4], acc[4];
  af_zero(q);
  af_zero(acc);
  if (row < p.Sq) R::load(p.q + b * p.qs[0] + (long long)row * p.qs[1] + h * p.qs[2], sub, q);
  const int keys = row >= p.Sq ? 0 : p.causal ? min(p.Sk, row + off + 1) : p.Sk;                 // this row's
  const int end = p.causal ? min(p.Sk, min(row0 + R::ROWS, p.Sq) + off) : p.Sk;                  // the CTA's
  float m = -INFINITY, l = 0.f;
  for (int j0 = 0; j0 < end; j0 += AF_TILE) {
    __syncthreads();
    af_tile<D>(sk, k, p.ks[1], j0, p.Sk);
    af_tile<D>(sv, v, p.vs[1], j0, p.Sk);
    __syncthreads();
    for (int j = 0; j < AF_TILE && j0 + j < end; j += 4) {
      float s[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float4 x[4];
        R::load(sk + (j + u) * D, sub, x);
        s[u] = R::dot(q, x);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s[u] = R::all(s[u]) * p.scale;
        if (j0 + j + u >= keys) s[u] = -INFINITY;
      }
      const float mn = fmaxf(m, fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3])));
      // no key of the group is seen by this row: all of them are -inf.  fmaxf passes over NaN, a sum does not.
      if (mn != -INFINITY || (s[0] + s[1]) + (s[2] + s[3]) != -INFINITY) {
        const float f = expf(m - mn);
        l *= f;
#pragma unroll
        for (int c = 0; c < 4; ++c) { acc[c].x *= f; acc[c].y *= f; acc[c].z *= f; acc[c].w *= f; }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float w = expf(s[u] - mn);
          l += w;
          float4 x[4];
          R::load(sv + (j + u) * D, sub, x);
          af_axpy(w, x, acc);
        }
        m = mn;
      }
    }
  }
  if (row >= p.Sq) return;
  const float inv = 1.f / l;
#pragma unroll
  for (int c = 0; c < 4; ++c) { acc[c].x *= inv; acc[c].y *= inv; acc[c].z *= inv; acc[c].w *= inv; }
  R::store(p.out + (((long long)b * p.Sq + row) * p.H + h) * D, sub, acc);
  if (sub == 0) p.lse[((long long)b * p.H + h) * p.Sq + row] = m + logf(l);
}

template <int D>
__global__ void __launch_bounds__(AF_THREADS) attn_f32_bwd_kernel(const AttnF32Params p, int query_blocks) {
  using R = AttnF32Row<D>;
  __shared__ __align__(16) float sa[AF_TILE * D], sb[AF_TILE * D];
  __shared__ float s_lse[AF_TILE], s_delta[AF_TILE];
  const int sub = threadIdx.x % R::LANES, b = blockIdx.z, h = blockIdx.y;
  const int off = p.Sk - p.Sq;
  const float* q = p.q + b * p.qs[0] + h * p.qs[2];
  const float* k = p.k + b * p.ks[0] + h * p.ks[2];
  const float* v = p.v + b * p.vs[0] + h * p.vs[2];
  const float* dout = p.dout + b * p.dos[0] + h * p.dos[2];
  const float* o = p.o + ((long long)b * p.Sq * p.H + h) * D;           // rows H * D apart
  const long long os = (long long)p.H * D;
  const float* lse = p.lse + ((long long)b * p.H + h) * p.Sq;
  float4 x[4], y[4];
  if ((int)blockIdx.x < query_blocks) {
    // ---- dQ of a block of queries ----
    const int row0 = (query_blocks - 1 - blockIdx.x) * R::ROWS, row = row0 + threadIdx.x / R::LANES;
    const bool live = row < p.Sq;
    float4 qr[4], g[4], acc[4];
    af_zero(qr);
    af_zero(g);
    af_zero(acc);
    float delta = 0.f, ls = 0.f;
    if (live) {
      R::load(q + (long long)row * p.qs[1], sub, qr);
      R::load(dout + (long long)row * p.dos[1], sub, g);
      R::load(o + row * os, sub, x);
      delta = R::dot(g, x);
      ls = lse[row];
    }
    delta = R::all(delta);
    const int keys = !live ? 0 : p.causal ? min(p.Sk, row + off + 1) : p.Sk;
    const int end = p.causal ? min(p.Sk, min(row0 + R::ROWS, p.Sq) + off) : p.Sk;
    for (int j0 = 0; j0 < end; j0 += AF_TILE) {
      __syncthreads();
      af_tile<D>(sa, k, p.ks[1], j0, p.Sk);
      af_tile<D>(sb, v, p.vs[1], j0, p.Sk);
      __syncthreads();
#pragma unroll 2
      for (int j = 0; j < AF_TILE; ++j) {
        if (j0 + j >= end) break;
        R::load(sa + j * D, sub, x);
        R::load(sb + j * D, sub, y);
        const float s = R::all(R::dot(qr, x)), dp = R::all(R::dot(g, y));
        const float w = j0 + j < keys ? expf(s * p.scale - ls) : 0.f;
        af_axpy(w * (dp - delta) * p.scale, x, acc);
      }
    }
    if (live) R::store(p.dq + b * p.dqs[0] + (long long)row * p.dqs[1] + h * p.dqs[2], sub, acc);
    return;
  }
  // ---- dK and dV of a block of keys ----
  const int row0 = (blockIdx.x - query_blocks) * R::ROWS, row = row0 + threadIdx.x / R::LANES;      // early keys, which most rows see, first
  const bool live = row < p.Sk;
  float4 kr[4], vr[4], dk[4], dv[4];
  af_zero(kr);
  af_zero(vr);
  af_zero(dk);
  af_zero(dv);
  if (live) {
    R::load(k + (long long)row * p.ks[1], sub, kr);
    R::load(v + (long long)row * p.vs[1], sub, vr);
  }
  const int first = p.causal ? max(0, row - off) : 0;                      // the first query that sees this key
  const int begin = p.causal ? max(0, row0 - off) / AF_TILE * AF_TILE : 0;
  for (int i0 = begin; i0 < p.Sq; i0 += AF_TILE) {
    __syncthreads();
    af_tile<D>(sa, q, p.qs[1], i0, p.Sq);
    // dO, and sum dO O of its rows: D / 4 lanes a row
    for (int i = threadIdx.x; i < AF_TILE * D / 4; i += AF_THREADS) {
      const int r = i / (D / 4), c = i % (D / 4);
      float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
      float part = 0.f;
      if (i0 + r < p.Sq) {
        g = *reinterpret_cast<const float4*>(dout + (long long)(i0 + r) * p.dos[1] + c * 4);
        const float4 u = *reinterpret_cast<const float4*>(o + (i0 + r) * os + c * 4);
        part = fmaf(g.x, u.x, fmaf(g.y, u.y, fmaf(g.z, u.z, g.w * u.w)));
      }
      *reinterpret_cast<float4*>(sb + r * D + c * 4) = g;
#pragma unroll
      for (int w = 1; w < D / 4; w <<= 1) part += __shfl_xor_sync(0xffffffffu, part, w);
      if (c == 0) {
        s_delta[r] = part;
        s_lse[r] = i0 + r < p.Sq ? lse[i0 + r] : 0.f;
      }
    }
    __syncthreads();
#pragma unroll 2
    for (int i = 0; i < AF_TILE; ++i) {
      if (i0 + i >= p.Sq) break;
      R::load(sa + i * D, sub, x);
      R::load(sb + i * D, sub, y);
      const float s = R::all(R::dot(kr, x)), dp = R::all(R::dot(vr, y));
      const float w = live && i0 + i >= first ? expf(s * p.scale - s_lse[i]) : 0.f;
      af_axpy(w, y, dv);
      af_axpy(w * (dp - s_delta[i]) * p.scale, x, dk);
    }
  }
  if (live) {
    R::store(p.dk + b * p.dks[0] + (long long)row * p.dks[1] + h * p.dks[2], sub, dk);
    R::store(p.dv + b * p.dvs[0] + (long long)row * p.dvs[1] + h * p.dvs[2], sub, dv);
  }
}

}  // namespace rb

extern "C" {

// fp32; head sizes 16, 32, 64, 128; rows of D numbers, 16-byte aligned; strides {batch, row, head}.  A causal call needs Sk >= Sq, so that every
// row sees a key.  20: not covered.
int rb_attn_f32_fwd(int D, const float* q, const float* k, const float* v, const long long* qs, const long long* ks, const long long* vs,
                    float* out, float* lse, int B, int H, int Sq, int Sk, int causal, float scale, void* stream) {
  using namespace rb;
  if (B <= 0 || H <= 0 || Sq <= 0) return 0;
  if (Sk <= 0 || (causal && Sk < Sq) || B > 65535 || H > 65535) return 20;
  AttnF32Params p{};
  p.q = q; p.k = k; p.v = v; p.out = out; p.lse = lse;
  for (int i = 0; i < 3; ++i) { p.qs[i] = qs[i]; p.ks[i] = ks[i]; p.vs[i] = vs[i]; }
  p.B = B; p.H = H; p.Sq = Sq; p.Sk = Sk; p.causal = causal; p.scale = scale;
  cudaStream_t st = (cudaStream_t)stream;
#define RB_AF(D_)                                                                                                                \
  if (D == D_) {                                                                                                                 \
    attn_f32_fwd_kernel<D_><<<dim3((Sq + AttnF32Row<D_>::ROWS - 1) / AttnF32Row<D_>::ROWS, H, B), AF_THREADS, 0, st>>>(p);       \
    cudaError_t e = cudaGetLastError();                                                                                          \
    return e == cudaSuccess ? 0 : 3000 + (int)e;                                                                                 \
  }
  RB_AF(16) RB_AF(32) RB_AF(64) RB_AF(128)
#undef RB_AF
  return 20;
}

int rb_attn_f32_bwd(int D, const float* q, const float* k, const float* v, const float* o, const float* dout, float* lse,
                    const long long* qs, const long long* ks, const long long* vs, const long long* dos, float* dq, float* dk, float* dv,
                    const long long* dqs, const long long* dks, const long long* dvs, int B, int H, int Sq, int Sk, int causal,
                    float scale, void* stream) {
  using namespace rb;
  if (B <= 0 || H <= 0 || Sq <= 0) return 0;
  if (Sk <= 0 || (causal && Sk < Sq) || B > 65535 || H > 65535) return 20;
  AttnF32Params p{};
  p.q = q; p.k = k; p.v = v; p.o = o; p.dout = dout; p.lse = lse; p.dq = dq; p.dk = dk; p.dv = dv;
  for (int i = 0; i < 3; ++i) {
    p.qs[i] = qs[i]; p.ks[i] = ks[i]; p.vs[i] = vs[i]; p.dos[i] = dos[i];
    p.dqs[i] = dqs[i]; p.dks[i] = dks[i]; p.dvs[i] = dvs[i];
  }
  p.B = B; p.H = H; p.Sq = Sq; p.Sk = Sk; p.causal = causal; p.scale = scale;
  cudaStream_t st = (cudaStream_t)stream;
#define RB_AF(D_)                                                                                                                \
  if (D == D_) {                                                                                                                 \
    constexpr int R = AttnF32Row<D_>::ROWS;                                                                                      \
    const int nq = (Sq + R - 1) / R, nk = (Sk + R - 1) / R;                                                                      \
    attn_f32_bwd_kernel<D_><<<dim3(nq + nk, H, B), AF_THREADS, 0, st>>>(p, nq);                                                  \
    cudaError_t e = cudaGetLastError();                                                                                          \
    return e == cudaSuccess ? 0 : 3000 + (int)e;                                                                                 \
  }
  RB_AF(16) RB_AF(32) RB_AF(64) RB_AF(128)
#undef RB_AF
  return 20;
}
}
