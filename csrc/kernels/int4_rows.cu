// INT4 products of decode batches (1..48 rows): Y[M, N] = X[M, K] . dequant(W4)[K, N] (+ bias) (+ residual)
//
// Bound by the packed weights' way from HBM (half a byte a weight, 14 MB for 4096 x 4096 x 1.5), so the weights go straight into
// the tensor cores' registers and nothing wider than four bits is ever stored:
//
//   * a warp owns 32 columns and takes 128 k a step: four 16-byte copies a lane (cp.async into a ring, two steps ahead).
//     With up to eight rows its activations come the same way and warps never wait for one another; with more rows, warps side by
//     side over columns share the activations of a step;
//   * a packed word holds eight consecutive k of one column.  mma.sync m16n8k16 takes the weights as its left operand: lane
//     (g, t) has the words of columns 4 g .. 4 g + 3 at k = 8 t .. 8 t + 7, which are the left operands of two 16 x 16 tiles of
//     two products, when the activations take the same order of k: nibbles p and p + 4 come out of a word together, so a piece
//     of eight is read as (0 4) (1 5) (2 6) (3 7);
//   * up to eight rows: the operand is q - 8, which is exact in 16 bits; the products of a group are summed in fp32 and scaled in fp32
//     after it: acc += scale (sum (q - 8) x - (zp - 8) sum x), with sum x of each row from a product with ones.  Only the result is
//     rounded, as in a product with fp32 weights.  More rows: the operand is (q - 8) scale + (8 - zp) scale in 16 bits, the
//     weights of w4a16_gemm.cu, and all of K goes into one sum;
//   * K is split over the warps of a CTA and, where the columns alone leave SMs idle, over a cluster of up to eight CTAs that
//     add their sums through distributed shared memory in a fixed order: no workspace, no second launch.
//
// The four products of a 7B layer (4096 x 12288, 4096 x 4096, 4096 x 22016, 11008 x 4096), microseconds in all, against the streaming GEMV (1, 8 rows) and
// the tcgen05 kernel that expands weights into shared memory (16 to 48 rows):  1 row 62 (102),  8 rows 65 (212),  16: 85 (181),  24: 94 (203),
// 32: 104 (219),  48: 132 (254); the weights' way from HBM is 17.  With few rows the SMs' integer pipes (seven operations a
// word) and the wait for the first words share the rest, with many the instructions of the products.
//
// Packed layout (rumus-vision/src/quant.rs:42-126): word (k/8)*N + n holds k..k+7 of column n, nibble k%8; scales and zero
// points are [K/group, N].
#include <cooperative_groups.h>

#include "warp_mma.cuh"

namespace rb {

constexpr int I4_GROUP = 128;      // k per pipeline step

struct I4Params {
  const void* x;                   // [M, K] of T
  const int* packed;
  const void *scales, *zps;
  const void* bias;                // [N] of T or null
  const void* residual;            // [M, N] of T or null
  void* y;                         // [M, N] of T
  int M, N, K, steps;              // steps of 128 k in the padded K
  int steps_per_group, slice;      // quantisation group / 128; steps per CTA of a cluster
};

template <typename T> struct I4Num;
template <> struct I4Num<__nv_bfloat16> {
  using V = __nv_bfloat162;
  static constexpr uint32_t magic = 0x43004300u, ones = 0x3f803f80u;      // 128 + q is exact
  static __device__ __forceinline__ V splat(float v) { return __float2bfloat162_rn(v); }
  static __device__ __forceinline__ V base() { return splat(136.f); }
};
template <> struct I4Num<__half> {
  using V = __half2;
  static constexpr uint32_t magic = 0x64006400u, ones = 0x3c003c00u;      // 1024 + q is exact
  static __device__ __forceinline__ V splat(float v) { return __float2half2_rn(v); }
  static __device__ __forceinline__ V base() { return splat(1032.f); }
};

template <typename T>
__device__ __forceinline__ void i4_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void i4_mma<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void i4_mma<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the first product of a step: nothing to add to
template <typename T>
__device__ __forceinline__ void i4_mma_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void i4_mma_first<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
template <>
__device__ __forceinline__ void i4_mma_first<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// nibbles (p, p + 4) of a word, minus 8, for p = 0..3
template <typename T>
__device__ __forceinline__ void i4_expand(uint32_t w, uint32_t (&v)[4]) {
  using V = typename I4Num<T>::V;
  const V base = I4Num<T>::base();
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    uint32_t u = ((w >> (4 * p)) & 0x000f000fu) | I4Num<T>::magic;
    V q = __hsub2(*reinterpret_cast<V*>(&u), base);
    v[p] = *reinterpret_cast<uint32_t*>(&q);
  }
}

template <typename TS> __device__ __forceinline__ void i4_load4(const uint8_t* p, float (&v)[4]);
template <> __device__ __forceinline__ void i4_load4<float>(const uint8_t* p, float (&v)[4]) {
  const float4 f = *reinterpret_cast<const float4*>(p);
  v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
template <> __device__ __forceinline__ void i4_load4<__half>(const uint8_t* p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack2<__half>(u.x), b = unpack2<__half>(u.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

template <int BYTES>
__device__ __forceinline__ void i4_copy(uint32_t dst, const void* src, bool live) {
  if constexpr (BYTES == 16) copy16(dst, src, live);
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(live ? 8 : 0) : "memory");
}

// NT: groups of eight rows; WN: warps over columns; WK: over K.
template <int NT_> struct I4Cfg {
  static constexpr int NT = NT_;
  static constexpr int WN = NT == 1 ? 1 : NT == 2 ? 2 : 4;
  static constexpr int WARPS = 8, THREADS = 32 * WARPS;
  static constexpr int WK = WARPS / WN;
  static constexpr int COLS = 32 * WN;
  static constexpr int STAGES = NT <= 4 ? 3 : 2;    // two CTAs of 48 rows fit an SM with two
  static constexpr int CTAS = 2;                    // per SM
};
// a warp's share of a stage: words, scales, zero points
template <typename TS> constexpr int i4_words_bytes() { return 2048 + 32 * 8 * (int)sizeof(TS); }
// Activations of a step: rows of 256 bytes, the halves of every other 128 bytes swapped in odd rows, so that the rows g and g + 1 that eight
// lanes read together lie in different banks.
__device__ __forceinline__ uint32_t i4_x_at(int row, int piece) { return row * 256 + ((piece ^ ((row & 1) << 2)) << 4); }

// The sums of one step, element by element, for a row whose sum x is not finite: an infinity times q - 8 and times zp - 8 would
// cancel to a NaN where the weight itself has a sign.
template <typename T>
__device__ __noinline__ float i4_plain(const uint8_t* words, const uint8_t* x, int row, int word, float s, float z) {
  float sum = 0.f;
  for (int k8 = 0; k8 < 16; ++k8) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(words + (k8 >> 2) * 512 + (k8 & 3) * 16 + word * 4);
    const T* xv = reinterpret_cast<const T*>(x + i4_x_at(row, k8));
    for (int k = 0; k < 8; ++k) sum = fmaf(to_f32<T>(xv[k]), ((float)((w >> (4 * k)) & 0xf) - z) * s, sum);
  }
  return sum;
}

template <typename T, typename TS, class C>
__global__ void __launch_bounds__(C::THREADS, C::CTAS) int4_rows_kernel(const I4Params p) {
  constexpr int NT = C::NT, ROWS = NT * 8;
  constexpr int WB = i4_words_bytes<TS>();
  constexpr bool ALONE = C::WN == 1;                  // each warp's activations are its own
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int wn = warp % C::WN, wk = warp / C::WN;
  const int x_bytes = p.M * 256;                      // of one step
  const int stage_bytes = 8 * WB + C::WK * x_bytes;
  const int n0 = blockIdx.x * C::COLS;
  const int col = n0 + wn * 32 + 4 * g;
  const bool live = col < p.N;
  const int s0 = blockIdx.y * p.slice, s1 = min(p.steps, s0 + p.slice);
  const int rounds = s1 > s0 ? (s1 - s0 + C::WK - 1) / C::WK : 0;

  // ---- copies: what a round adds to each address is constant ----
  constexpr int B = 4 * sizeof(TS);
  const long long row4 = 16ll * p.N, word_round = (long long)C::WK * 64 * p.N;
  const char* wsrc = reinterpret_cast<const char*>(p.packed + (live ? col : 0) + (long long)((s0 + wk) * 16 + t) * p.N);
  const TS* scales = static_cast<const TS*>(p.scales) + (live ? col : 0);
  const TS* zps = static_cast<const TS*>(p.zps) + (live ? col : 0);
  const uint32_t wdst = smem_u32(smem) + warp * WB + lane * 16, sdst = smem_u32(smem) + warp * WB + 2048 + lane * B;
  // activations: a thread copies the same piece of every XR-th row
  constexpr int XT = ALONE ? 32 : C::THREADS, XR = XT / 16 / (ALONE ? 1 : C::WK), XU = (ROWS + XR - 1) / XR;
  static_assert(XR % 2 == 0, "the swizzle of a thread's rows is one");
  const int xe = ALONE ? lane : threadIdx.x;
  const int x_w = ALONE ? wk : (xe >> 4) % C::WK, x_row = ALONE ? xe >> 4 : (xe >> 4) / C::WK;
  int x_k = (s0 + x_w) * I4_GROUP + (xe & 15) * 8;
  const T* x_base = static_cast<const T*>(p.x) + (long long)x_row * p.K;
  const long long x_step = (long long)XR * p.K;
  const uint32_t xdst = smem_u32(smem) + 8 * WB + x_w * x_bytes + i4_x_at(x_row, xe & 15);
  int f_step = s0 + wk, f_x = s0 + x_w, f_stage = 0;
  auto fetch = [&]() {
    const uint32_t at = f_stage * stage_bytes;
    if (f_step < s1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) copy16(wdst + at + j * 512, wsrc + j * row4, live);
      const long long q = (long long)(p.steps_per_group == 1 ? f_step : f_step / p.steps_per_group) * p.N;
      i4_copy<B>(sdst + at, scales + q, live);
      i4_copy<B>(sdst + at + 32 * B, zps + q, live);
    }
    if (f_x < s1) {
      const bool in = x_k < p.K;
      const T* src = x_base + (in ? x_k : 0);
#pragma unroll
      for (int u = 0; u < XU; ++u)
        if (x_row + u * XR < p.M) copy16(xdst + at + u * (XR * 256), src + u * x_step, in);
    }
    f_step += C::WK;
    f_x += C::WK;
    wsrc += word_round;
    x_k += C::WK * I4_GROUP;
    f_stage = f_stage == C::STAGES - 1 ? 0 : f_stage + 1;
    copy_commit();
  };
#pragma unroll
  for (int i = 0; i < C::STAGES - 1; ++i) fetch();

  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][n][c] = 0.f;
  // rows beyond M read the last one; their sums are never stored
  uint32_t xoff[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) xoff[n] = i4_x_at(min(n * 8 + g, p.M - 1), t);
  auto x_of = [&](const uint8_t* sx, uint32_t off, int j) { return *reinterpret_cast<const uint4*>(sx + (off ^ (j * 64))); };
  // sum x over a step for two rows, 2 t and 2 t + 1 of eight: any order of k will do
  auto sum_of = [&](const uint8_t* sx, uint32_t off) {
    float c[2][4];
    constexpr uint32_t one = I4Num<T>::ones;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 b = x_of(sx, off, j);
      if (j == 0) {
        i4_mma_first<T>(c[0], one, one, one, one, b.x, b.y);
        i4_mma_first<T>(c[1], one, one, one, one, b.z, b.w);
      } else {
        i4_mma<T>(c[0], one, one, one, one, b.x, b.y);
        i4_mma<T>(c[1], one, one, one, one, b.z, b.w);
      }
    }
    return make_float2(c[0][0] + c[1][0], c[0][1] + c[1][1]);
  };

  int at = 0;
  for (int i = 0; i < rounds; ++i) {
    copy_wait<C::STAGES - 2>();
    if constexpr (ALONE) __syncwarp();
    else __syncthreads();
    const uint8_t* stage = smem + at * stage_bytes;
    at = at == C::STAGES - 1 ? 0 : at + 1;
    const uint8_t* words = stage + warp * WB;
    const uint8_t* sx = stage + 8 * WB + wk * x_bytes;
    const int base = s0 + i * C::WK;
    const bool work = base + wk < s1;
    fetch();
    if (work) {
      float sc[4], zp[4];
      i4_load4<TS>(words + 2048 + lane * 4 * sizeof(TS), sc);
      i4_load4<TS>(words + 2048 + (32 + lane) * 4 * sizeof(TS), zp);
      using V = typename I4Num<T>::V;
      V s2[4], o2[4];
      if constexpr (!ALONE) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          s2[k] = I4Num<T>::splat(sc[k]);
          o2[k] = I4Num<T>::splat((8.f - zp[k]) * sc[k]);
        }
      }
      float part[2][4];
      uint4 w = *reinterpret_cast<const uint4*>(words + lane * 16);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint4 b[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) b[n] = x_of(sx, xoff[n], j);
        uint4 next = w;
        if (j < 3) next = *reinterpret_cast<const uint4*>(words + (j + 1) * 512 + lane * 16);
        uint32_t v[4][4];
        i4_expand<T>(w.x, v[0]);
        i4_expand<T>(w.y, v[1]);
        i4_expand<T>(w.z, v[2]);
        i4_expand<T>(w.w, v[3]);
        if constexpr (!ALONE) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const V r = __hfma2(*reinterpret_cast<V*>(&v[k][q]), s2[k], o2[k]);
              v[k][q] = *reinterpret_cast<const uint32_t*>(&r);
            }
        }
        w = next;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const uint32_t b0 = __byte_perm(b[n].x, b[n].z, 0x5410), b1 = __byte_perm(b[n].x, b[n].z, 0x7632);
          const uint32_t b2 = __byte_perm(b[n].y, b[n].w, 0x5410), b3 = __byte_perm(b[n].y, b[n].w, 0x7632);
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            float(&c)[4] = ALONE ? part[a] : acc[a][n];
            if (ALONE && j == 0) i4_mma_first<T>(c, v[2 * a][0], v[2 * a + 1][0], v[2 * a][1], v[2 * a + 1][1], b0, b1);
            else i4_mma<T>(c, v[2 * a][0], v[2 * a + 1][0], v[2 * a][1], v[2 * a + 1][1], b0, b1);
          }
#pragma unroll
          for (int a = 0; a < 2; ++a) i4_mma<T>(ALONE ? part[a] : acc[a][n], v[2 * a][2], v[2 * a + 1][2], v[2 * a][3], v[2 * a + 1][3], b2, b3);
        }
      }
      if constexpr (ALONE) {
        const float2 xs = sum_of(sx, xoff[0]);
        // x - x is zero for a finite number only
        if (__any_sync(0xffffffffu, !((xs.x - xs.x) + (xs.y - xs.y) == 0.f))) {
#pragma unroll
          for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const int k = 2 * a + (c >> 1);
              acc[a][0][c] += i4_plain<T>(words + g * 64, sx, min(2 * t + (c & 1), p.M - 1), k, sc[k], zp[k]);
            }
        } else {
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            const float z0 = 8.f - zp[2 * a], z1 = 8.f - zp[2 * a + 1];
            acc[a][0][0] = fmaf(sc[2 * a], fmaf(z0, xs.x, part[a][0]), acc[a][0][0]);
            acc[a][0][1] = fmaf(sc[2 * a], fmaf(z0, xs.y, part[a][1]), acc[a][0][1]);
            acc[a][0][2] = fmaf(sc[2 * a + 1], fmaf(z1, xs.x, part[a][2]), acc[a][0][2]);
            acc[a][0][3] = fmaf(sc[2 * a + 1], fmaf(z1, xs.y, part[a][3]), acc[a][0][3]);
          }
        }
      }
    }
  }

  // ---- sums of the warps, then of the cluster ----
  copy_wait<0>();
  __syncthreads();
  float* red = reinterpret_cast<float*>(smem);          // [WK][ROWS][COLS]
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      float* r = red + (wk * ROWS + n * 8 + 2 * t) * C::COLS + wn * 32 + 4 * g + 2 * a;
      *reinterpret_cast<float2*>(r) = make_float2(acc[a][n][0], acc[a][n][2]);
      *reinterpret_cast<float2*>(r + C::COLS) = make_float2(acc[a][n][1], acc[a][n][3]);
    }
  __syncthreads();
  constexpr int Q = C::COLS / 4;
  const int total = p.M * Q;
  auto local = [&](int e) {
    float4 v = *reinterpret_cast<const float4*>(red + e * 4);
#pragma unroll
    for (int w = 1; w < C::WK; ++w) {
      const float4 o = *reinterpret_cast<const float4*>(red + w * ROWS * C::COLS + e * 4);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    return v;
  };
  auto store = [&](int e, float4 v) {
    const int m = e / Q, n = n0 + (e - m * Q) * 4;
    if (n >= p.N) return;
    if (p.bias) {
      const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const T*>(p.bias) + n);
      const float2 b0 = unpack2<T>(u.x), b1 = unpack2<T>(u.y);
      v.x += b0.x; v.y += b0.y; v.z += b1.x; v.w += b1.y;
    }
    const long long at = (long long)m * p.N + n;
    if (p.residual) {
      const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const T*>(p.residual) + at);
      const float2 b0 = unpack2<T>(u.x), b1 = unpack2<T>(u.y);
      v.x += b0.x; v.y += b0.y; v.z += b1.x; v.w += b1.y;
    }
    *reinterpret_cast<uint2*>(static_cast<T*>(p.y) + at) = make_uint2(pack2<T>(v.x, v.y), pack2<T>(v.z, v.w));
  };
  const int ranks = gridDim.y;
  if (ranks == 1) {
    for (int e = threadIdx.x; e < total; e += C::THREADS) store(e, local(e));
    return;
  }
  for (int e = threadIdx.x; e < total; e += C::THREADS) *reinterpret_cast<float4*>(red + e * 4) = local(e);
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int e = blockIdx.y * C::THREADS + threadIdx.x; e < total; e += ranks * C::THREADS) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < ranks; ++r) {
      const float4 o = *reinterpret_cast<const float4*>(cluster.map_shared_rank(red, r) + e * 4);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    store(e, v);
  }
  cluster.sync();                  // no CTA leaves while others read its sums
}

template <typename T, typename TS, class C>
int launch_int4_rows(I4Params p, int split, cudaStream_t st) {
  constexpr int ROWS = C::NT * 8;
  const int tiles = (p.N + C::COLS - 1) / C::COLS;
  const int red = 8 * 32 * ROWS * 4;
  const int smem = max(C::STAGES * (8 * i4_words_bytes<TS>() + C::WK * p.M * 256), red);
  if (smem > 227 * 1024) return 51;
  const int ctas = (smem + 1024) * C::CTAS <= 228 * 1024 ? C::CTAS : 1;
  // An SM's rounds, one CTA's after the other's, and what starting and finishing a wave of CTAs takes (about three rounds).  Clusters
  // of three or five to seven do not fill the chip's groups of SMs: 21.8 us with three against 16.9 with four (48 rows, 4096 x 4096).
  int least = 1 << 30, best = 0;
  for (int s = 1; s <= 8; ++s) {
    const int slice = (p.steps + s - 1) / s, sms = rbh::sm_count();
    if (split > 0 ? s != split : (s & (s - 1)) != 0 || (s - 1) * slice >= p.steps) continue;
    const int cost = (tiles * s + sms - 1) / sms * ((slice + C::WK - 1) / C::WK) + (tiles * s + sms * ctas - 1) / (sms * ctas) * 3;
    if (cost < least) { least = cost; best = s; p.slice = slice; }
  }
  if (best == 0) return 51;
  auto kern = int4_rows_kernel<T, TS, C>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return 2000 + (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles, best);
  cfg.blockDim = dim3(C::THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {1, (unsigned)best, 1};
  cfg.attrs = at;
  cfg.numAttrs = best > 1 ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kern, p);
  return e == cudaSuccess ? 0 : 3000 + (int)e;
}

}  // namespace rb

extern "C" {

// 51: sizes or alignment that this kernel does not cover.  split: CTAs that share K (0: by the rule above).
int rb_int4_rows(int x_dtype, int scale_dtype, const void* x, const int* packed, const void* scales, const void* zps,
                 const void* bias, const void* residual, void* y, int M, int N, int K, int Kp, int group, int split, void* stream) {
  using namespace rb;
  if (M <= 0 || N <= 0) return 0;
  if (M > 48 || split < 0 || split > 8) return 51;
  if (group % I4_GROUP || Kp % group || K > Kp || K <= 0 || K % 8 || N % 4) return 51;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(packed) | reinterpret_cast<uintptr_t>(scales) |
       reinterpret_cast<uintptr_t>(zps)) & 15) return 51;
  if ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(residual)) & 7) return 51;
  I4Params p;
  p.x = x; p.packed = packed; p.scales = scales; p.zps = zps; p.bias = bias; p.residual = residual; p.y = y;
  p.M = M; p.N = N; p.K = K; p.steps = Kp / I4_GROUP; p.steps_per_group = group / I4_GROUP;
  p.slice = 0;
  if (split > p.steps) return 51;
  cudaStream_t st = (cudaStream_t)stream;
#define RB_I4(T, TS)                                                              \
  do {                                                                            \
    if (M <= 8) return launch_int4_rows<T, TS, I4Cfg<1>>(p, split, st);           \
    if (M <= 16) return launch_int4_rows<T, TS, I4Cfg<2>>(p, split, st);          \
    if (M <= 24) return launch_int4_rows<T, TS, I4Cfg<3>>(p, split, st);          \
    if (M <= 32) return launch_int4_rows<T, TS, I4Cfg<4>>(p, split, st);          \
    return launch_int4_rows<T, TS, I4Cfg<6>>(p, split, st);                       \
  } while (0)
  if (x_dtype == rbh::DT_BF16 && scale_dtype == rbh::DT_F16) RB_I4(__nv_bfloat16, __half);
  if (x_dtype == rbh::DT_BF16 && scale_dtype == rbh::DT_F32) RB_I4(__nv_bfloat16, float);
  if (x_dtype == rbh::DT_F16 && scale_dtype == rbh::DT_F16) RB_I4(__half, __half);
  if (x_dtype == rbh::DT_F16 && scale_dtype == rbh::DT_F32) RB_I4(__half, float);
#undef RB_I4
  return 51;
}
}
