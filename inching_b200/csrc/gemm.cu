// Dense layers of the warm-start network: C = A B (+ beta C) in FP32 with arbitrary
// element strides, so the same call serves X W, X^T dY (weight gradients, a reduction
// over the long dimension) and dY W^T.
//
// FP32 FMAs bound the layers (2 * 132 * 128 flops for 1 KB of an edge's row), so the
// main kernel is a register-tiled one: 128 x 128 outputs a block, 8 x 8 a thread as
// packed f32x2 FMAs, 16 steps of K staged at a time through registers into the other
// of two shared buffers.  Up to K = 2,048 every output sums its terms in the order of K
// with one rounding a term, whatever the tile, so the choice of kernel does not change
// the bits (beyond it K may be split, and the skinny kernel sums 8 interleaved parts of
// K).  Forward and backward pass on the bead graph of the 100k-atom assembly:
// 16.8 ms with 64 x 64 tiles of 4 x 4 outputs a thread, staged element by element, for
// every product (14.5 ms of it in them), 5.7 ms with these kernels (3.4 ms).
//
// Few outputs over a long K (weight gradients, bias gradients) split K over blocks;
// the parts are added in a fixed order, so the result does not depend on timing.  A
// product with at most 8 rows (or columns) reads its long operand once and has its own
// kernel: in a 128-row tile 15/16 of the FMAs would be on padding.
#include <algorithm>

#include "common.cuh"

namespace inch {

thread_local int last_launches = 0;  // of the calling thread's last product or order

namespace {

constexpr int kBN = 128, kBK = 16;
constexpr int kSkinny = 8;           // most rows of the skinny kernel
// K beyond which K is split and few rows or columns are skinny.  Splitting would pay below it
// too (48 x 48: K = 2,048 unsplit 124 us, K = 2,049 split 17), but up to the line
// a sum keeps the order of K, and its bits.
constexpr int kLongK = 2048;

struct Gemm {
  int M, N, K;
  const float* A;
  int64_t sai, sak;
  const float* B;
  int64_t sbk, sbn;
  float* C;
  int64_t ldc;
  float beta;
  int kchunk;
  float* part;
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// AK / BN: the unit stride of A is along K / that of B along N (else the other one).
// Both row strides are multiples of 4 and both bases 16-byte aligned; the extent along
// a unit stride is a multiple of 4, so a float4 never crosses it.
template <int BM, bool AK, bool BN>
__global__ void __launch_bounds__(256, 2) k_gemm_tile(Gemm g) {
  constexpr int TM = BM / 16;        // rows of a thread
  constexpr int AV = BM / 64;        // float4 of A a thread stages
  __shared__ __align__(16) float As[2][kBK][BM + 4];
  __shared__ __align__(16) float Bs[2][kBK][kBN + 4];
  const int t = threadIdx.x;
  // a warp covers 4 x 8 threads, so that its fragment loads touch 64 and 128 bytes
  const int tx = (t & 7) | ((t >> 2) & 8), ty = ((t >> 3) & 3) | ((t >> 6) << 2);
  const int bm = blockIdx.x * BM, bn = blockIdx.y * kBN;
  const int k_beg = blockIdx.z * g.kchunk;
  const int k_end = g.K - k_beg < g.kchunk ? g.K : k_beg + g.kchunk;
  float4 ra[AV], rb[2];
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < AV; ++i) {
      const int s = t + i * 256;
      const int m = bm + (AK ? s >> 2 : (s % (BM / 4)) * 4), k = k0 + (AK ? (s & 3) * 4 : s / (BM / 4));
      ra[i] = m < g.M && k < k_end ? ld4(g.A + (AK ? m * g.sai + k : k * g.sak + m)) : zero;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int s = t + i * 256;
      const int n = bn + (BN ? (s & 31) * 4 : s >> 2), k = k0 + (BN ? s >> 5 : (s & 3) * 4);
      rb[i] = n < g.N && k < k_end ? ld4(g.B + (BN ? k * g.sbk + n : n * g.sbn + k)) : zero;
    }
  };
  auto stage = [&](int b) {
#pragma unroll
    for (int i = 0; i < AV; ++i) {
      const int s = t + i * 256;
      if constexpr (AK) {
        const int m = s >> 2, k = (s & 3) * 4;
        As[b][k][m] = ra[i].x;
        As[b][k + 1][m] = ra[i].y;
        As[b][k + 2][m] = ra[i].z;
        As[b][k + 3][m] = ra[i].w;
      } else {
        *reinterpret_cast<float4*>(&As[b][s / (BM / 4)][(s % (BM / 4)) * 4]) = ra[i];
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int s = t + i * 256;
      if constexpr (BN) {
        *reinterpret_cast<float4*>(&Bs[b][s >> 5][(s & 31) * 4]) = rb[i];
      } else {
        const int n = s >> 2, k = (s & 3) * 4;
        Bs[b][k][n] = rb[i].x;
        Bs[b][k + 1][n] = rb[i].y;
        Bs[b][k + 2][n] = rb[i].z;
        Bs[b][k + 3][n] = rb[i].w;
      }
    }
  };
  float2 acc[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  auto step = [&](int b, int kk) {
    float a[TM];
#pragma unroll
    for (int h = 0; h < TM / 4; ++h) {
      const float4 v = *reinterpret_cast<const float4*>(&As[b][kk][h * 64 + ty * 4]);
      a[4 * h] = v.x;
      a[4 * h + 1] = v.y;
      a[4 * h + 2] = v.z;
      a[4 * h + 3] = v.w;
    }
    const float4 b0 = *reinterpret_cast<const float4*>(&Bs[b][kk][tx * 4]);
    const float4 b1 = *reinterpret_cast<const float4*>(&Bs[b][kk][64 + tx * 4]);
    const float2 bp[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y),
                          make_float2(b1.z, b1.w)};
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const float2 ai = make_float2(a[i], a[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(ai, bp[j], acc[i][j]);
    }
  };
  fetch(k_beg);
  stage(0);
  __syncthreads();
  int b = 0;
  for (int k0 = k_beg; k0 < k_end; k0 += kBK, b ^= 1) {
    const bool more = k0 + kBK < k_end;
    if (more) fetch(k0 + kBK);
    if (k_end - k0 >= kBK) {
#pragma unroll
      for (int kk = 0; kk < kBK; ++kk) step(b, kk);
    } else {
      for (int kk = 0; kk < k_end - k0; ++kk) step(b, kk);
    }
    if (more) {
      stage(b ^ 1);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = bm + (i / 4) * 64 + ty * 4 + (i & 3);
    if (m >= g.M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = bn + (j / 2) * 64 + tx * 4 + (j & 1) * 2;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (n + c >= g.N) continue;
        const float v = c ? acc[i][j].y : acc[i][j].x;
        if (g.part != nullptr) {
          g.part[((int64_t)blockIdx.z * g.M + m) * g.N + n + c] = v;
        } else {
          float* cp = g.C + m * g.ldc + n + c;
          *cp = g.beta != 0.f ? fmaf(g.beta, *cp, v) : v;
        }
      }
    }
  }
}

// Any strides: 64 x 64 tiles staged element by element.  A chunk's eight loads a thread
// bound it on few tiles (12 x 12 over K = 1,000: 107 us as loops, one load after another;
// 55 unrolled, all in flight).
constexpr int kGM = 64, kGN = 64;
__global__ void __launch_bounds__(256) k_gemm_any(Gemm g) {
  __shared__ float As[kBK][kGM + 4];
  __shared__ float Bs[kBK][kGN + 4];
  const int bm = blockIdx.y * kGM, bn = blockIdx.x * kGN;
  const int k_beg = blockIdx.z * g.kchunk;
  const int k_end = g.K - k_beg < g.kchunk ? g.K : k_beg + g.kchunk;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
  for (int k0 = k_beg; k0 < k_end; k0 += kBK) {
    // consecutive threads along whichever index is unit-stride
#pragma unroll
    for (int i = 0; i < kGM * kBK / 256; ++i) {
      const int t = threadIdx.x + i * 256;
      const int mm = g.sak == 1 ? t / kBK : t % kGM, kk = g.sak == 1 ? t % kBK : t / kGM;
      const int gi = bm + mm, gk = k0 + kk;
      As[kk][mm] = gi < g.M && gk < k_end ? g.A[gi * g.sai + gk * g.sak] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kGN * kBK / 256; ++i) {
      const int t = threadIdx.x + i * 256;
      const int nn = g.sbn == 1 ? t % kGN : t / kBK, kk = g.sbn == 1 ? t / kGN : t % kBK;
      const int gj = bn + nn, gk = k0 + kk;
      Bs[kk][nn] = gj < g.N && gk < k_end ? g.B[gk * g.sbk + gj * g.sbn] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kBK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) a[r] = As[kk][ty * 4 + r];
#pragma unroll
      for (int c = 0; c < 4; ++c) b[c] = Bs[kk][tx * 4 + c];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a[r], b[c], acc[r][c]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = bm + ty * 4 + r;
    if (i >= g.M) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = bn + tx * 4 + c;
      if (j >= g.N) continue;
      if (g.part != nullptr) {
        g.part[((int64_t)blockIdx.z * g.M + i) * g.N + j] = acc[r][c];
      } else {
        float* cp = g.C + i * g.ldc + j;
        *cp = g.beta != 0.f ? fmaf(g.beta, *cp, acc[r][c]) : acc[r][c];
      }
    }
  }
}

// Skinny products, part[z][m][n] = sum over block z's K of S[m][k] L[k][n], m < M <= 8:
// 8 threads deep in K and 128 columns wide, float4 a thread where the rows of L allow it
// (V = 4), else one column a thread (V = 1, 32 columns).
template <int V>
__global__ void __launch_bounds__(256)
k_gemm_skinny(int M, int N, int K, const float* __restrict__ S, int64_t sm, int64_t sk, const float* __restrict__ L,
              int64_t ldl, int kchunk, float* __restrict__ part) {
  __shared__ float red[8][32 * V];
  const int cx = threadIdx.x & 31, kz = threadIdx.x >> 5;
  const int n = (blockIdx.x * 32 + cx) * V;
  const int k_beg = blockIdx.z * kchunk;
  const int k_end = K - k_beg < kchunk ? K : k_beg + kchunk;
  float acc[kSkinny][V];
#pragma unroll
  for (int m = 0; m < kSkinny; ++m)
#pragma unroll
    for (int v = 0; v < V; ++v) acc[m][v] = 0.f;
  if (n < N) {
#pragma unroll 4
    for (int k = k_beg + kz; k < k_end; k += 8) {
      float l[V];
      if constexpr (V == 4) {
        const float4 x = ld4(L + k * ldl + n);
        l[0] = x.x;
        l[1] = x.y;
        l[2] = x.z;
        l[3] = x.w;
      } else {
        l[0] = __ldg(L + k * ldl + n);
      }
#pragma unroll
      for (int m = 0; m < kSkinny; ++m) {
        if (m >= M) break;
        const float s = __ldg(S + m * sm + k * sk);
#pragma unroll
        for (int v = 0; v < V; ++v) acc[m][v] = fmaf(s, l[v], acc[m][v]);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < kSkinny; ++m) {
    if (m >= M) break;
    __syncthreads();
#pragma unroll
    for (int v = 0; v < V; ++v) red[kz][cx * V + v] = acc[m][v];
    __syncthreads();
    for (int c = threadIdx.x; c < 32 * V; c += 256) {
      const int col = blockIdx.x * 32 * V + c;
      if (col >= N) continue;
      float s = 0.f;
#pragma unroll
      for (int z = 0; z < 8; ++z) s += red[z][c];
      part[((int64_t)blockIdx.z * M + m) * N + col] = s;
    }
  }
}

// One output column: a thread walks its row, in the order of K.
__global__ void __launch_bounds__(128) k_gemv(Gemm g, bool vec) {
  for (int64_t m = blockIdx.x * 128ll + threadIdx.x; m < g.M; m += gridDim.x * 128ll) {
    const float* a = g.A + m * g.sai;
    float acc = 0.f;
    if (vec) {
#pragma unroll 8
      for (int k = 0; k < g.K; k += 4) {
        const float4 v = ld4(a + k);
        acc = fmaf(v.x, __ldg(g.B + k * g.sbk), acc);
        acc = fmaf(v.y, __ldg(g.B + (k + 1) * g.sbk), acc);
        acc = fmaf(v.z, __ldg(g.B + (k + 2) * g.sbk), acc);
        acc = fmaf(v.w, __ldg(g.B + (k + 3) * g.sbk), acc);
      }
    } else {
      for (int k = 0; k < g.K; ++k) acc = fmaf(__ldg(a + k * g.sak), __ldg(g.B + k * g.sbk), acc);
    }
    float* cp = g.C + m * g.ldc;
    *cp = g.beta != 0.f ? fmaf(g.beta, *cp, acc) : acc;
  }
}

// C[i * sci + j * scj] = sum over the parts (+ beta C): 8 threads an output, each over
// every 8th part, added in a fixed order.
__global__ void __launch_bounds__(256)
k_gemm_reduce(int M, int N, int splits, const float* __restrict__ part, float* C, int64_t sci, int64_t scj,
              float beta) {
  __shared__ float s[8][33];
  const int64_t total = (int64_t)M * N;
  const int o = threadIdx.x & 31, z = threadIdx.x >> 5;
  for (int64_t t0 = blockIdx.x * 32ll; t0 < total; t0 += gridDim.x * 32ll) {
    const int64_t t = t0 + o;
    float sum = 0.f;
    if (t < total)
#pragma unroll 4
      for (int p = z; p < splits; p += 8) sum += part[p * total + t];
    __syncthreads();
    s[z][o] = sum;
    __syncthreads();
    if (z == 0 && t < total) {
#pragma unroll
      for (int q = 1; q < 8; ++q) sum += s[q][o];
      float* cp = C + (t / N) * sci + (t % N) * scj;
      *cp = beta != 0.f ? fmaf(beta, *cp, sum) : sum;
    }
  }
}

constexpr int kGridY = 65535;        // a grid's second dimension

int cdiv(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// K splits of a product with `tiles` output tiles: two blocks an SM, at least 256 steps
// of K each; none where the output fills the SMs or K is short.
int splits_for(int64_t tiles, int K) {
  if (tiles >= 148 || K <= kLongK) return 1;
  int sp = cdiv(2 * 148, tiles);
  const int by_k = cdiv(K, 256);
  if (sp > by_k) sp = by_k;
  return sp < 1 ? 1 : sp;
}

// The largest count of splits of any kernel that may take the product (the workspace
// query knows the sizes only).
int most_splits(int M, int N, int K) {
  const int tall = splits_for((int64_t)cdiv(M, 128) * cdiv(N, kBN), K);
  const int any = splits_for((int64_t)cdiv(M, kGM) * cdiv(N, kGN), K);
  int sp = tall > any ? tall : any;
  if (M <= kSkinny || N <= kSkinny) {
    const int skinny = splits_for(cdiv(M <= kSkinny ? N : M, 32), K);
    sp = skinny > sp ? skinny : sp;
  }
  return sp;
}

template <int V>
cudaError_t skinny(int M, int N, int K, const float* S, int64_t sm, int64_t sk, const float* L, int64_t ldl, float* C,
                   int64_t sci, int64_t scj, float beta, int splits, float* part, cudaStream_t s) {
  const int kchunk = cdiv(K, splits);
  const int zs = cdiv(K, kchunk);
  k_gemm_skinny<V><<<dim3(cdiv(N, 32 * V), 1, zs), 256, 0, s>>>(M, N, K, S, sm, sk, L, ldl, kchunk, part);
  k_gemm_reduce<<<grid_for((int64_t)M * N, 32, 148 * 8), 256, 0, s>>>(M, N, zs, part, C, sci, scj, beta);
  return cudaGetLastError();
}

}  // namespace
}  // namespace inch

using namespace inch;

extern "C" int32_t inch_last_launches(void) { return last_launches; }

extern "C" size_t inch_mp_gemm_workspace_size(int32_t M, int32_t N, int32_t K) {
  if (M < 1 || N < 1 || K < 1) return 256;
  const int sp = most_splits(M, N, K);
  // the skinny kernel leaves its one part in the workspace too
  const bool narrow = (M <= kSkinny || N <= kSkinny) && K > kLongK;
  size_t need = sp > 1 || narrow ? (size_t)sp * M * N * sizeof(float) + 256 : 256;
  if (M > 128 && M % 128 != 0 && M % 128 <= kSkinny) {     // whole tiles and the rest apart
    const size_t whole = inch_mp_gemm_workspace_size(M / 128 * 128, N, K);
    const size_t rest = inch_mp_gemm_workspace_size(M % 128, N, K);
    need = whole > need ? whole : need;
    need = rest > need ? rest : need;
  }
  return need;
}

extern "C" inch_status inch_mp_gemm(int32_t M, int32_t N, int32_t K, const float* A, int64_t sai, int64_t sak,
                                    const float* B, int64_t sbk, int64_t sbn, float* C, int64_t ldc, float beta,
                                    void* ws, size_t ws_bytes, cudaStream_t s) {
  INCH_REQUIRE(A && B && C && M >= 1 && N >= 1 && K >= 1 && ldc >= N, INCH_INVALID_ARG, "inch_mp_gemm: bad args");
  INCH_REQUIRE(most_splits(M, N, K) == 1 || (ws != nullptr && ws_bytes >= inch_mp_gemm_workspace_size(M, N, K)),
               INCH_OOM, "inch_mp_gemm: workspace of %zu bytes, need %zu", ws_bytes,
               inch_mp_gemm_workspace_size(M, N, K));
  float* part = ws != nullptr && ws_bytes >= inch_mp_gemm_workspace_size(M, N, K) ? static_cast<float*>(ws) : nullptr;
  const auto al16 = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  // skinny products over a long K: the long operand's unit stride lies along the output
  const bool few_rows = M <= kSkinny && sbn == 1 && K > kLongK;
  const bool few_cols = N <= kSkinny && sai == 1 && K > kLongK && !few_rows;
  if ((few_rows || few_cols) && part != nullptr) {
    const int n = few_rows ? N : M;
    const float* L = few_rows ? B : A;
    const int64_t ldl = few_rows ? sbk : sak;
    const bool v4 = n % 4 == 0 && ldl % 4 == 0 && al16(L);
    const int sp = splits_for(cdiv(n, v4 ? 128 : 32), K);
    const auto run = v4 ? skinny<4> : skinny<1>;
    const cudaError_t e = few_rows ? run(M, N, K, A, sai, sak, L, ldl, C, ldc, 1, beta, sp, part, s)
                                   : run(N, M, K, B, sbn, sbk, L, ldl, C, 1, ldc, beta, sp, part, s);
    INCH_REQUIRE(e == cudaSuccess, INCH_CUDA_ERROR, "inch_mp_gemm: %s", cudaGetErrorString(e));
    last_launches = 2;
    return INCH_OK;
  }
  Gemm g{M, N, K, A, sai, sak, B, sbk, sbn, C, ldc, beta, K, nullptr};
  if (N == 1 && K <= kLongK) {
    k_gemv<<<grid_for(M, 128, 148 * 16), 128, 0, s>>>(g, sak == 1 && sai % 4 == 0 && K % 4 == 0 && al16(A));
    INCH_LAUNCH_CHECK();
    last_launches = 1;
    return INCH_OK;
  }
  const bool ak = sak == 1 && sai % 4 == 0 && K % 4 == 0, am = sai == 1 && sak % 4 == 0 && M % 4 == 0;
  const bool bn = sbn == 1 && sbk % 4 == 0 && N % 4 == 0, bk = sbk == 1 && sbn % 4 == 0 && K % 4 == 0;
  // Register tiles pay where K is long enough to hide their prologue and epilogue and the
  // tiles are full.  Where its own tiles fill the SMs the general kernel is faster on a
  // short K (20,000 x 128: K = 4, 7.3 us against 10.2; K = 32, 11.0 both), and up to 64
  // rows or columns on a middling one (20,000 x 16: K = 16, 4.9 and 6.9; K = 256, 36 and
  // 46).  Up to 32 rows stay with the tiles (16 x 100,000, K = 4: 12.1 general, 7.6).
  // Below 16 rows or columns the tiles are mostly padding.
  const int narrow = std::min(M, N);
  const bool shallow = M > 32 && (int64_t)cdiv(M, kGM) * cdiv(N, kGN) >= 200 &&
                       (narrow <= 64 ? K <= 256 : (int64_t)K * cdiv(narrow, 64) <= 48);
  const bool fast = (ak || am) && (bn || bk) && al16(A) && al16(B) && narrow >= 16 && !shallow;
  // a few rows beyond whole tiles over a long K (132 = 128 + 4 features by the edges) go
  // to the skinny kernel instead of a second, nearly empty tile
  if (fast && am && bn && K > kLongK && M > 128 && M % 128 != 0 && M % 128 <= kSkinny && part != nullptr) {
    const int M0 = M / 128 * 128;
    inch_status st = inch_mp_gemm(M0, N, K, A, sai, sak, B, sbk, sbn, C, ldc, beta, ws, ws_bytes, s);
    if (st != INCH_OK) return st;
    const int whole = last_launches;
    st = inch_mp_gemm(M - M0, N, K, A + M0, sai, sak, B, sbk, sbn, C + M0 * ldc, ldc, beta, ws, ws_bytes, s);
    last_launches += whole;
    return st;
  }
  // 128-row tiles where they fill the SMs or K is split anyway, else 64-row ones; these too
  // where half of a 128 x 128 tile would be padding (20,000 x 16 over K = 1,000: 185 us
  // with 128 rows, 166 with 64)
  const bool tall = K > kLongK || (narrow > 64 && (int64_t)cdiv(M, 128) * cdiv(N, kBN) >= 148);
  const int bm = fast ? (tall ? 128 : 64) : kGM;
  const int mt = cdiv(M, bm), nt = cdiv(N, fast ? kBN : kGN);
  const int sp = splits_for((int64_t)mt * nt, K);
  if (sp > 1) {
    g.kchunk = cdiv(cdiv(K, sp), kBK) * kBK;
    g.part = part;
  }
  const int zs = cdiv(K, g.kchunk);
  // The general kernel walks the column tiles of a row of tiles first, the register tiles
  // the rows of a column of tiles (20,000 x 129 over K = 2,052 through the general kernel:
  // 1,165 us with the rows first, 1,008 the columns, as an A of 164 MB is read once; with
  // the staging loads issued together 658).  The other direction is a grid's second
  // dimension, so more tiles than that holds go in several launches (never of a split
  // product).
  last_launches = 0;
  const int across = fast ? kGridY * kBN : kGridY * kGM;
  for (int64_t at = 0; at < (fast ? N : M); at += across) {
    Gemm h = g;
    if (fast) {
      h.N = std::min<int64_t>(N - at, across);
      h.B += at * sbn;
      h.C += at;
    } else {
      h.M = std::min<int64_t>(M - at, across);
      h.A += at * sai;
      h.C += at * ldc;
    }
    const dim3 grid(fast ? mt : nt, cdiv(fast ? h.N : h.M, fast ? kBN : kGM), zs);
#define TILE(BMV, AKV, BNV) k_gemm_tile<BMV, AKV, BNV><<<grid, 256, 0, s>>>(h)
    if (!fast) k_gemm_any<<<grid, 256, 0, s>>>(h);
    else if (bm == 128 && ak && bn) TILE(128, true, true);
    else if (bm == 128 && ak) TILE(128, true, false);
    else if (bm == 128 && bn) TILE(128, false, true);
    else if (bm == 128) TILE(128, false, false);
    else if (ak && bn) TILE(64, true, true);
    else if (ak) TILE(64, true, false);
    else if (bn) TILE(64, false, true);
    else TILE(64, false, false);
#undef TILE
    INCH_LAUNCH_CHECK();
    ++last_launches;
  }
  if (g.part != nullptr) {
    k_gemm_reduce<<<grid_for((int64_t)M * N, 32, 148 * 8), 256, 0, s>>>(M, N, zs, part, C, ldc, 1, beta);
    INCH_LAUNCH_CHECK();
    ++last_launches;
  }
  return INCH_OK;
}
