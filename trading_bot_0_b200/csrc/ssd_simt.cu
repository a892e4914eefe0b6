// Exact-fp32 CUDA-core kernels for the SSD operator: every stage of forward and backward for
// any storage dtype, any chunk <= 256 and ragged sequence tails.  This family is the fp32-mode
// path (1e-4 relative parity) and the building block the sequence-parallel split reuses; the
// bf16 throughput path lives in ssd_tensor.cu.
//
// Four launches forward (cumsum, chunk states + C B^T, scan over chunks, outputs), five backward (six with a gate).
#include <atomic>
#include "common.cuh"
#include "ssd_internal.h"

namespace ssd {
namespace {

// ---------------------------------------------------------------------------------------------
// Contractions.  Every one is cut into 64 x 32 output tiles (TM x TN), 128 threads with 4 x 4 outputs each, K in slabs of 32
// staged in shared memory.  Bound: the shared-memory data path, which hands a warp 128 bytes of registers per cycle whatever
// is broadcast, and latency; the FMA pipes are a third busy.  More outputs per thread ease the first and lose to the second:
// 8 x 4 with 64 threads and 8 x 8 with a warp per tile took 414 and 569 us for a training step of 16 x 1000 tokens, 8 heads of
// 32 x 64, this 348, the 64 x 64 scalar tiles before them 876.  What pays is keeping everything else out of the way: operands
// are read in 16-byte pieces in the layout they have in memory (k-contiguous or m/n-contiguous, three forms of the inner loop)
// with the next slab's loads in flight during the arithmetic, products go through the packed fma.rn.f32x2 (same rounding, half
// the issue slots), and decays ride on whole rows (`exp(cs_i - cs_j) = exp(cs_i - cs_r) exp(cs_r - cs_j)` with r at the edge of
// the output tile, both exponents <= 0) so that only a tile on the diagonal evaluates an exponential per element.  32 columns
// fit a head of 32 features.
constexpr int ST = 256;   // threads of the kernels without a contraction
constexpr int TM = 64, TN = 32, KC = 32, NT = 128;
constexpr int PA = TM + 4, PB = TN + 4;   // row pitch of the m- and n-contiguous slabs
constexpr int A_FLOATS = (TM * KC > KC * PA) ? TM * KC : KC * PA, B_FLOATS = (TN * KC > KC * PB) ? TN * KC : KC * PB;

// A row-major block in global memory: `rows` rows of `cols` valid elements, `sl` elements apart.
template <typename T> struct Mat {
  const T* p;
  long long sl;
  int rows, cols;
  bool vec;   // 4-element pieces are aligned
  __device__ __forceinline__ Mat(const T* p_, long long sl_, int rows_, int cols_)
      : p(p_), sl(sl_), rows(rows_), cols(cols_), vec(((uintptr_t)p_ % (4 * sizeof(T))) == 0 && (sl_ % 4) == 0) {}
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
  const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
  return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
}
__device__ __forceinline__ float4 scale4(float4 v, float f) { return make_float4(v.x * f, v.y * f, v.z * f, v.w * f); }
// The piece at (r, c .. c + 3), zero outside the matrix's valid part.
template <typename T> __device__ __forceinline__ float4 piece(const Mat<T>& m, int r, int c) {
  float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
  if (r < m.rows && c < m.cols) {
    const T* p = m.p + r * m.sl + c;
    if (m.vec && c + 3 < m.cols) t = ld4(p);
    else {
      t.x = ldf(p);
      if (c + 1 < m.cols) t.y = ldf(p + 1);
      if (c + 2 < m.cols) t.z = ldf(p + 2);
      if (c + 3 < m.cols) t.w = ldf(p + 3);
    }
  }
  return t;
}

// ROWS x COLS elements of a matrix in the registers of the block.
template <int ROWS, int COLS> struct Slab {
  static constexpr int V = ROWS * COLS / 4 / NT, Q4 = COLS / 4;
  float4 v[V];
  template <typename T> __device__ __forceinline__ void load(const Mat<T>& m, int r0, int c0) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int e = threadIdx.x + i * NT;
      v[i] = piece(m, r0 + e / Q4, c0 + (e % Q4) * 4);
    }
  }
  // f(r, c, x): what element (r, c .. c + 3) of the slab becomes.  k-contiguous slabs keep their rows 32 floats apart with the
  // 16-byte pieces swizzled by the row's group of four, so that threads reading one k of neighbouring row groups hit
  // different banks.
  template <class F> __device__ __forceinline__ void store_k(float* s, F f) const {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int e = threadIdx.x + i * NT, r = e / Q4, q = e % Q4;
      *reinterpret_cast<float4*>(s + r * KC + ((q ^ (r >> 2)) & 7) * 4) = f(r, q * 4, v[i]);
    }
  }
  template <int PITCH, class F> __device__ __forceinline__ void store_r(float* s, F f) const {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int e = threadIdx.x + i * NT, r = e / Q4, q = e % Q4;
      *reinterpret_cast<float4*>(s + r * PITCH + q * 4) = f(r, q * 4, v[i]);
    }
  }
};
struct Same { __device__ __forceinline__ float4 operator()(int, int, float4 v) const { return v; } };

// Accumulators of a thread: rows 4 ty + r, columns 4 tx + c (tx = thread % 8, ty = thread / 8).  `n` holds column pairs, `k`
// even / odd k sums (both operands k-contiguous); the value is their sum.
struct Acc {
  f32x2 n[4][2], k[4][4];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      n[r][0] = n[r][1] = 0ull;
#pragma unroll
      for (int c = 0; c < 4; ++c) k[r][c] = 0ull;
    }
  }
  __device__ __forceinline__ void get(float (&o)[4][4]) const {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      unpack2(n[r][0], o[r][0], o[r][1]);
      unpack2(n[r][1], o[r][2], o[r][3]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float a, b;
        unpack2(k[r][c], a, b);
        o[r][c] += a + b;
      }
    }
  }
  __device__ __forceinline__ void scale(const float (&f)[4]) {   // row r times f[r]
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const f32x2 d = pack2(f[r], f[r]);
      n[r][0] = fma2(n[r][0], d, 0ull);
      n[r][1] = fma2(n[r][1], d, 0ull);
#pragma unroll
      for (int c = 0; c < 4; ++c) k[r][c] = fma2(k[r][c], d, 0ull);
    }
  }
};

template <bool A_K, bool B_K> __device__ __forceinline__ void mac(Acc& acc, const float* As, const float* Bs) {
  static_assert(!B_K || A_K, "an m-contiguous A goes with an n-contiguous B");
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
#pragma unroll
  for (int q = 0; q < KC / 4; ++q) {
    if constexpr (A_K && B_K) {
      ulonglong2 a[4], b[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        a[r] = *reinterpret_cast<const ulonglong2*>(As + (4 * ty + r) * KC + ((q ^ ty) & 7) * 4);
        b[r] = *reinterpret_cast<const ulonglong2*>(Bs + (4 * tx + r) * KC + ((q ^ tx) & 7) * 4);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc.k[r][c] = fma2(a[r].y, b[c].y, fma2(a[r].x, b[c].x, acc.k[r][c]));
    } else {
      float a[4][4];   // [k][row]
      if constexpr (A_K) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float4 t = *reinterpret_cast<const float4*>(As + (4 * ty + r) * KC + ((q ^ ty) & 7) * 4);
          a[0][r] = t.x; a[1][r] = t.y; a[2][r] = t.z; a[3][r] = t.w;
        }
      } else {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const float4 t = *reinterpret_cast<const float4*>(As + (4 * q + kk) * PA + 4 * ty);
          a[kk][0] = t.x; a[kk][1] = t.y; a[kk][2] = t.z; a[kk][3] = t.w;
        }
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(Bs + (4 * q + kk) * PB + 4 * tx);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const f32x2 d = pack2(a[kk][r], a[kk][r]);
          acc.n[r][0] = fma2(d, b.x, acc.n[r][0]);
          acc.n[r][1] = fma2(d, b.y, acc.n[r][1]);
        }
      }
    }
  }
}

// acc += A B over k in [k0, k1).  A: rows = m if A_K else k; B: rows = n if B_K else k; both start at the tile's first m / n.
// fa, fb: transforms of the staged pieces, called with (the slab's first k, row and first column in the slab, value).
template <bool A_K, bool B_K, typename TA, typename TB, class FA, class FB>
__device__ __forceinline__ void contract(Acc& acc, const Mat<TA>& A, const Mat<TB>& B, int k0, int k1, float* As, float* Bs, FA fa, FB fb) {
  Slab<A_K ? TM : KC, A_K ? KC : TM> a;
  Slab<B_K ? TN : KC, B_K ? KC : TN> b;
  auto load = [&](int k) {
    if (A_K) a.load(A, 0, k); else a.load(A, k, 0);
    if (B_K) b.load(B, 0, k); else b.load(B, k, 0);
  };
  load(k0);
  for (int k = k0; k < k1; k += KC) {
    __syncthreads();   // the previous slab has been read
    auto ga = [&](int r, int c, float4 v) { return fa(k, r, c, v); };
    auto gb = [&](int r, int c, float4 v) { return fb(k, r, c, v); };
    if constexpr (A_K) a.store_k(As, ga); else a.template store_r<PA>(As, ga);
    if constexpr (B_K) b.store_k(Bs, gb); else b.template store_r<PB>(Bs, gb);
    __syncthreads();
    if (k + KC < k1) load(k + KC);
    mac<A_K, B_K>(acc, As, Bs);
  }
}
struct Keep { __device__ __forceinline__ float4 operator()(int, int, int, float4 v) const { return v; } };

// Sum over the 8 threads (tx) that share a tile row; every one of them gets it.
__device__ __forceinline__ float row_reduce(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}


__device__ __forceinline__ size_t cs_idx(const Geo& g, int b, int h, int c) {
  return ((size_t)(b * g.H + h) * g.nc + c) * g.Q;
}
__device__ __forceinline__ size_t st_idx(const Geo& g, int b, int c, int h) {
  return ((size_t)(b * g.nc + c) * g.H + h) * g.P * g.N;
}
__device__ __forceinline__ size_t cb_idx(const Geo& g, int b, int c, int grp) {
  return ((size_t)(b * g.nc + c) * g.G + grp) * g.Q * g.Q;
}

// ---------------------------------------------------------------------------------------------
// Stage 1: cs = inclusive within-chunk cumsum of dt*A (fp32), dtf = dt as fp32, both [B,H,nc,Q]; dt here is the
// step size after the optional bias / softplus, which every later stage reads from dtf or the decay tables.
// One block per (chunk, batch, HG heads), as k_ddt: thread q reads the HG contiguous dt values of position q and the block scans
// them together with warp shuffles.
template <typename T, int HG>
__global__ void __launch_bounds__(256) k_cumsum(Geo g, const T* __restrict__ dt, const float* __restrict__ dt_bias,
                                               const float* __restrict__ A, float* __restrict__ cs,
                                               float* __restrict__ dtf, float* __restrict__ tab, int* __restrict__ hand,
                                               int* __restrict__ status) {
  pdl_wait();
  const int c = blockIdx.x, b = blockIdx.y, q = threadIdx.x;
  __shared__ float wsum[8][HG];
  const int t = c * g.Q + q;
  if (c == 0 && blockIdx.z == 0) {   // first kernel of a pass: the status word, the counters of the state scan
    if (b == 0 && q == 0) *status = 0;
    if (hand)
      for (int i = q, n = g.H * g.P / 128; i < n; i += blockDim.x) hand[b * n + i] = 0;
  }
  const bool live = (q < g.Q) && (t < g.L);
  const int lane = q & 31, w = q >> 5;
  const T* row = dt + b * g.dtsb + (long long)t * g.dtsl;
  for (int h0 = blockIdx.z * HG; h0 < g.H; h0 += HG * gridDim.z) {
    float d[HG], v[HG];
#pragma unroll
    for (int k = 0; k < HG; ++k) {
      const int h = h0 + k;
      d[k] = (live && h < g.H) ? dt_activation(ldf(row + h), dt_bias ? dt_bias[h] : 0.f, g.dt_softplus) : 0.f;
      v[k] = (h < g.H) ? d[k] * A[h] : 0.f;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int k = 0; k < HG; ++k) {
        const float n = __shfl_up_sync(0xffffffffu, v[k], o);
        if (lane >= o) v[k] += n;
      }
    }
    if (lane == 31) {
#pragma unroll
      for (int k = 0; k < HG; ++k) wsum[w][k] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < HG; ++k) {
      float base = 0.f;
      for (int i = 0; i < w; ++i) base += wsum[i][k];
      v[k] += base;
    }
    {
#pragma unroll
      for (int k = 0; k < HG; ++k) {
        const int h = h0 + k;
        if (h < g.H && q < g.Q) {
          const size_t o = cs_idx(g, b, h, c) + q;
          cs[o] = v[k];
          dtf[o] = d[k];
        }
        // tensor-core family (chunk 128 only): the per-head decay table [cs*log2e | dt | exp(cs_r - cs) dt |
        // exp(dt_{l+1} A)], r = last position of the 32-block (lane 31 of this warp)
        const float vend = __shfl_sync(0xffffffffu, v[k], 31);
        if (tab && h < g.H && q < g.Q) {
          const float L2E = 1.4426950408889634f;
          float* t = tab + ((size_t)(b * g.nc + c) * g.H + h) * SSD_TAB_FLOATS + q;
          t[0] = v[k] * L2E;
          t[128] = d[k];
          t[256] = exp2f((vend - v[k]) * L2E) * d[k];
          if (q > 0) t[384 - 1] = expf(d[k] * A[h]);   // section 3, entry l = decay of step l+1
          if (q == 0) t[384 + 127] = 1.f;
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// Decays exp(cs_i - cs_j) of one row i and four columns j .. j + 3 (zero above the diagonal) from one exponential: that of the last
// column, then leftwards by the steps st[c] = exp(dt_{j+c+1} A), restarting at 1 on the diagonal.  No exponent is positive.  Against
// exp(cs_i - cs_j) per element: up to three more rounded factors (a few ulp), but steps carry no rounding of the running sums, whose
// difference loses ulp(cs) - more than those ulp as soon as |cs| exceeds a few units.
// d = i - j.
__device__ __forceinline__ void walk4(float ci, float c3, int d, const float (&st)[3], float (&o)[4]) {
  o[3] = d >= 3 ? expf(ci - c3) : 0.f;
#pragma unroll
  for (int c = 2; c >= 0; --c) o[c] = d == c ? 1.f : o[c + 1] * st[c];
}
// Where a block stands: `u` counts tiles of a (batch, chunk, head) or (batch, chunk, group) entry, fastest first.
struct Place { int tile, x, c, b; };   // x: head or group
__device__ __forceinline__ Place place_of(unsigned u, int tiles, int nx, int nc) {
  Place q;
  q.tile = (int)(u % tiles); u /= tiles;
  q.x = (int)(u % nx); u /= nx;
  q.c = (int)(u % nc);
  q.b = (int)(u / nc);
  return q;
}
__device__ __forceinline__ int valid_rows(const Geo& g, int c) { return min(g.Q, g.L - c * g.Q); }
template <typename T> __device__ __forceinline__ const T* seq_at(const T* p, long long sb, long long sl, int b, int t, long long col) {
  return p + b * sb + t * sl + col;
}
// Four values, at most n of them.
__device__ __forceinline__ void st4(float* p, const float (&v)[4], int n) {
  if (n >= 4 && ((uintptr_t)p & 15) == 0) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); return; }
#pragma unroll
  for (int i = 0; i < 4; ++i) if (i < n) p[i] = v[i];
}
__device__ __forceinline__ void st4(__nv_bfloat16* p, const float (&v)[4], int n) {
  if (n >= 4 && ((uintptr_t)p & 7) == 0) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) if (i < n) stf(p + i, v[i]);
}
template <typename T> __device__ __forceinline__ void get4(const Mat<T>& m, int r, int c, float (&o)[4]) {
  const float4 t = piece(m, r, c);
  o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
}

// Stage 2 (and its backward twin): out[b,c,h,p,n] = sum_l w_l * X[l,h,p] * Y[l,g,n]; m = n, columns = p.
//   MODE 0: w_l = exp(cs_end - cs_l) * dt_l   (chunk_state: X = x, Y = B)
//   MODE 1: w_l = exp(cs_l)                    (local state gradient: X = dy, Y = C)
template <int MODE, typename TX, typename TY>
__device__ __forceinline__ void state_tile(const Geo& g, unsigned u, const TX* X, long long xsb, long long xsl, const TY* Y, long long ysb,
                                           long long ysl, const float* __restrict__ cs, const float* __restrict__ dtf, float* __restrict__ out,
                                           float* As, float* Bs, float* row) {
  const int ntn = (g.N + TM - 1) / TM, ntp = (g.P + TN - 1) / TN;
  const Place q = place_of(u, ntn * ntp, g.H, g.nc);
  const int n0 = (q.tile % ntn) * TM, p0 = (q.tile / ntn) * TN, h = q.x, grp = h / g.hpg, t0 = q.c * g.Q, nv = valid_rows(g, q.c);
  const size_t co = cs_idx(g, q.b, h, q.c);
  const float cs_end = cs[co + g.Q - 1];
  for (int l = threadIdx.x; l < g.Q; l += NT) row[l] = MODE == 0 ? expf(cs_end - cs[co + l]) * dtf[co + l] : expf(cs[co + l]);
  Acc acc;
  acc.zero();
  const Mat<TY> A(seq_at(Y, ysb, ysl, q.b, t0, (long long)grp * g.N + n0), ysl, nv, min(TM, g.N - n0));
  const Mat<TX> B(seq_at(X, xsb, xsl, q.b, t0, (long long)h * g.P + p0), xsl, nv, min(TN, g.P - p0));
  contract<false, false>(acc, A, B, 0, nv, As, Bs, Keep(), [&](int k, int r, int, float4 v) { return scale4(v, k + r < g.Q ? row[k + r] : 0.f); });
  float o[4][4];
  acc.get(o);
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int p = p0 + 4 * tx + c, n = n0 + 4 * ty;
    const float v[4] = {o[0][c], o[1][c], o[2][c], o[3][c]};
    if (p < g.P && n < g.N) st4(out + st_idx(g, q.b, q.c, h) + (size_t)p * g.N + n, v, g.N - n);
  }
}

// Stage 4a: cb[b,c,g,i,j] = C_i . B_j for tiles that reach below the diagonal.  Tiles of a 64-row strip: the 32-column strips
// up to its end.
__device__ __forceinline__ int tri_tiles(int Q) {
  int n = 0;
  for (int i0 = 0; i0 < Q; i0 += TM) n += (min(i0 + TM, Q) + TN - 1) / TN;
  return n;
}
__device__ __forceinline__ void tri_at(int Q, int tile, int& i0, int& j0) {
  i0 = 0;
  for (;; i0 += TM) {
    const int n = (min(i0 + TM, Q) + TN - 1) / TN;
    if (tile < n) break;
    tile -= n;
  }
  j0 = tile * TN;
}
template <typename T>
__device__ __forceinline__ void cb_tile(const Geo& g, unsigned u, const T* Bm, const T* Cm, float* __restrict__ cb, float* As, float* Bs) {
  const Place q = place_of(u, tri_tiles(g.Q), g.G, g.nc);
  int i0, j0;
  tri_at(g.Q, q.tile, i0, j0);
  const int t0 = q.c * g.Q, nv = valid_rows(g, q.c);
  Acc acc;
  acc.zero();
  const Mat<T> A(seq_at(Cm, g.csb, g.csl, q.b, t0 + i0, (long long)q.x * g.N), g.csl, nv - i0, g.N);
  const Mat<T> B(seq_at(Bm, g.bsb, g.bsl, q.b, t0 + j0, (long long)q.x * g.N), g.bsl, nv - j0, g.N);
  contract<true, true>(acc, A, B, 0, g.N, As, Bs, Keep(), Keep());
  float o[4][4];
  acc.get(o);
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3, j = j0 + 4 * tx;
  float* dst = cb + cb_idx(g, q.b, q.c, q.x);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + 4 * ty + r;
    if (i < g.Q && j < g.Q) st4(dst + (size_t)i * g.Q + j, o[r], g.Q - j);
  }
}

// The part of a forward that needs no state from other chunks, one launch: chunk states, then C B^T.
template <typename T>
__global__ void __launch_bounds__(NT, 4) k_local(Geo g, unsigned n_state, const T* __restrict__ x, const T* __restrict__ Bm,
                                                 const T* __restrict__ Cm, const float* __restrict__ cs, const float* __restrict__ dtf,
                                                 float* __restrict__ states, float* __restrict__ cb) {
  pdl_wait();
  __shared__ __align__(16) float As[A_FLOATS], Bs[B_FLOATS], row[256];
  if (blockIdx.x < n_state) state_tile<0>(g, blockIdx.x, x, g.xsb, g.xsl, Bm, g.bsb, g.bsl, cs, dtf, states, As, Bs, row);
  else cb_tile(g, blockIdx.x - n_state, Bm, Cm, cb, As, Bs);
}

// Stage 4b: chunk_scan.  acc[i,p] = sum_{j<=i} cb[i,j] exp(cs_i-cs_j) dt_j x[j,p] + exp(cs_i) sum_n C[i,n] prev[p,n]
//   GATE_BWD false (forward):      y = acc + D x, optional silu gate, store.
//   GATE_BWD true (gated backward): from acc form dz and the pre-gate gradient dyp.
template <typename T, bool GATE_BWD>
__global__ void __launch_bounds__(NT, 4) k_chunk_scan(Geo g, const T* __restrict__ x, const T* __restrict__ Cm, const float* __restrict__ A,
                                                      const float* __restrict__ D, const T* __restrict__ z, const float* __restrict__ cs, const float* __restrict__ dtf,
                                                      const float* __restrict__ cb, const float* __restrict__ prev, T* __restrict__ y,
                                                      const T* __restrict__ dy, float* __restrict__ dyp, T* __restrict__ dz) {
  pdl_wait();
  __shared__ __align__(16) float As[A_FLOATS], Bs[B_FLOATS], css[256], dts[256], fj[256], stp[256];
  const int nti = (g.Q + TM - 1) / TM, ntp = (g.P + TN - 1) / TN;
  const Place q = place_of(blockIdx.x, nti * ntp, g.H, g.nc);
  // the last strip of a chunk has the most work: it starts first
  const int i0 = (nti - 1 - q.tile % nti) * TM, p0 = (q.tile / nti) * TN, h = q.x, grp = h / g.hpg, t0 = q.c * g.Q, nv = valid_rows(g, q.c);
  if (i0 >= nv) return;
  const size_t co = cs_idx(g, q.b, h, q.c);
  const float ref = cs[co + i0], eref = expf(ref);
  for (int l = threadIdx.x; l < g.Q; l += NT) {
    const float c = cs[co + l], d = dtf[co + l];
    css[l] = c;
    dts[l] = d;
    if (l < i0) fj[l] = expf(ref - c) * d;
    stp[l] = l + 1 < g.Q ? expf(dtf[co + l + 1] * A[h]) : 0.f;
  }
  const int pc = min(TN, g.P - p0);
  const Mat<float> M(cb + cb_idx(g, q.b, q.c, grp) + (size_t)i0 * g.Q, g.Q, min(TM, g.Q - i0), g.Q);
  const Mat<T> X(seq_at(x, g.xsb, g.xsl, q.b, t0, (long long)h * g.P + p0), g.xsl, nv, pc);
  const Mat<T> Ci(seq_at(Cm, g.csb, g.csl, q.b, t0 + i0, (long long)grp * g.N), g.csl, nv - i0, g.N);
  const Mat<float> S(prev + st_idx(g, q.b, q.c, h) + (size_t)p0 * g.N, g.N, pc, g.N);
  Acc acc;
  acc.zero();
  if (i0 > 0) contract<true, false>(acc, M, X, 0, i0, As, Bs, Keep(), [&](int k, int r, int, float4 v) { return scale4(v, fj[k + r]); });
  contract<true, true>(acc, Ci, S, 0, g.N, As, Bs, Keep(), [&](int, int, int, float4 v) { return scale4(v, eref); });
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  float e[4];   // decay between the tile's first row and each of this thread's rows
#pragma unroll
  for (int r = 0; r < 4; ++r) e[r] = i0 + 4 * ty + r < g.Q ? expf(css[i0 + 4 * ty + r] - ref) : 0.f;
  acc.scale(e);
  contract<true, false>(acc, M, X, i0, min(i0 + TM, nv), As, Bs, [&](int k, int r, int c, float4 v) {
    const int i = i0 + r, j = k + c;
    if (i >= g.Q || j > i) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 s4 = *reinterpret_cast<const float4*>(stp + j), d4 = *reinterpret_cast<const float4*>(dts + j);
    const float st[3] = {s4.x, s4.y, s4.z};
    float e[4];
    walk4(css[i], css[min(j + 3, g.Q - 1)], i - j, st, e);
    return make_float4(v.x * e[0] * d4.x, i - j >= 1 ? v.y * e[1] * d4.y : 0.f, i - j >= 2 ? v.z * e[2] * d4.z : 0.f, i - j >= 3 ? v.w * e[3] * d4.w : 0.f);
  }, Keep());
  float o[4][4];
  acc.get(o);
  const float Dh = D ? D[h] : 0.f;
  const int p = p0 + 4 * tx, np = g.P - p;
  if (np <= 0) return;
  const Mat<T> Z(z ? seq_at(z, g.zsb, g.zsl, q.b, t0, (long long)h * g.P + p0) : x, g.zsl, nv, pc);
  const Mat<T> DY(GATE_BWD ? seq_at(dy, g.ysb, g.ysl, q.b, t0, (long long)h * g.P + p0) : x, g.ysl, nv, pc);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + 4 * ty + r;
    if (i >= nv) continue;
    float xv[4], zv[4];
    float (&v)[4] = o[r];
    get4(X, i, 4 * tx, xv);
    if (GATE_BWD || z) get4(Z, i, 4 * tx, zv);
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] += Dh * xv[c];
    if constexpr (!GATE_BWD) {
      if (z) {
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] *= zv[c] * sigmoidf_(zv[c]);
      }
      st4(y + q.b * g.ysb + (t0 + i) * g.ysl + (long long)h * g.P + p, v, np);
    } else {
      float dv[4], a[4];
      get4(DY, i, 4 * tx, dv);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float sg = 1.f / (1.f + expf(-zv[c]));
        a[c] = dv[c] * v[c] * sg * (1.f + zv[c] * (1.f - sg));
        dv[c] *= zv[c] * sg;
      }
      const size_t od = ((size_t)(q.b * (size_t)g.L + t0 + i) * g.H + h) * g.P + p;
      st4(dz + od, a, np);
      st4(dyp + od, dv, np);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Backward.  `dy` is the gradient w.r.t. the pre-gate output: dy itself, or (gated) the fp32 copy in the workspace.
//
// W: wsum[b,c,g,i,j] = sum_{h in g} W_h,  W_h[i,j] = exp(cs_h,i-cs_h,j) dt_h,j (dy[i,h,:] . x[j,h,:]),  j <= i.  Two sums of
// the dt / decay gradients fall out of it: dcs_i's intra-chunk part is sum_j W_h[i,j] cb[i,j] (one partial per column strip),
// and ddot_i = dy[i,h,:] . x[i,h,:] is the undecayed diagonal.
template <typename T, typename TD>
__device__ __forceinline__ void w_tile(const Geo& g, unsigned u, const T* x, const TD* dy, long long dsb, long long dsl, const float* __restrict__ A,
                                       const float* __restrict__ cs, const float* __restrict__ dtf, const float* __restrict__ cb,
                                       float* __restrict__ wsum, float* __restrict__ dcs_part, float* __restrict__ ddot, float* As, float* Bs) {
  const Place q = place_of(u, tri_tiles(g.Q), g.G, g.nc);
  int i0, j0;
  tri_at(g.Q, q.tile, i0, j0);
  const int t0 = q.c * g.Q, nv = valid_rows(g, q.c), tx = threadIdx.x & 7, ty = threadIdx.x >> 3, i = i0 + 4 * ty, j = j0 + 4 * tx;
  const size_t nq = (size_t)g.B * g.H * g.nc * g.Q;
  const Mat<float> CB(cb + cb_idx(g, q.b, q.c, q.x), g.Q, g.Q, g.Q);
  float cbv[4][4], sum[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    get4(CB, i + r, j, cbv[r]);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (j + c > i + r) cbv[r][c] = 0.f;
      sum[r][c] = 0.f;
    }
  }
  const bool apart = j0 + TN <= i0;   // no element on the diagonal: the decay splits at row i0
  const int ks = (g.P + KC - 1) / KC, total = g.hpg * ks;
  Slab<TM, KC> a;
  Slab<TN, KC> b;
  auto load = [&](int it) {
    const int hl = ks == 1 ? it : it / ks, h = q.x * g.hpg + hl, k = (it - hl * ks) * KC;
    a.load(Mat<TD>(seq_at(dy, dsb, dsl, q.b, t0 + i0, (long long)h * g.P), dsl, nv - i0, g.P), 0, k);
    b.load(Mat<T>(seq_at(x, g.xsb, g.xsl, q.b, t0 + j0, (long long)h * g.P), g.xsl, nv - j0, g.P), 0, k);
  };
  Acc acc;
  acc.zero();
  load(0);
  for (int it = 0; it < total; ++it) {
    __syncthreads();
    a.store_k(As, Same());
    b.store_k(Bs, Same());
    __syncthreads();
    if (it + 1 < total) load(it + 1);
    const int hl = ks == 1 ? it : it / ks, h = q.x * g.hpg + hl;
    const bool last = it + 1 == (hl + 1) * ks;
    const size_t co = cs_idx(g, q.b, h, q.c);
    float ci[4], cj[4], dj[4], ref = 0.f;
    if (last) {   // on the way during the arithmetic
      ref = cs[co + i0];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        ci[r] = i + r < g.Q ? cs[co + i + r] : 0.f;
        cj[r] = j + r < g.Q ? cs[co + j + r] : 0.f;
        dj[r] = j + r < g.Q ? dtf[co + j + r] : 0.f;
      }
    }
    mac<true, true>(acc, As, Bs);
    if (!last) continue;
    float o[4][4], rs[4];
    acc.get(o);
    acc.zero();
    float e[4], f[4], st[3];
    if (apart) {
#pragma unroll
      for (int r = 0; r < 4; ++r) { e[r] = expf(ci[r] - ref); f[r] = expf(ref - cj[r]) * dj[r]; }
    } else {
#pragma unroll
      for (int r = 0; r < 3; ++r) st[r] = expf(dj[r + 1] * A[h]);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      rs[r] = 0.f;
      float wk[4];
      if (!apart) walk4(ci[r], cj[3], i + r - j, st, wk);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (i + r == j + c && i + r < g.Q) ddot[co + i + r] = o[r][c];
        const float l = apart ? e[r] * f[c] : (j + c <= i + r ? wk[c] * dj[c] : 0.f);
        const float w = o[r][c] * l;
        sum[r][c] += w;
        rs[r] = fmaf(w, cbv[r][c], rs[r]);
      }
      rs[r] = row_reduce(rs[r]);
    }
    if (tx == 0) {
      float* dst = dcs_part + (size_t)(j0 / TN) * nq + co;
#pragma unroll
      for (int r = 0; r < 4; ++r) if (i + r < g.Q) dst[i + r] = rs[r];
    }
  }
  float* dst = wsum + cb_idx(g, q.b, q.c, q.x);
#pragma unroll
  for (int r = 0; r < 4; ++r)
    if (i + r < g.Q && j < g.Q) st4(dst + (size_t)(i + r) * g.Q + j, sum[r], g.Q - j);
}

// The part of a backward that needs no state gradient from other chunks, one launch: W, then the local state gradients.
template <typename T, typename TD>
__global__ void __launch_bounds__(NT, 4) k_bwd_local(Geo g, unsigned n_w, const T* __restrict__ x, const TD* __restrict__ dy, long long dsb,
                                                     long long dsl, const float* __restrict__ A, const T* __restrict__ Cm, const float* __restrict__ cs,
                                                     const float* __restrict__ dtf, const float* __restrict__ cb, float* __restrict__ wsum,
                                                     float* __restrict__ dcs_part, float* __restrict__ ddot, float* __restrict__ dstates) {
  pdl_wait();
  __shared__ __align__(16) float As[A_FLOATS], Bs[B_FLOATS], row[256];
  if (blockIdx.x < n_w) w_tile(g, blockIdx.x, x, dy, dsb, dsl, A, cs, dtf, cb, wsum, dcs_part, ddot, As, Bs);
  else state_tile<1>(g, blockIdx.x - n_w, dy, dsb, dsl, Cm, g.csb, g.csl, cs, dtf, dstates, As, Bs, row);
}

// dx:  u[j,p] = sum_{i>=j} cb[i,j] exp(cs_i-cs_j) dy[i,p] + exp(cs_end-cs_j) sum_n B[j,n] dS[p,n]
//      dx = D dy + dt_j u ;  ddtd[j] = sum_p x[j,p] u[j,p] (one partial per 32 features)
template <typename T, typename TD>
__device__ __forceinline__ void dx_tile(const Geo& g, unsigned u, const T* x, const T* Bm, const float* A, const float* D, const TD* dy, long long dsb,
                                        long long dsl, const float* __restrict__ cs, const float* __restrict__ dtf,
                                        const float* __restrict__ cb, const float* __restrict__ dS, T* dx, float* __restrict__ ddt_part,
                                        float* As, float* Bs, float* css, float* stp) {
  const int ntj = (g.Q + TM - 1) / TM, ntp = (g.P + TN - 1) / TN;
  const Place q = place_of(u, ntj * ntp, g.H, g.nc);
  const int j0 = (q.tile % ntj) * TM, pt = q.tile / ntj, p0 = pt * TN, h = q.x, grp = h / g.hpg, t0 = q.c * g.Q, nv = valid_rows(g, q.c);
  const size_t co = cs_idx(g, q.b, h, q.c), nq = (size_t)g.B * g.H * g.nc * g.Q;
  const float a = A[h];
  for (int l = threadIdx.x; l < g.Q; l += NT) {
    const float c = cs[co + l], dn = dtf[co + min(l + 1, g.Q - 1)];
    css[l] = c;
    stp[l] = expf(dn * a);
  }
  __syncthreads();
  const float ref = css[min(j0 + TM, g.Q) - 1], eend = expf(css[g.Q - 1] - ref);
  const int pc = min(TN, g.P - p0);
  const Mat<float> M(cb + cb_idx(g, q.b, q.c, grp) + j0, g.Q, g.Q, min(TM, g.Q - j0));
  const Mat<TD> DY(seq_at(dy, dsb, dsl, q.b, t0, (long long)h * g.P + p0), dsl, nv, pc);
  const Mat<T> X(seq_at(x, g.xsb, g.xsl, q.b, t0, (long long)h * g.P + p0), g.xsl, nv, pc);
  const Mat<T> Bj(seq_at(Bm, g.bsb, g.bsl, q.b, t0 + j0, (long long)grp * g.N), g.bsl, nv - j0, g.N);
  const Mat<float> S(dS + st_idx(g, q.b, q.c, h) + (size_t)p0 * g.N, g.N, pc, g.N);
  Acc acc;
  acc.zero();
  if (j0 + TM < nv)
    contract<false, false>(acc, M, DY, j0 + TM, nv, As, Bs, Keep(),
                           [&](int k, int r, int, float4 v) { return scale4(v, k + r < g.Q ? expf(css[k + r] - ref) : 0.f); });
  contract<true, true>(acc, Bj, S, 0, g.N, As, Bs, Keep(), [&](int, int, int, float4 v) { return scale4(v, eend); });
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  float e[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) e[r] = j0 + 4 * ty + r < g.Q ? expf(ref - css[j0 + 4 * ty + r]) : 0.f;
  acc.scale(e);
  contract<false, false>(acc, M, DY, j0, min(j0 + TM, g.Q), As, Bs, [&](int k, int r, int c, float4 v) {
    const int i = k + r, j = j0 + c;   // row i of cb, columns j .. j + 3
    if (i >= g.Q || j > i) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 s4 = *reinterpret_cast<const float4*>(stp + j);
    const float st[3] = {s4.x, s4.y, s4.z};
    float e[4];
    walk4(css[i], css[min(j + 3, g.Q - 1)], i - j, st, e);
    return make_float4(v.x * e[0], i - j >= 1 ? v.y * e[1] : 0.f, i - j >= 2 ? v.z * e[2] : 0.f, i - j >= 3 ? v.w * e[3] : 0.f);
  }, Keep());
  float o[4][4];
  acc.get(o);
  const float Dh = D ? D[h] : 0.f;
  const int np = pc - 4 * tx;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int j = j0 + 4 * ty + r;
    float xv[4], dv[4], s = 0.f;
    get4(X, j, 4 * tx, xv);
    get4(DY, j, 4 * tx, dv);
    const float dtj = j < nv ? dtf[co + j] : 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      s = fmaf(xv[c], o[r][c], s);
      dv[c] = Dh * dv[c] + dtj * o[r][c];
    }
    if (j < nv && np > 0) st4(dx + ((size_t)(q.b * (size_t)g.L + t0 + j) * g.H + h) * g.P + p0 + 4 * tx, dv, np);
    s = row_reduce(s);
    if (tx == 0 && j < g.Q) ddt_part[(size_t)pt * nq + co + j] = s;
  }
}

// dC (MODE 0) and dB (MODE 1):
//   dC[i,n] = sum_{j<=i} wsum[i,j] B[j,n] + sum_{h,p} exp(cs_h,i) dy[i,h,p] prev[h,p,n]
//   dB[j,n] = sum_{i>=j} wsum[i,j] C[i,n] + sum_{h,p} exp(cs_h,end-cs_h,j) dt_h,j x[j,h,p] dS[h,p,n]
// dcs_i's inter-chunk part of head h is the head's summand of dC[i,:] dotted with C[i,:] (one partial per 32 columns).
template <int MODE, typename T, typename TH>
__device__ __forceinline__ void dbc_tile(const Geo& g, unsigned u, const T* Other, long long osb, long long osl, const T* Cm, const TH* hp,
                                         long long hsb, long long hsl, const float* __restrict__ cs, const float* __restrict__ dtf,
                                         const float* __restrict__ wsum, const float* __restrict__ st, T* out, float* __restrict__ dcs_part,
                                         float* As, float* Bs) {
  const int ntr = (g.Q + TM - 1) / TM, ntn = (g.N + TN - 1) / TN;
  const Place q = place_of(u, ntr * ntn, g.G, g.nc);
  const int r0 = (q.tile % ntr) * TM, nt = q.tile / ntr, n0 = nt * TN, t0 = q.c * g.Q, nv = valid_rows(g, q.c), nc4 = min(TN, g.N - n0);
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3, row = r0 + 4 * ty, nn = nc4 - 4 * tx;
  const size_t nq = (size_t)g.B * g.H * g.nc * g.Q;
  const float* wp = wsum + cb_idx(g, q.b, q.c, q.x);
  Acc tot;
  tot.zero();
  const Mat<T> O(seq_at(Other, osb, osl, q.b, t0, (long long)q.x * g.N + n0), osl, nv, nc4);
  if constexpr (MODE == 0)
    contract<true, false>(tot, Mat<float>(wp + (size_t)r0 * g.Q, g.Q, min(TM, g.Q - r0), g.Q), O, 0, min(r0 + TM, g.Q), As, Bs, Keep(), Keep());
  else
    contract<false, false>(tot, Mat<float>(wp + r0, g.Q, g.Q, min(TM, g.Q - r0)), O, r0, g.Q, As, Bs, Keep(), Keep());
  float cv[4][4];
  if constexpr (MODE == 0) {
    const Mat<T> CI(seq_at(Cm, g.csb, g.csl, q.b, t0, (long long)q.x * g.N + n0), g.csl, nv, nc4);
#pragma unroll
    for (int r = 0; r < 4; ++r) get4(CI, row + r, 4 * tx, cv[r]);
  }
  const int ks = (g.P + KC - 1) / KC, total = g.hpg * ks;
  Slab<TM, KC> a;
  Slab<KC, TN> b;
  float sc[Slab<TM, KC>::V];   // the staged rows' factors
  auto load = [&](int it) {
    const int hl = ks == 1 ? it : it / ks, h = q.x * g.hpg + hl, k = (it - hl * ks) * KC;
    a.load(Mat<TH>(seq_at(hp, hsb, hsl, q.b, t0 + r0, (long long)h * g.P), hsl, nv - r0, g.P), 0, k);
    b.load(Mat<float>(st + st_idx(g, q.b, q.c, h) + n0, g.N, g.P, nc4), k, 0);
    const size_t co = cs_idx(g, q.b, h, q.c);
#pragma unroll
    for (int v = 0; v < Slab<TM, KC>::V; ++v) {
      const int r = r0 + (threadIdx.x + v * NT) / (KC / 4);
      sc[v] = r >= g.Q ? 0.f : MODE == 0 ? expf(cs[co + r]) : expf(cs[co + g.Q - 1] - cs[co + r]) * dtf[co + r];
    }
  };
  load(0);
  Acc acc;
  acc.zero();
  for (int it = 0; it < total; ++it) {
    __syncthreads();
#pragma unroll
    for (int v = 0; v < Slab<TM, KC>::V; ++v) a.v[v] = scale4(a.v[v], sc[v]);
    a.store_k(As, Same());
    b.template store_r<PB>(Bs, Same());
    __syncthreads();
    if (it + 1 < total) load(it + 1);
    if constexpr (MODE == 1) {
      mac<true, false>(tot, As, Bs);
    } else {
      const int hl = ks == 1 ? it : it / ks, h = q.x * g.hpg + hl;
      mac<true, false>(acc, As, Bs);
      if (it + 1 != (hl + 1) * ks) continue;
      float* dst = dcs_part + (size_t)nt * nq + cs_idx(g, q.b, h, q.c);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float o[4];
        unpack2(acc.n[r][0], o[0], o[1]);
        unpack2(acc.n[r][1], o[2], o[3]);
        float s = o[0] * cv[r][0];
        s = fmaf(o[1], cv[r][1], s); s = fmaf(o[2], cv[r][2], s); s = fmaf(o[3], cv[r][3], s);
        s = row_reduce(s);
        if (tx == 0 && row + r < g.Q) dst[row + r] = s;
        tot.n[r][0] = add2(tot.n[r][0], acc.n[r][0]);
        tot.n[r][1] = add2(tot.n[r][1], acc.n[r][1]);
        acc.n[r][0] = acc.n[r][1] = 0ull;
      }
    }
  }
  float o[4][4];
  tot.get(o);
  if (nn <= 0) return;
#pragma unroll
  for (int r = 0; r < 4; ++r)
    if (row + r < nv) st4(out + ((size_t)(q.b * (size_t)g.L + t0 + row + r) * g.G + q.x) * g.N + n0 + 4 * tx, o[r], nn);
}

// What follows the reverse scan over chunks, one launch: dC, dB (the longest tiles), dx.
template <typename T, typename TD>
__global__ void __launch_bounds__(NT, 4) k_bwd_final(Geo g, unsigned n_bc, const T* __restrict__ x, const T* __restrict__ Bm,
                                                     const T* __restrict__ Cm, const float* __restrict__ A, const float* __restrict__ D,
                                                     const TD* __restrict__ dy, long long dsb, long long dsl, const float* __restrict__ cs,
                                                     const float* __restrict__ dtf, const float* __restrict__ cb, const float* __restrict__ wsum,
                                                     const float* __restrict__ prev, const float* __restrict__ dS, T* __restrict__ dx,
                                                     T* __restrict__ dB, T* __restrict__ dC, float* __restrict__ dcs_part,
                                                     float* __restrict__ ddt_part) {
  pdl_wait();
  __shared__ __align__(16) float As[A_FLOATS], Bs[B_FLOATS], css[256], stp[256];
  const unsigned u = blockIdx.x;
  if (u < n_bc) dbc_tile<0>(g, u, Bm, g.bsb, g.bsl, Cm, dy, dsb, dsl, cs, dtf, wsum, prev, dC, dcs_part, As, Bs);
  else if (u < 2 * n_bc) dbc_tile<1>(g, u - n_bc, Cm, g.csb, g.csl, Cm, x, g.xsb, g.xsl, cs, dtf, wsum, dS, dB, dcs_part, As, Bs);
  else dx_tile(g, u - 2 * n_bc, x, Bm, A, D, dy, dsb, dsl, cs, dtf, cb, dS, dx, ddt_part, As, Bs, css, stp);
}

// ---------------------------------------------------------------------------------------------
// Stage 3 for states whose size is no multiple of 4 (k_state_passing_v4 takes the others): exclusive scan over chunks, in place.  Forward direction turns per-chunk states into
// the state ENTERING each chunk and emits the final state; reverse direction does the same for
// the state gradient (entering from the right) and emits the gradient of the initial state.
//   WRITE=false only produces `last` (used by the sequence-parallel split to get the slice total).
template <bool WRITE>
__global__ void __launch_bounds__(ST) k_state_passing(Geo g, float* __restrict__ st, const float* __restrict__ cs,
                                                      const float* __restrict__ init, float* __restrict__ last,
                                                      float* __restrict__ last2, int reverse) {
  pdl_wait();
  const int e = blockIdx.x * ST + threadIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int PN = g.P * g.N;
  if (e >= PN) return;
  float run = init ? init[((size_t)(b * g.H + h)) * PN + e] : 0.f;
  for (int s = 0; s < g.nc; ++s) {
    const int c = reverse ? g.nc - 1 - s : s;
    float* ptr = st + st_idx(g, b, c, h) + e;
    const float v = *ptr;
    if (WRITE) *ptr = run;
    run = expf(cs[cs_idx(g, b, h, c) + g.Q - 1]) * run + v;
  }
  if (last) last[((size_t)(b * g.H + h)) * PN + e] = run;
  if (last2) last2[((size_t)(b * g.H + h)) * PN + e] = run;
}

// ---------------------------------------------------------------------------------------------
// Backward, beside k_state_passing: sdot[b,c,h] = <dS_end_c, S_end_c>, with S_end_c = state entering chunk c+1 (or final).
__global__ void __launch_bounds__(ST) k_sdot(Geo g, const float* __restrict__ dS, const float* __restrict__ prev,
                                             const float* __restrict__ fin, float* __restrict__ sdot) {
  pdl_wait();
  const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int PN = g.P * g.N;
  const float* a = dS + st_idx(g, b, c, h);
  const float* s = (c + 1 < g.nc) ? prev + st_idx(g, b, c + 1, h) : fin + ((size_t)(b * g.H + h)) * PN;
  float v = 0.f;
  for (int e = threadIdx.x; e < PN; e += ST) v = fmaf(a[e], s[e], v);
  __shared__ float red[ST / 32];
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < ST / 32; ++i) t += red[i];
    sdot[(size_t)(b * g.nc + c) * g.H + h] = t;
  }
}

// ---------------------------------------------------------------------------------------------
// Backward: da_k = sum_{i>=k in chunk}(dcsp_i - dt_i*ddtd_i) + sdot ; ddt_k = ddtd_k + A*da_k (times the derivative
// of the step-size activation when dt_softplus is set) ;
// per-chunk partial sums for dA (= sum dt*da) and dD (= sum ddot).  One block per (chunk, batch, HG
// heads); sdot arrives as `nw` partial sums per (batch, chunk, head), added in fixed order.
// How dcsp and ddtd arrive: the tensor family sums them itself ({1, 0, 1}); the CUDA-core family leaves one part of dcsp per
// 32-column strip of the chunk (strips; only those up to the position's own hold anything), one per 32 state columns, and one
// part of ddtd per 32 features, `stride` elements apart.
struct DdtParts { int strips, columns, features; size_t stride; };
// HG heads at a time: 4 keep the registers low enough for a full SM (16 x 4096 tokens of 24 heads 19.5 us with 8, 13.7 with 4, and
// k_cumsum 14.0, 9.7; 512 x 1024 of 8 heads the same); 2 give a short batch twice the blocks (its time is one chain
// of loads and scans).  PARTS: the CUDA-core family's partial sums (their loops cost the other family 30 of 60 us at 512 x
// 1024 tokens of 8 heads).  The two sums over the chunk fold 2 HG values across the warp together: 16 shuffles instead of 80.
template <int HG, bool PARTS>
__global__ void __launch_bounds__(ST) k_ddt(Geo g, const float* __restrict__ A, const float* __restrict__ dtf,
                                            DdtParts parts, const float* __restrict__ dcsp,
                                            const float* __restrict__ ddtd, const float* __restrict__ ddot, const float* __restrict__ sdot, int nw,
                                            float* __restrict__ ddt, float* __restrict__ dapart,
                                            float* __restrict__ ddpart, float* __restrict__ dbpart) {
  pdl_wait();
  const int c = blockIdx.x, b = blockIdx.y, q = threadIdx.x;
  __shared__ float wsum[ST / 32][HG], red[ST / 32][2 * HG], red3[ST / 32][HG], ssd[HG];
  const int qr = g.Q - 1 - q;   // reversed position: an inclusive prefix scan over q is a suffix sum over qr
  const bool ok = (q < g.Q);
  const int lane = q & 31, w = q >> 5, nwarp = blockDim.x >> 5;   // launched with 128 threads when the chunk is <= 128 long
  const int t = c * g.Q + qr;
  for (int h0 = blockIdx.z * HG; h0 < g.H; h0 += HG * gridDim.z) {
    for (int hh = w; hh < HG; hh += nwarp) {   // a warp adds the partial sums of head h0 + hh (fixed order: lane-strided, then a butterfly)
      float s = 0.f;
      if (h0 + hh < g.H) {
        const float* sp = sdot + ((size_t)(b * g.nc + c) * g.H + h0 + hh) * nw;
        for (int i = lane; i < nw; i += 32) s += sp[i];
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) ssd[hh] = s;
    }
    float d[HG], dd[HG], v[HG], s12[2 * HG];   // s12: the dA terms, then the dD terms
#pragma unroll
    for (int k = 0; k < HG; ++k) {
      const int h = h0 + k;
      const bool live = ok && h < g.H;
      const size_t o = live ? cs_idx(g, b, h, c) + qr : 0;
      d[k] = live ? dtf[o] : 0.f;
      dd[k] = live ? ddtd[o] : 0.f;
      float dc = live ? dcsp[o] : 0.f;
      if (PARTS && live) {   // further parts, in a fixed order
#pragma unroll 4
        for (int s = 1; s < parts.features; ++s) dd[k] += ddtd[s * parts.stride + o];
        const int strips = min(parts.strips - 1, qr / TN);
#pragma unroll 4
        for (int s = 1; s <= strips; ++s) dc += dcsp[s * parts.stride + o];
#pragma unroll 4
        for (int s = 0; s < parts.columns; ++s) dc += dcsp[(parts.strips + s) * parts.stride + o];
      }
      v[k] = live ? dc - d[k] * dd[k] : 0.f;
      s12[HG + k] = live ? ddot[o] : 0.f;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int k = 0; k < HG; ++k) {
        const float n = __shfl_up_sync(0xffffffffu, v[k], o);
        if (lane >= o) v[k] += n;
      }
    }
    if (lane == 31) {
#pragma unroll
      for (int k = 0; k < HG; ++k) wsum[w][k] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < HG; ++k) {
      float base = 0.f;
      for (int i = 0; i < w; ++i) base += wsum[i][k];
      const float da = v[k] + base + ssd[k];
      s12[k] = ok ? d[k] * da : 0.f;
      v[k] = dd[k] + ((h0 + k < g.H) ? A[h0 + k] : 0.f) * da;   // gradient w.r.t. the step size of this position
      // ... and through softplus to the dt that was passed in: softplus'(r) = sigmoid(r) = 1 - exp(-softplus(r))
      if (g.dt_softplus) v[k] *= 1.f - __expf(-d[k]);
    }
    if (ok && t < g.L) {
      float* o = ddt + ((size_t)b * g.L + t) * g.H + h0;
      if (HG % 4 == 0 && h0 + HG <= g.H && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
#pragma unroll
        for (int k = 0; k + 3 < HG; k += 4) *reinterpret_cast<float4*>(o + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
      } else {
#pragma unroll
        for (int k = 0; k < HG; ++k)
          if (h0 + k < g.H) o[k] = v[k];
      }
    }
    int which;
    const float s = fold_rows<32, 2 * HG>(s12, lane, which);
    if (lane % (32 / (2 * HG)) == 0) red[w][which] = s;
    if (dbpart) {   // the chunk's share of the step-size bias gradient
      if (!(ok && t < g.L)) {
#pragma unroll
        for (int k = 0; k < HG; ++k) v[k] = 0.f;
      }
      const float s3 = fold_rows<32, HG>(v, lane, which);
      if (lane % (32 / HG) == 0) red3[w][which] = s3;
    }
    __syncthreads();
    if (q < HG && h0 + q < g.H) {
      float a1 = 0.f, a2 = 0.f;
      for (int i = 0; i < nwarp; ++i) { a1 += red[i][q]; a2 += red[i][HG + q]; }
      if (dbpart) {
        float a3 = 0.f;
        for (int i = 0; i < nwarp; ++i) a3 += red3[i][q];
        dbpart[(size_t)(b * g.nc + c) * g.H + h0 + q] = a3;
      }
      dapart[(size_t)(b * g.nc + c) * g.H + h0 + q] = a1;
      ddpart[(size_t)(b * g.nc + c) * g.H + h0 + q] = a2;
    }
    __syncthreads();
  }
}

// dA[h] = sum over (b,c) of dapart; dD, ddt_bias likewise.  One block per head, fixed summation order.  The block is as large
// as it gets because the kernel is a chain of dependent memory round trips: rows / 1024 of them.
constexpr int RH_THREADS = 1024;
__global__ void __launch_bounds__(RH_THREADS) k_reduce_heads(int rows, int H, const float* __restrict__ dapart,
                                                             const float* __restrict__ ddpart, const float* __restrict__ dbpart,
                                                             float* __restrict__ dA, float* __restrict__ dD, float* __restrict__ dbias) {
  pdl_wait();
  const int h = blockIdx.x;
  float a = 0.f, d = 0.f, e = 0.f;
#pragma unroll 4
  for (int r = threadIdx.x; r < rows; r += RH_THREADS) {
    a += dapart[(size_t)r * H + h];
    d += ddpart[(size_t)r * H + h];
    if (dbpart) e += dbpart[(size_t)r * H + h];
  }
  __shared__ float red[3][RH_THREADS / 32];
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    d += __shfl_xor_sync(0xffffffffu, d, o);
    e += __shfl_xor_sync(0xffffffffu, e, o);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { red[0][w] = a; red[1][w] = d; red[2][w] = e; }
  __syncthreads();
  if (w < 3) {
    float t = red[w][lane];
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    float* out = w == 0 ? dA : w == 1 ? dD : dbias;
    if (lane == 0 && out) out[h] = t;
  }
}

}  // namespace

// =============================================================================================
// Host launchers
// =============================================================================================
template <auto K> struct Fn { static constexpr auto value = K; };   // a kernel as a value of its own type

// Blocks of the CUDA-core kernels (one tile each); pick_family has checked that they fit a grid.
struct Tiles {
  unsigned state, cb, scan, bc;
  int strips;      // 32-column strips of a chunk
  size_t nq;       // positions x heads, chunks padded
  explicit Tiles(const Geo& g) {
    const long long bc_ = (long long)g.B * g.nc, q = cdiv(g.Q, TM);
    state = (unsigned)(bc_ * g.H * cdiv(g.N, TM) * cdiv(g.P, TN));
    int tri = 0;
    for (int i0 = 0; i0 < g.Q; i0 += TM) tri += cdiv(i0 + TM < g.Q ? i0 + TM : g.Q, TN);
    cb = (unsigned)(bc_ * g.G * tri);
    scan = (unsigned)(bc_ * g.H * q * cdiv(g.P, TN));
    bc = (unsigned)(bc_ * g.G * q * cdiv(g.N, TN));
    strips = cdiv(g.Q, TN);
    nq = (size_t)g.B * g.H * g.nc * g.Q;
  }
};

// Stage 3 of the CUDA-core family: four elements per thread where sizes and pointers allow it (that kernel stages one decay
// per chunk in shared memory).
static int core_state_passing(const Geo& g, float* st, const float* cs, const float* init, float* last, float* last2, int reverse, bool write,
                              const float* prev, const float* fin, float* sdot, int* sdot_nw, cudaStream_t s) {
  const uintptr_t low = (uintptr_t)init | (uintptr_t)last | (uintptr_t)last2;
  if ((g.P * g.N) % 4 == 0 && (low & 15) == 0 && g.nc <= 32768)
    return tensor_state_passing(g, st, cs, init, last, last2, nullptr, reverse, write, prev, nullptr, fin, sdot, sdot_nw, s);
  const dim3 grid(cdiv(g.P * g.N, ST), g.H, g.B);
  if (write) launch<k_state_passing<true>>(grid, ST, 0, s, g, st, cs, init, last, last2, reverse);
  else launch<k_state_passing<false>>(grid, ST, 0, s, g, st, cs, init, last, last2, reverse);
  SSD_CUDA_CHECK_LAUNCH("state_passing");
  if (sdot) {
    if (sdot_nw) *sdot_nw = 1;
    launch<k_sdot>(dim3(g.nc, g.H, g.B), ST, 0, s, g, st, prev, fin, sdot);
    SSD_CUDA_CHECK_LAUNCH("sdot");
  }
  return SSD_OK;
}

template <typename T>
static int fwd_stages_t(const Geo& g, bool tc, const SsdFwdPtrs& p, char* ws, const WsLayout& w, cudaStream_t s,
                        int stages, bool keep_fin) {
  int* status = (int*)(ws + w.status);
  float* cs = (float*)(ws + w.cs);
  float* dtf = (float*)(ws + w.dtf);
  float* states = (float*)(ws + w.states);
  float* cb = (float*)(ws + w.cb);
  // the final state: the workspace's copy is the backward's, the other the caller's; both are written where it is formed
  float* fin = keep_fin ? (float*)(ws + w.fin) : p.final_state;
  float* fin2 = keep_fin ? p.final_state : nullptr;
  float* tab = (float*)(ws + w.tab);
  void* prev_bf = ws + w.prev_bf;
  const T* x = (const T*)p.x;
  // a full pass (no sequence-parallel staging) computes the chunk states inside the scan over chunks where that kernel applies
  const bool fused = tc && stages == (SSD_STAGE_LOCAL | SSD_STAGE_FINISH) && tensor_state_fused_applies(g);
  if (stages & (SSD_STAGE_LOCAL | SSD_STAGE_LOCAL_STATES)) {
    const bool wide = (long long)g.nc * g.B >= 2LL * sm_count();
    auto cumsum = [&](auto kernel) {
      launch<kernel.value>(dim3(g.nc, g.B, wide ? cdiv(g.H, 4) : cdiv(g.H, 2)), g.Q <= 128 ? 128 : 256, 0, s, g, (const T*)p.dt, p.dt_bias, p.A, cs, dtf,
                           tc ? tab : nullptr, tc ? (int*)(ws + w.hand) : nullptr, status);
    };
    wide ? cumsum(Fn<k_cumsum<T, 4>>()) : cumsum(Fn<k_cumsum<T, 2>>());
    SSD_CUDA_CHECK_LAUNCH("cumsum");
    if (tc && fused) {
      // chunk states and the scan over chunks run as one kernel in the FINISH stage
    } else if (tc) {
      int rc = tensor_chunk_state(g, 0, p.x, g.xsb, g.xsl, p.Bm, g.bsb, g.bsl, tab, states, status, s);
      if (rc) return rc;
    } else {
      const Tiles n(g);
      launch<k_local<T>>(n.state + n.cb, NT, 0, s, g, n.state, x, (const T*)p.Bm, (const T*)p.Cm, cs, dtf, states, cb);
      SSD_CUDA_CHECK_LAUNCH("chunk_state");
    }
  }
  if (stages & SSD_STAGE_TOTAL) {
    if (tc) {
      int rc = tensor_state_passing(g, states, cs, nullptr, fin, fin2, nullptr, 0, false, nullptr, nullptr, nullptr, nullptr, nullptr, s);
      if (rc) return rc;
    } else {
      int rc = core_state_passing(g, states, cs, nullptr, fin, fin2, 0, false, nullptr, nullptr, nullptr, nullptr, s);
      if (rc) return rc;
    }
  }
  if (stages & SSD_STAGE_FINISH) {
    if (tc && fused) {
      // no fp32 copy of the chunk-entry states: every reader in this family takes the bf16 one
      int rc = tensor_state_fused(g, 0, p.x, g.xsb, g.xsl, p.Bm, g.bsb, g.bsl, tab, states, (int*)(ws + w.hand), prev_bf,
                                  p.init_state, fin, fin2, nullptr, nullptr, nullptr, nullptr, status, s);
      if (rc) return rc;
    } else if (tc) {
      int rc = tensor_state_passing(g, states, cs, p.init_state, fin, fin2, prev_bf, 0, true, nullptr, nullptr, nullptr, nullptr, nullptr, s);
      if (rc) return rc;
    } else {
      int rc = core_state_passing(g, states, cs, p.init_state, fin, fin2, 0, true, nullptr, nullptr, nullptr, nullptr, s);
      if (rc) return rc;
    }
    if (p.y && tc) {
      int rc = tensor_chunk_scan(g, p, tab, prev_bf, status, s);
      if (rc) return rc;
    } else if (p.y) {
      launch<k_chunk_scan<T, false>>(Tiles(g).scan, NT, 0, s, g, x, (const T*)p.Cm, p.A, p.D, (const T*)p.z, cs, dtf, cb, states, (T*)p.y,
                                     nullptr, nullptr, nullptr);
      SSD_CUDA_CHECK_LAUNCH("chunk_scan");
    }
  }
  return SSD_OK;
}

int run_forward(const Geo& g, int dtype, bool tc, const SsdFwdPtrs& p, char* ws, const WsLayout& w, cudaStream_t s,
                int stages, bool for_backward) {
  return dtype == SSD_BF16 ? fwd_stages_t<__nv_bfloat16>(g, tc, p, ws, w, s, stages, for_backward)
                           : fwd_stages_t<float>(g, false, p, ws, w, s, stages, for_backward);
}

template <typename T>
static int bwd_stages_t(const Geo& g, bool tc, const SsdBwdPtrs& p, char* ws, const WsLayout& w, cudaStream_t s,
                        int stages) {
  int* status = (int*)(ws + w.status);
  float* cs = (float*)(ws + w.cs);
  float* dtf = (float*)(ws + w.dtf);
  float* states = (float*)(ws + w.states);
  float* cb = (float*)(ws + w.cb);
  float* fin = (float*)(ws + w.fin);
  float* tab = (float*)(ws + w.tab);
  void* prev_bf = ws + w.prev_bf;
  void* ds_bf = ws + w.ds_bf;
  float* dst = (float*)(ws + w.dstates);
  float* wsum = (float*)(ws + w.wsum);   // CUDA-core family: a segment of its own, so the forward's C B^T survives a backward
  float* dyp = (float*)(ws + w.dyp);
  float* dcsp = (float*)(ws + w.dcsp);
  float* ddtd = (float*)(ws + w.ddtd);
  float* ddot = (float*)(ws + w.ddot);
  float* sdot = (float*)(ws + w.sdot);
  float* dapart = (float*)(ws + w.dapart);
  float* ddpart = (float*)(ws + w.ddpart);
  float* dini = p.dinit_state ? p.dinit_state : (float*)(ws + w.dini);
  const T* x = (const T*)p.x;
  // tensor-core family: the pre-gate gradient is dy itself, or (gated) a dense bf16 copy in the workspace
  const void* tc_dy = p.z ? (const void*)dyp : p.dy;
  const bool tc_dense = p.z != nullptr;
  const bool fused = tc && stages == (SSD_STAGE_LOCAL | SSD_STAGE_FINISH) && tensor_state_fused_applies(g);
  // LOCAL in two halves (see SSD_STAGE_LOCAL_STATES / _REST): the recompute pass is only read by FINISH unless a z gate
  // makes the local state gradients depend on the pre-gate dy it writes.
  const bool want_states = (stages & (SSD_STAGE_LOCAL | SSD_STAGE_LOCAL_STATES)) != 0;
  const bool want_rest = (stages & (SSD_STAGE_LOCAL | SSD_STAGE_LOCAL_REST)) != 0;
  const bool do_recompute = p.z ? want_states : want_rest;
  if (want_states) {
    if (!p.fwd_saved) {
      SsdFwdPtrs f{};
      f.x = p.x; f.dt = p.dt; f.A = p.A; f.Bm = p.Bm; f.Cm = p.Cm; f.D = p.D; f.z = p.z; f.dt_bias = p.dt_bias;
      f.init_state = p.init_state; f.y = nullptr; f.final_state = nullptr;
      int rc = fwd_stages_t<T>(g, tc, f, ws, w, s, SSD_STAGE_LOCAL | SSD_STAGE_FINISH, true);
      if (rc) return rc;
    }
  }
  if (do_recompute) {
    if (tc) {
      // ungated (dstate 64, or dstate 128): the recompute pass is folded into the dx kernel of the FINISH stage
      int rc = tensor_bwd_merged_applies(g, p) ? SSD_OK : tensor_scan_bwd(g, p, tab, prev_bf, dyp, dcsp, ddot, status, s);
      if (rc) return rc;
    } else {
      // only the gate needs the forward's outputs again: dz and the pre-gate dy (the row sums come out of W and dC)
      if (p.z) {
        launch<k_chunk_scan<T, true>>(Tiles(g).scan, NT, 0, s, g, x, (const T*)p.Cm, p.A, p.D, (const T*)p.z, cs, dtf, cb, states, nullptr,
                                      (const T*)p.dy, dyp, (T*)p.dz);
        SSD_CUDA_CHECK_LAUNCH("chunk_scan_bwd_epilogue");
      }
    }
  }
  const Tiles n(g);
  const long long HP = (long long)g.H * g.P;
  if (want_states) {
    if (tc) {
      if (!fused) {
        int rc = tensor_chunk_state(g, 1, tc_dy, tc_dense ? (long long)g.L * g.H * g.P : g.ysb,
                                    tc_dense ? (long long)g.H * g.P : g.ysl, p.Cm, g.csb, g.csl, tab, dst, status, s);
        if (rc) return rc;
      }
    } else {
      if (p.z)
        launch<k_bwd_local<T, float>>(n.state + n.cb, NT, 0, s, g, n.cb, x, dyp, HP * g.L, HP, p.A, (const T*)p.Cm, cs, dtf, cb, wsum, dcsp, ddot, dst);
      else
        launch<k_bwd_local<T, T>>(n.state + n.cb, NT, 0, s, g, n.cb, x, (const T*)p.dy, g.ysb, g.ysl, p.A, (const T*)p.Cm, cs, dtf, cb, wsum, dcsp,
                                  ddot, dst);
      SSD_CUDA_CHECK_LAUNCH("bwd_local");
    }
  }
  if (stages & SSD_STAGE_TOTAL) {
    int rc = tc ? tensor_state_passing(g, dst, cs, nullptr, dini, nullptr, nullptr, 1, false, nullptr, nullptr, nullptr, nullptr, nullptr, s)
                : core_state_passing(g, dst, cs, nullptr, dini, nullptr, 1, false, nullptr, nullptr, nullptr, nullptr, s);
    if (rc) return rc;
  }
  int sdot_nw = 1;
  if (stages & SSD_STAGE_FINISH) {
    if (tc && fused) {
      // local state gradients, the reverse scan and the <dS_end, S_end> partial sums in one kernel (no fp32 copy is kept)
      int rc = tensor_state_fused(g, 1, tc_dy, tc_dense ? (long long)g.L * g.H * g.P : g.ysb,
                                  tc_dense ? (long long)g.H * g.P : g.ysl, p.Cm, g.csb, g.csl, tab, dst, (int*)(ws + w.hand), ds_bf,
                                  p.dfinal_state, dini, nullptr, prev_bf, fin, sdot, &sdot_nw, status, s);
      if (rc) return rc;
    } else if (tc) {
      // the reverse scan also leaves the warp-partial sums of <dS_end, S_end> per chunk
      int rc = tensor_state_passing(g, dst, cs, p.dfinal_state, dini, nullptr, ds_bf, 1, true, states, prev_bf, fin, sdot, &sdot_nw, s);
      if (rc) return rc;
    } else {
      int rc = core_state_passing(g, dst, cs, p.dfinal_state, dini, nullptr, 1, true, states, fin, sdot, &sdot_nw, s);
      if (rc) return rc;
    }
    if (tc) {
      int rc = tensor_bwd_merged_applies(g, p) ? tensor_bwd_merged(g, p, tab, prev_bf, ds_bf, dcsp, ddot, ddtd, status, s)
                                                : tensor_dx(g, p, tc_dy, tc_dense, tab, ds_bf, ddtd, status, s);
      if (rc) return rc;
      rc = tensor_dbc(g, p, tc_dy, tc_dense, tab, prev_bf, ds_bf, status, s);
      if (rc) return rc;
    } else {
      float* dcs_cols = dcsp + (size_t)n.strips * n.nq;
      const unsigned blocks = 2 * n.bc + n.scan;
      if (p.z)
        launch<k_bwd_final<T, float>>(blocks, NT, 0, s, g, n.bc, x, (const T*)p.Bm, (const T*)p.Cm, p.A, p.D, dyp, HP * g.L, HP, cs, dtf, cb, wsum,
                                      states, dst, (T*)p.dx, (T*)p.dB, (T*)p.dC, dcs_cols, ddtd);
      else
        launch<k_bwd_final<T, T>>(blocks, NT, 0, s, g, n.bc, x, (const T*)p.Bm, (const T*)p.Cm, p.A, p.D, (const T*)p.dy, g.ysb, g.ysl, cs, dtf, cb,
                                  wsum, states, dst, (T*)p.dx, (T*)p.dB, (T*)p.dC, dcs_cols, ddtd);
      SSD_CUDA_CHECK_LAUNCH("bwd_final");
    }
    const DdtParts parts = tc ? DdtParts{1, 0, 1, 0} : DdtParts{n.strips, cdiv(g.N, TN), cdiv(g.P, TN), n.nq};
    float* dbpart = p.ddt_bias ? (float*)(ws + w.dbpart) : nullptr;
    const bool wide = (long long)g.nc * g.B >= 2LL * sm_count();   // four heads per block fill the SMs twice
    auto ddt = [&](auto kernel) {
      launch<kernel.value>(dim3(g.nc, g.B, wide ? cdiv(g.H, 4) : cdiv(g.H, 2)), g.Q <= 128 ? 128 : 256, 0, s, g, p.A, dtf, parts, dcsp, ddtd, ddot, sdot,
                           sdot_nw, p.ddt, dapart, ddpart, dbpart);
    };
    if (tc) wide ? ddt(Fn<k_ddt<4, false>>()) : ddt(Fn<k_ddt<2, false>>());
    else wide ? ddt(Fn<k_ddt<4, true>>()) : ddt(Fn<k_ddt<2, true>>());
    SSD_CUDA_CHECK_LAUNCH("ddt");
    launch<k_reduce_heads>(g.H, RH_THREADS, 0, s, g.B * g.nc, g.H, dapart, ddpart, dbpart, p.dA, p.dD, p.ddt_bias);
    SSD_CUDA_CHECK_LAUNCH("reduce_heads");
  }
  return SSD_OK;
}

int run_backward(const Geo& g, int dtype, bool tc, const SsdBwdPtrs& p, char* ws, const WsLayout& w, cudaStream_t s,
                 int stages) {
  return dtype == SSD_BF16 ? bwd_stages_t<__nv_bfloat16>(g, tc, p, ws, w, s, stages)
                           : bwd_stages_t<float>(g, false, p, ws, w, s, stages);
}

}  // namespace ssd
