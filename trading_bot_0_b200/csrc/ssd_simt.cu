// Exact-fp32 CUDA-core kernels for the SSD operator: every stage of forward and backward for
// any storage dtype, any chunk <= 256 and ragged sequence tails.  This family is the fp32-mode
// path (1e-4 relative parity) and the building block the sequence-parallel split reuses; the
// bf16 throughput path lives in ssd_tensor.cu.
//
// All contractions share one tile routine: a 256-thread block accumulates a 64x64 output tile,
// 4x4 per thread, staging 16-deep slabs of both operands in shared memory through element
// functors, so a stage is defined by "what is A(m,k), what is B(n,k), what does the epilogue do".
#include <atomic>
#include "common.cuh"
#include "ssd_internal.h"

namespace ssd {
namespace {

constexpr int TM = 64, TN = 64, TK = 16, LDS = 68, NT = 256;

template <bool A_KFAST, bool B_KFAST, class FA, class FB>
__device__ __forceinline__ void tile_mac(float (&acc)[4][4], int kbeg, int kend, FA fa, FB fb,
                                         float* As, float* Bs) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int k0 = kbeg; k0 < kend; k0 += TK) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      int m, kk;
      if (A_KFAST) { kk = tid & 15; m = (tid >> 4) + 16 * r; } else { m = tid & 63; kk = (tid >> 6) + 4 * r; }
      int k = k0 + kk;
      As[kk * LDS + m] = (k < kend) ? fa(m, k) : 0.f;
      if (B_KFAST) { kk = tid & 15; m = (tid >> 4) + 16 * r; } else { m = tid & 63; kk = (tid >> 6) + 4 * r; }
      k = k0 + kk;
      Bs[kk * LDS + m] = (k < kend) ? fb(m, k) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      const float4 a = *reinterpret_cast<const float4*>(&As[kk * LDS + ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&Bs[kk * LDS + tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(av[r], bv[c], acc[r][c]);
    }
    __syncthreads();
  }
}

__device__ __forceinline__ void zero_acc(float (&acc)[4][4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
}

// Sum over the 16 threads (tx) that share a tile row; every lane of the half-warp gets the sum.
__device__ __forceinline__ float row_reduce16(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 8);
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

// Gradient w.r.t. the pre-gate output: either the fp32 workspace copy (gated case) or dy itself.
template <typename T>
struct DySrc {
  const float* f;
  const T* t;
  long long sb, sl;
  __device__ __forceinline__ float get(const Geo& g, int b, int tt, int h, int p) const {
    if (f) return f[((size_t)(b * (size_t)g.L + tt) * g.H + h) * g.P + p];
    return ldf(t + b * sb + tt * sl + (long long)h * g.P + p);
  }
};

// ---------------------------------------------------------------------------------------------
// Stage 1: cs = inclusive within-chunk cumsum of dt*A (fp32), dtf = dt as fp32, both [B,H,nc,Q]; dt here is the
// step size after the optional bias / softplus, which every later stage reads from dtf or the decay tables.
// One block per (chunk, batch): thread q reads the H contiguous dt values of position q once and
// the block scans 8 heads at a time with warp shuffles.
template <typename T>
__global__ void __launch_bounds__(NT) k_cumsum(Geo g, const T* __restrict__ dt, const float* __restrict__ dt_bias,
                                               const float* __restrict__ A, float* __restrict__ cs,
                                               float* __restrict__ dtf, float* __restrict__ tab, int* __restrict__ hmax,
                                               int tag, int* __restrict__ status) {
  pdl_wait();
  constexpr int HG = 8;
  const int c = blockIdx.x, b = blockIdx.y, q = threadIdx.x;
  __shared__ float wsum[NT / 32][HG];
  const int t = c * g.Q + q;
  if (c == 0 && b == 0 && q == 0) {   // first kernel of a pass: the status word and the tag of this launch
    *status = 0;
    if (hmax) hmax[g.H] = tag;
  }
  const bool live = (q < g.Q) && (t < g.L);
  const int lane = q & 31, w = q >> 5;
  const T* row = dt + b * g.dtsb + (long long)t * g.dtsl;
  for (int h0 = 0; h0 < g.H; h0 += HG) {
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
        // per head: does any chunk of the call accumulate a decay exponent beyond the range inside which dB/dC may carry the
        // decay on the operands?  Only then this launch's tag is written to the head's word (plain store), so the usual case
        // costs nothing and nothing has to be zeroed.
        if (hmax && h < g.H && q == g.Q - 1 && fabsf(v[k]) > SSD_SEP_LOG_RANGE) hmax[h] = tag;
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
// Stage 2 (and its backward twin): out[b,c,h,p,n] = sum_l w_l * X[l,h,p] * Y[l,g,n]
//   MODE 0: w_l = exp(cs_end - cs_l) * dt_l   (chunk_state: X = x, Y = B)
//   MODE 1: w_l = exp(cs_l)                    (local state gradient: X = dy, Y = C)
template <typename T, int MODE>
__global__ void __launch_bounds__(NT) k_chunk_state(Geo g, const T* __restrict__ x, long long xsb, long long xsl,
                                                    DySrc<T> dys, const T* __restrict__ Y, long long ysb,
                                                    long long ysl, const float* __restrict__ cs,
                                                    const float* __restrict__ dtf, float* __restrict__ out) {
  pdl_wait();
  __shared__ __align__(16) float As[TK * LDS];
  __shared__ __align__(16) float Bs[TK * LDS];
  __shared__ float wl[256];
  const int ntn = (g.N + TN - 1) / TN;
  const int p0 = (blockIdx.x / ntn) * TM, n0 = (blockIdx.x % ntn) * TN;
  const int c = blockIdx.y / g.H, h = blockIdx.y % g.H, b = blockIdx.z, grp = h / g.hpg;
  const size_t co = cs_idx(g, b, h, c);
  const float cs_end = cs[co + g.Q - 1];
  for (int l = threadIdx.x; l < g.Q; l += NT)
    wl[l] = (MODE == 0) ? expf(cs_end - cs[co + l]) * dtf[co + l] : expf(cs[co + l]);
  __syncthreads();
  float acc[4][4];
  zero_acc(acc);
  const int tbase = c * g.Q;
  auto fa = [&](int m, int k) -> float {
    const int p = p0 + m, t = tbase + k;
    if (p >= g.P || t >= g.L) return 0.f;
    float v = (MODE == 0) ? ldf(x + b * xsb + t * xsl + (long long)h * g.P + p) : dys.get(g, b, t, h, p);
    return v * wl[k];
  };
  auto fb = [&](int n, int k) -> float {
    const int nn = n0 + n, t = tbase + k;
    if (nn >= g.N || t >= g.L) return 0.f;
    return ldf(Y + b * ysb + t * ysl + (long long)grp * g.N + nn);
  };
  tile_mac<false, false>(acc, 0, g.Q, fa, fb, As, Bs);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float* o = out + st_idx(g, b, c, h);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int p = p0 + ty * 4 + r;
    if (p >= g.P) continue;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      const int n = n0 + tx * 4 + cc;
      if (n < g.N) o[(size_t)p * g.N + n] = acc[r][cc];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Stage 3: exclusive scan over chunks, in place.  Forward direction turns per-chunk states into
// the state ENTERING each chunk and emits the final state; reverse direction does the same for
// the state gradient (entering from the right) and emits the gradient of the initial state.
//   WRITE=false only produces `last` (used by the sequence-parallel split to get the slice total).
template <bool WRITE>
__global__ void __launch_bounds__(NT) k_state_passing(Geo g, float* __restrict__ st, const float* __restrict__ cs,
                                                      const float* __restrict__ init, float* __restrict__ last,
                                                      float* __restrict__ last2, int reverse) {
  pdl_wait();
  const int e = blockIdx.x * NT + threadIdx.x, h = blockIdx.y, b = blockIdx.z;
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
// Stage 4a: cb[b,c,g,i,j] = C_i . B_j for j-tiles at or below the diagonal.
template <typename T>
__global__ void __launch_bounds__(NT) k_cb(Geo g, const T* __restrict__ Bm, const T* __restrict__ Cm,
                                           float* __restrict__ cb) {
  pdl_wait();
  __shared__ __align__(16) float As[TK * LDS];
  __shared__ __align__(16) float Bs[TK * LDS];
  const int nt = (g.Q + TM - 1) / TM;
  const int it = blockIdx.x / nt, jt = blockIdx.x % nt;
  if (jt > it) return;
  const int i0 = it * TM, j0 = jt * TN;
  const int c = blockIdx.y / g.G, grp = blockIdx.y % g.G, b = blockIdx.z;
  const int tbase = c * g.Q;
  float acc[4][4];
  zero_acc(acc);
  auto fa = [&](int m, int k) -> float {
    const int i = i0 + m, t = tbase + i;
    if (i >= g.Q || t >= g.L) return 0.f;
    return ldf(Cm + b * g.csb + t * g.csl + (long long)grp * g.N + k);
  };
  auto fb = [&](int n, int k) -> float {
    const int j = j0 + n, t = tbase + j;
    if (j >= g.Q || t >= g.L) return 0.f;
    return ldf(Bm + b * g.bsb + t * g.bsl + (long long)grp * g.N + k);
  };
  tile_mac<true, true>(acc, 0, g.N, fa, fb, As, Bs);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float* o = cb + cb_idx(g, b, c, grp);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + ty * 4 + r;
    if (i >= g.Q) continue;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      const int j = j0 + tx * 4 + cc;
      if (j < g.Q) o[(size_t)i * g.Q + j] = acc[r][cc];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Stage 4b: chunk_scan.  acc[i,p] = sum_{j<=i} cb[i,j] exp(cs_i-cs_j) dt_j x[j,p]
//                                   + exp(cs_i) sum_n C[i,n] prev[p,n]
//   EPI 0 (forward):  y = acc + D x, optional silu gate, store.
//   EPI 1 (backward recompute): from acc form dz and the pre-gate gradient, and the per-position
//                     sums  dcsp[i] = sum_p dyp*acc  and  ddot[i] = sum_p dyp*x.
template <typename T, int EPI>
__global__ void __launch_bounds__(NT) k_chunk_scan(Geo g, const T* __restrict__ x, const T* __restrict__ Cm,
                                                   const float* __restrict__ D, const T* __restrict__ z,
                                                   const float* __restrict__ cs, const float* __restrict__ dtf,
                                                   const float* __restrict__ cb, const float* __restrict__ prev,
                                                   T* __restrict__ y, const T* __restrict__ dy,
                                                   float* __restrict__ dyp, T* __restrict__ dz,
                                                   float* __restrict__ dcsp, float* __restrict__ ddot) {
  pdl_wait();
  __shared__ __align__(16) float As[TK * LDS];
  __shared__ __align__(16) float Bs[TK * LDS];
  __shared__ float css[256], dts[256];
  const int ntp = (g.P + TN - 1) / TN;
  const int i0 = (blockIdx.x / ntp) * TM, p0 = (blockIdx.x % ntp) * TN;
  const int c = blockIdx.y / g.H, h = blockIdx.y % g.H, b = blockIdx.z, grp = h / g.hpg;
  const int tbase = c * g.Q;
  const size_t co = cs_idx(g, b, h, c);
  for (int l = threadIdx.x; l < g.Q; l += NT) { css[l] = cs[co + l]; dts[l] = dtf[co + l]; }
  __syncthreads();
  float acc[4][4];
  zero_acc(acc);
  const float* cbp = cb + cb_idx(g, b, c, grp);
  {
    auto fa = [&](int m, int k) -> float {
      const int i = i0 + m;
      if (i >= g.Q || k > i) return 0.f;
      return cbp[(size_t)i * g.Q + k] * expf(css[i] - css[k]) * dts[k];
    };
    auto fb = [&](int n, int k) -> float {
      const int p = p0 + n, t = tbase + k;
      if (p >= g.P || t >= g.L) return 0.f;
      return ldf(x + b * g.xsb + t * g.xsl + (long long)h * g.P + p);
    };
    const int kend = min(g.Q, i0 + TM);
    tile_mac<true, false>(acc, 0, kend, fa, fb, As, Bs);
  }
  {
    const float* pv = prev + st_idx(g, b, c, h);
    auto fa = [&](int m, int k) -> float {
      const int i = i0 + m, t = tbase + i;
      if (i >= g.Q || t >= g.L) return 0.f;
      return expf(css[i]) * ldf(Cm + b * g.csb + t * g.csl + (long long)grp * g.N + k);
    };
    auto fb = [&](int n, int k) -> float {
      const int p = p0 + n;
      if (p >= g.P) return 0.f;
      return pv[(size_t)p * g.N + k];
    };
    tile_mac<true, true>(acc, 0, g.N, fa, fb, As, Bs);
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const float Dh = D ? D[h] : 0.f;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + ty * 4 + r, t = tbase + i;
    const bool rowok = (i < g.Q) && (t < g.L);
    float s_cs = 0.f, s_dd = 0.f;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      const int p = p0 + tx * 4 + cc;
      if (!rowok || p >= g.P) continue;
      const float xv = ldf(x + b * g.xsb + t * g.xsl + (long long)h * g.P + p);
      if (EPI == 0) {
        float v = acc[r][cc] + Dh * xv;
        if (z) {
          const float zv = ldf(z + b * g.zsb + t * g.zsl + (long long)h * g.P + p);
          v *= zv * sigmoidf_(zv);
        }
        stf(y + b * g.ysb + t * g.ysl + (long long)h * g.P + p, v);
      } else {
        float dyv = ldf(dy + b * g.ysb + t * g.ysl + (long long)h * g.P + p);
        if (z) {
          const float zv = ldf(z + b * g.zsb + t * g.zsl + (long long)h * g.P + p);
          const float sg = 1.f / (1.f + expf(-zv));
          const float ypre = acc[r][cc] + Dh * xv;
          const size_t od = ((size_t)(b * (size_t)g.L + t) * g.H + h) * g.P + p;
          stf(dz + od, dyv * ypre * sg * (1.f + zv * (1.f - sg)));
          dyv *= zv * sg;
          dyp[od] = dyv;
        }
        s_cs += dyv * acc[r][cc];
        s_dd += dyv * xv;
      }
    }
    if (EPI == 1) {
      s_cs = row_reduce16(s_cs);
      s_dd = row_reduce16(s_dd);
      if (tx == 0 && rowok) {
        atomicAdd(dcsp + co + i, s_cs);
        atomicAdd(ddot + co + i, s_dd);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Backward, dx:  u[j,p] = sum_{i>=j} cb[i,j] exp(cs_i-cs_j) dyp[i,p] + exp(cs_end-cs_j) sum_n B[j,n] dS[p,n]
//                dx = D*dyp + dt_j*u ;  ddtd[j] = sum_p x[j,p]*u[j,p]
template <typename T>
__global__ void __launch_bounds__(NT) k_dx(Geo g, const T* __restrict__ x, const T* __restrict__ Bm,
                                           const float* __restrict__ D, DySrc<T> dys,
                                           const float* __restrict__ cs, const float* __restrict__ dtf,
                                           const float* __restrict__ cb, const float* __restrict__ dS,
                                           T* __restrict__ dx, float* __restrict__ ddtd) {
  pdl_wait();
  __shared__ __align__(16) float As[TK * LDS];
  __shared__ __align__(16) float Bs[TK * LDS];
  __shared__ float css[256];
  const int ntp = (g.P + TN - 1) / TN;
  const int j0 = (blockIdx.x / ntp) * TM, p0 = (blockIdx.x % ntp) * TN;
  const int c = blockIdx.y / g.H, h = blockIdx.y % g.H, b = blockIdx.z, grp = h / g.hpg;
  const int tbase = c * g.Q;
  const size_t co = cs_idx(g, b, h, c);
  for (int l = threadIdx.x; l < g.Q; l += NT) css[l] = cs[co + l];
  __syncthreads();
  const float cs_end = css[g.Q - 1];
  float acc[4][4];
  zero_acc(acc);
  const float* cbp = cb + cb_idx(g, b, c, grp);
  {
    auto fa = [&](int m, int k) -> float {  // m -> j, k -> i
      const int j = j0 + m;
      if (j >= g.Q || k < j) return 0.f;
      return cbp[(size_t)k * g.Q + j] * expf(css[k] - css[j]);
    };
    auto fb = [&](int n, int k) -> float {
      const int p = p0 + n, t = tbase + k;
      if (p >= g.P || t >= g.L) return 0.f;
      return dys.get(g, b, t, h, p);
    };
    tile_mac<false, false>(acc, j0, g.Q, fa, fb, As, Bs);
  }
  {
    const float* ds = dS + st_idx(g, b, c, h);
    auto fa = [&](int m, int k) -> float {
      const int j = j0 + m, t = tbase + j;
      if (j >= g.Q || t >= g.L) return 0.f;
      return expf(cs_end - css[j]) * ldf(Bm + b * g.bsb + t * g.bsl + (long long)grp * g.N + k);
    };
    auto fb = [&](int n, int k) -> float {
      const int p = p0 + n;
      if (p >= g.P) return 0.f;
      return ds[(size_t)p * g.N + k];
    };
    tile_mac<true, true>(acc, 0, g.N, fa, fb, As, Bs);
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const float Dh = D ? D[h] : 0.f;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int j = j0 + ty * 4 + r, t = tbase + j;
    const bool rowok = (j < g.Q) && (t < g.L);
    const float dtj = rowok ? dtf[co + j] : 0.f;
    float s = 0.f;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      const int p = p0 + tx * 4 + cc;
      if (!rowok || p >= g.P) continue;
      const float xv = ldf(x + b * g.xsb + t * g.xsl + (long long)h * g.P + p);
      const float u = acc[r][cc];
      const float dyv = dys.get(g, b, t, h, p);
      stf(dx + ((size_t)(b * (size_t)g.L + t) * g.H + h) * g.P + p, Dh * dyv + dtj * u);
      s += xv * u;
    }
    s = row_reduce16(s);
    if (tx == 0 && rowok) atomicAdd(ddtd + co + j, s);
  }
}

// ---------------------------------------------------------------------------------------------
// Backward, W:  wsum[b,c,g,i,j] = sum_{h in g} exp(cs_h,i-cs_h,j) dt_h,j (dyp[i,h,:] . x[j,h,:]),  j<=i
template <typename T>
__global__ void __launch_bounds__(NT) k_dw(Geo g, const T* __restrict__ x, DySrc<T> dys,
                                           const float* __restrict__ cs, const float* __restrict__ dtf,
                                           float* __restrict__ wsum) {
  pdl_wait();
  __shared__ __align__(16) float As[TK * LDS];
  __shared__ __align__(16) float Bs[TK * LDS];
  const int nt = (g.Q + TM - 1) / TM;
  const int it = blockIdx.x / nt, jt = blockIdx.x % nt;
  if (jt > it) return;
  const int i0 = it * TM, j0 = jt * TN;
  const int c = blockIdx.y / g.G, grp = blockIdx.y % g.G, b = blockIdx.z;
  const int tbase = c * g.Q;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float sum[4][4];
  zero_acc(sum);
  for (int hh = 0; hh < g.hpg; ++hh) {
    const int h = grp * g.hpg + hh;
    float acc[4][4];
    zero_acc(acc);
    auto fa = [&](int m, int k) -> float {
      const int i = i0 + m, t = tbase + i;
      if (i >= g.Q || t >= g.L) return 0.f;
      return dys.get(g, b, t, h, k);
    };
    auto fb = [&](int n, int k) -> float {
      const int j = j0 + n, t = tbase + j;
      if (j >= g.Q || t >= g.L) return 0.f;
      return ldf(x + b * g.xsb + t * g.xsl + (long long)h * g.P + k);
    };
    tile_mac<true, true>(acc, 0, g.P, fa, fb, As, Bs);
    const size_t co = cs_idx(g, b, h, c);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = i0 + ty * 4 + r;
      if (i >= g.Q) continue;
      const float ci = cs[co + i];
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        const int j = j0 + tx * 4 + cc;
        if (j < g.Q && j <= i) sum[r][cc] += acc[r][cc] * expf(ci - cs[co + j]) * dtf[co + j];
      }
    }
  }
  float* o = wsum + cb_idx(g, b, c, grp);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + ty * 4 + r;
    if (i >= g.Q) continue;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      const int j = j0 + tx * 4 + cc;
      if (j < g.Q) o[(size_t)i * g.Q + j] = (j <= i) ? sum[r][cc] : 0.f;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Backward, dC (MODE 0) and dB (MODE 1):
//   dC[i,n] = sum_{j<=i} wsum[i,j] B[j,n] + sum_{h,p} exp(cs_h,i) dyp[i,h,p] prev[h,p,n]
//   dB[j,n] = sum_{i>=j} wsum[i,j] C[i,n] + sum_{h,p} exp(cs_h,end-cs_h,j) dt_h,j x[j,h,p] dS[h,p,n]
template <typename T, int MODE>
__global__ void __launch_bounds__(NT) k_dbc(Geo g, const T* __restrict__ x, const T* __restrict__ Other,
                                            long long osb, long long osl, DySrc<T> dys,
                                            const float* __restrict__ cs, const float* __restrict__ dtf,
                                            const float* __restrict__ wsum, const float* __restrict__ st,
                                            T* __restrict__ out) {
  pdl_wait();
  __shared__ __align__(16) float As[TK * LDS];
  __shared__ __align__(16) float Bs[TK * LDS];
  const int ntn = (g.N + TN - 1) / TN;
  const int r0 = (blockIdx.x / ntn) * TM, n0 = (blockIdx.x % ntn) * TN;
  const int c = blockIdx.y / g.G, grp = blockIdx.y % g.G, b = blockIdx.z;
  const int tbase = c * g.Q;
  float acc[4][4];
  zero_acc(acc);
  const float* wp = wsum + cb_idx(g, b, c, grp);
  {
    auto fa = [&](int m, int k) -> float {
      const int rr = r0 + m;
      if (rr >= g.Q) return 0.f;
      if (MODE == 0) return (k <= rr) ? wp[(size_t)rr * g.Q + k] : 0.f;
      return (k >= rr) ? wp[(size_t)k * g.Q + rr] : 0.f;
    };
    auto fb = [&](int n, int k) -> float {
      const int nn = n0 + n, t = tbase + k;
      if (nn >= g.N || t >= g.L) return 0.f;
      return ldf(Other + b * osb + t * osl + (long long)grp * g.N + nn);
    };
    if (MODE == 0) tile_mac<true, false>(acc, 0, min(g.Q, r0 + TM), fa, fb, As, Bs);
    else tile_mac<false, false>(acc, r0, g.Q, fa, fb, As, Bs);
  }
  {
    const int K2 = g.hpg * g.P;
    auto fa = [&](int m, int k) -> float {
      const int rr = r0 + m, t = tbase + rr;
      if (rr >= g.Q || t >= g.L) return 0.f;
      const int h = grp * g.hpg + k / g.P, p = k % g.P;
      const size_t co = cs_idx(g, b, h, c);
      if (MODE == 0) return expf(cs[co + rr]) * dys.get(g, b, t, h, p);
      return expf(cs[co + g.Q - 1] - cs[co + rr]) * dtf[co + rr] *
             ldf(x + b * g.xsb + t * g.xsl + (long long)h * g.P + p);
    };
    auto fb = [&](int n, int k) -> float {
      const int nn = n0 + n;
      if (nn >= g.N) return 0.f;
      const int h = grp * g.hpg + k / g.P, p = k % g.P;
      return st[st_idx(g, b, c, h) + (size_t)p * g.N + nn];
    };
    tile_mac<true, false>(acc, 0, K2, fa, fb, As, Bs);
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int rr = r0 + ty * 4 + r, t = tbase + rr;
    if (rr >= g.Q || t >= g.L) continue;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      const int n = n0 + tx * 4 + cc;
      if (n < g.N) stf(out + ((size_t)(b * (size_t)g.L + t) * g.G + grp) * g.N + n, acc[r][cc]);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Backward: sdot[b,c,h] = <dS_end_c, S_end_c>, with S_end_c = state entering chunk c+1 (or final).
__global__ void __launch_bounds__(NT) k_sdot(Geo g, const float* __restrict__ dS, const float* __restrict__ prev,
                                             const float* __restrict__ fin, float* __restrict__ sdot) {
  pdl_wait();
  const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int PN = g.P * g.N;
  const float* a = dS + st_idx(g, b, c, h);
  const float* s = (c + 1 < g.nc) ? prev + st_idx(g, b, c + 1, h) : fin + ((size_t)(b * g.H + h)) * PN;
  float v = 0.f;
  for (int e = threadIdx.x; e < PN; e += NT) v = fmaf(a[e], s[e], v);
  __shared__ float red[NT / 32];
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < NT / 32; ++i) t += red[i];
    sdot[(size_t)(b * g.nc + c) * g.H + h] = t;
  }
}

// ---------------------------------------------------------------------------------------------
// Backward: da_k = sum_{i>=k in chunk}(dcsp_i - dt_i*ddtd_i) + sdot ; ddt_k = ddtd_k + A*da_k (times the derivative
// of the step-size activation when dt_softplus is set) ;
// per-chunk partial sums for dA (= sum dt*da) and dD (= sum ddot).  One block per (chunk, batch),
// 8 heads at a time; sdot arrives as `nw` partial sums per (batch, chunk, head), added in fixed order.
__global__ void __launch_bounds__(NT) k_ddt(Geo g, const float* __restrict__ A, const float* __restrict__ dtf,
                                            const float* __restrict__ dcsp, const float* __restrict__ ddtd,
                                            const float* __restrict__ ddot, const float* __restrict__ sdot, int nw,
                                            float* __restrict__ ddt, float* __restrict__ dapart,
                                            float* __restrict__ ddpart, float* __restrict__ dbpart) {
  pdl_wait();
  constexpr int HG = 8;
  const int c = blockIdx.x, b = blockIdx.y, q = threadIdx.x;
  __shared__ float wsum[NT / 32][HG], red1[NT / 32][HG], red2[NT / 32][HG], red3[NT / 32][HG], ssd[HG];
  const int qr = g.Q - 1 - q;   // reversed position: an inclusive prefix scan over q is a suffix sum over qr
  const bool ok = (q < g.Q);
  const int lane = q & 31, w = q >> 5, nwarp = blockDim.x >> 5;   // launched with 128 threads when the chunk is <= 128 long
  const int t = c * g.Q + qr;
  for (int h0 = 0; h0 < g.H; h0 += HG) {
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
    float d[HG], dd[HG], v[HG], s2[HG];
#pragma unroll
    for (int k = 0; k < HG; ++k) {
      const int h = h0 + k;
      const bool live = ok && h < g.H;
      const size_t o = live ? cs_idx(g, b, h, c) + qr : 0;
      d[k] = live ? dtf[o] : 0.f;
      dd[k] = live ? ddtd[o] : 0.f;
      v[k] = live ? dcsp[o] - d[k] * dd[k] : 0.f;
      s2[k] = live ? ddot[o] : 0.f;
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
    float s1[HG];
#pragma unroll
    for (int k = 0; k < HG; ++k) {
      float base = 0.f;
      for (int i = 0; i < w; ++i) base += wsum[i][k];
      const float da = v[k] + base + ssd[k];
      s1[k] = ok ? d[k] * da : 0.f;
      v[k] = dd[k] + ((h0 + k < g.H) ? A[h0 + k] : 0.f) * da;   // gradient w.r.t. the step size of this position
      // ... and through softplus to the dt that was passed in: softplus'(r) = sigmoid(r) = 1 - exp(-softplus(r))
      if (g.dt_softplus) v[k] *= 1.f - __expf(-d[k]);
    }
    if (ok && t < g.L) {
      float* o = ddt + ((size_t)b * g.L + t) * g.H + h0;
      if (h0 + HG <= g.H && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
        reinterpret_cast<float4*>(o)[0] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(o)[1] = make_float4(v[4], v[5], v[6], v[7]);
      } else {
#pragma unroll
        for (int k = 0; k < HG; ++k)
          if (h0 + k < g.H) o[k] = v[k];
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
#pragma unroll
      for (int k = 0; k < HG; ++k) {
        s1[k] += __shfl_xor_sync(0xffffffffu, s1[k], o);
        s2[k] += __shfl_xor_sync(0xffffffffu, s2[k], o);
      }
    }
    if (dbpart) {   // the chunk's share of the step-size bias gradient
#pragma unroll
      for (int k = 0; k < HG; ++k) {
        float s3 = (ok && t < g.L) ? v[k] : 0.f;
#pragma unroll
        for (int o = 16; o; o >>= 1) s3 += __shfl_xor_sync(0xffffffffu, s3, o);
        if (lane == 0) red3[w][k] = s3;
      }
    }
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < HG; ++k) { red1[w][k] = s1[k]; red2[w][k] = s2[k]; }
    }
    __syncthreads();
    if (q < HG && h0 + q < g.H) {
      float a1 = 0.f, a2 = 0.f;
      for (int i = 0; i < nwarp; ++i) { a1 += red1[i][q]; a2 += red2[i][q]; }
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
  const int tp = cdiv(g.P, TM), tn = cdiv(g.N, TN), tq = cdiv(g.Q, TM);
  // a full pass (no sequence-parallel staging) computes the chunk states inside the scan over chunks where that kernel applies
  const bool fused = tc && stages == (SSD_STAGE_LOCAL | SSD_STAGE_FINISH) && tensor_state_fused_applies(g);
  if (stages & (SSD_STAGE_LOCAL | SSD_STAGE_LOCAL_STATES)) {
    int* hmax = tc ? (int*)(ws + w.hmax) : nullptr;
    static std::atomic<int> launch_tag{1};
    int tag = launch_tag.fetch_add(1, std::memory_order_relaxed);
    if (tag == 0) tag = launch_tag.fetch_add(1, std::memory_order_relaxed);
    launch<k_cumsum<T>>(dim3(g.nc, g.B), g.Q <= 128 ? 128 : NT, 0, s, g, (const T*)p.dt, p.dt_bias, p.A, cs, dtf, tc ? tab : nullptr,
                        hmax, tag, status);
    SSD_CUDA_CHECK_LAUNCH("cumsum");
    if (tc && fused) {
      // chunk states and the scan over chunks run as one kernel in the FINISH stage
    } else if (tc) {
      int rc = tensor_chunk_state(g, 0, p.x, g.xsb, g.xsl, p.Bm, g.bsb, g.bsl, tab, states, status, s);
      if (rc) return rc;
    } else {
      DySrc<T> none{nullptr, nullptr, 0, 0};
      launch<k_chunk_state<T, 0>>(dim3(tp * tn, g.nc * g.H, g.B), NT, 0, s, g, x, g.xsb, g.xsl, none, (const T*)p.Bm, g.bsb, g.bsl, cs, dtf, states);
      SSD_CUDA_CHECK_LAUNCH("chunk_state");
    }
  }
  if (stages & SSD_STAGE_TOTAL) {
    if (tc) {
      int rc = tensor_state_passing(g, states, cs, nullptr, fin, fin2, nullptr, 0, false, nullptr, nullptr, nullptr, nullptr, nullptr, s);
      if (rc) return rc;
    } else {
      launch<k_state_passing<false>>(dim3(cdiv(g.P * g.N, NT), g.H, g.B), NT, 0, s, g, states, cs, nullptr, fin, fin2, 0);
      SSD_CUDA_CHECK_LAUNCH("state_total");
    }
  }
  if (stages & SSD_STAGE_FINISH) {
    if (tc && fused) {
      // no fp32 copy of the chunk-entry states: every reader in this family takes the bf16 one
      int rc = tensor_state_fused(g, 0, p.x, g.xsb, g.xsl, p.Bm, g.bsb, g.bsl, tab, nullptr, prev_bf,
                                  p.init_state, fin, fin2, nullptr, nullptr, nullptr, nullptr, status, s);
      if (rc) return rc;
    } else if (tc) {
      int rc = tensor_state_passing(g, states, cs, p.init_state, fin, fin2, prev_bf, 0, true, nullptr, nullptr, nullptr, nullptr, nullptr, s);
      if (rc) return rc;
    } else {
      launch<k_state_passing<true>>(dim3(cdiv(g.P * g.N, NT), g.H, g.B), NT, 0, s, g, states, cs, p.init_state, fin, fin2, 0);
      SSD_CUDA_CHECK_LAUNCH("state_passing");
    }
    if (!tc) {
      launch<k_cb<T>>(dim3(tq * tq, g.nc * g.G, g.B), NT, 0, s, g, (const T*)p.Bm, (const T*)p.Cm, cb);
      SSD_CUDA_CHECK_LAUNCH("cb");
    }
    if (p.y && tc) {
      int rc = tensor_chunk_scan(g, p, tab, prev_bf, status, s);
      if (rc) return rc;
    } else if (p.y) {
      launch<k_chunk_scan<T, 0>>(dim3(tq * tp, g.nc * g.H, g.B), NT, 0, s, g, x, (const T*)p.Cm, p.D, (const T*)p.z, cs, dtf, cb, states,
                                 (T*)p.y, nullptr, nullptr, nullptr, nullptr, nullptr);
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
  const int tp = cdiv(g.P, TM), tn = cdiv(g.N, TN), tq = cdiv(g.Q, TM);
  DySrc<T> dys{p.z ? dyp : nullptr, (const T*)p.dy, g.ysb, g.ysl};
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
    if (!tc) {  // the CUDA-core kernels accumulate these row sums with atomics; the tensor-core ones store them
      const size_t nq = (size_t)g.B * g.H * g.nc * g.Q * sizeof(float);
      cudaMemsetAsync(dcsp, 0, nq, s);
      cudaMemsetAsync(ddtd, 0, nq, s);
      cudaMemsetAsync(ddot, 0, nq, s);
    }
  }
  if (do_recompute) {
    if (tc) {
      // ungated (dstate 64, or dstate 128): the recompute pass is folded into the dx kernel of the FINISH stage
      int rc = tensor_bwd_merged_applies(g, p) ? SSD_OK : tensor_scan_bwd(g, p, tab, prev_bf, dyp, dcsp, ddot, status, s);
      if (rc) return rc;
    } else {
      // forward recompute with the backward epilogue: dz, pre-gate dy, dcsp, ddot
      launch<k_chunk_scan<T, 1>>(dim3(tq * tp, g.nc * g.H, g.B), NT, 0, s, g, x, (const T*)p.Cm, p.D, (const T*)p.z, cs, dtf, cb, states,
                                 nullptr, (const T*)p.dy, dyp, (T*)p.dz, dcsp, ddot);
      SSD_CUDA_CHECK_LAUNCH("chunk_scan_bwd_epilogue");
    }
  }
  if (want_states) {
    if (tc) {
      if (!fused) {
        int rc = tensor_chunk_state(g, 1, tc_dy, tc_dense ? (long long)g.L * g.H * g.P : g.ysb,
                                    tc_dense ? (long long)g.H * g.P : g.ysl, p.Cm, g.csb, g.csl, tab, dst, status, s);
        if (rc) return rc;
      }
    } else {
      launch<k_chunk_state<T, 1>>(dim3(tp * tn, g.nc * g.H, g.B), NT, 0, s, g, x, g.xsb, g.xsl, dys, (const T*)p.Cm, g.csb, g.csl, cs, dtf, dst);
      SSD_CUDA_CHECK_LAUNCH("dstates_local");
    }
  }
  if (stages & SSD_STAGE_TOTAL) {
    if (tc) {
      int rc = tensor_state_passing(g, dst, cs, nullptr, dini, nullptr, nullptr, 1, false, nullptr, nullptr, nullptr, nullptr, nullptr, s);
      if (rc) return rc;
    } else {
      launch<k_state_passing<false>>(dim3(cdiv(g.P * g.N, NT), g.H, g.B), NT, 0, s, g, dst, cs, nullptr, dini, nullptr, 1);
      SSD_CUDA_CHECK_LAUNCH("dstate_total");
    }
  }
  int sdot_nw = 1;
  if (stages & SSD_STAGE_FINISH) {
    if (tc && fused) {
      // local state gradients, the reverse scan and the <dS_end, S_end> partial sums in one kernel (no fp32 copy is kept)
      int rc = tensor_state_fused(g, 1, tc_dy, tc_dense ? (long long)g.L * g.H * g.P : g.ysb,
                                  tc_dense ? (long long)g.H * g.P : g.ysl, p.Cm, g.csb, g.csl, tab, nullptr, ds_bf,
                                  p.dfinal_state, dini, nullptr, prev_bf, fin, sdot, &sdot_nw, status, s);
      if (rc) return rc;
    } else if (tc) {
      // the reverse scan also leaves the warp-partial sums of <dS_end, S_end> per chunk
      int rc = tensor_state_passing(g, dst, cs, p.dfinal_state, dini, nullptr, ds_bf, 1, true, states, prev_bf, fin, sdot, &sdot_nw, s);
      if (rc) return rc;
    } else {
      launch<k_state_passing<true>>(dim3(cdiv(g.P * g.N, NT), g.H, g.B), NT, 0, s, g, dst, cs, p.dfinal_state, dini, nullptr, 1);
      SSD_CUDA_CHECK_LAUNCH("dstate_passing");
      launch<k_sdot>(dim3(g.nc, g.H, g.B), NT, 0, s, g, dst, states, fin, sdot);
      SSD_CUDA_CHECK_LAUNCH("sdot");
    }
    if (tc) {
      int rc = tensor_bwd_merged_applies(g, p) ? tensor_bwd_merged(g, p, tab, prev_bf, ds_bf, dcsp, ddot, ddtd, status, s)
                                                : tensor_dx(g, p, tc_dy, tc_dense, tab, ds_bf, ddtd, status, s);
      if (rc) return rc;
      rc = tensor_dbc(g, p, tc_dy, tc_dense, tab, (const float*)(ws + w.hmax), prev_bf, ds_bf, status, s);
      if (rc) return rc;
    } else {
      launch<k_dx<T>>(dim3(tq * tp, g.nc * g.H, g.B), NT, 0, s, g, x, (const T*)p.Bm, p.D, dys, cs, dtf, cb, dst, (T*)p.dx, ddtd);
      SSD_CUDA_CHECK_LAUNCH("dx");
      launch<k_dw<T>>(dim3(tq * tq, g.nc * g.G, g.B), NT, 0, s, g, x, dys, cs, dtf, wsum);
      SSD_CUDA_CHECK_LAUNCH("dw");
      launch<k_dbc<T, 0>>(dim3(tq * tn, g.nc * g.G, g.B), NT, 0, s, g, x, (const T*)p.Bm, g.bsb, g.bsl, dys, cs, dtf, wsum, states, (T*)p.dC);
      SSD_CUDA_CHECK_LAUNCH("dC");
      launch<k_dbc<T, 1>>(dim3(tq * tn, g.nc * g.G, g.B), NT, 0, s, g, x, (const T*)p.Cm, g.csb, g.csl, dys, cs, dtf, wsum, dst, (T*)p.dB);
      SSD_CUDA_CHECK_LAUNCH("dB");
    }
    float* dbpart = p.ddt_bias ? (float*)(ws + w.dbpart) : nullptr;
    launch<k_ddt>(dim3(g.nc, g.B), g.Q <= 128 ? 128 : NT, 0, s, g, p.A, dtf, dcsp, ddtd, ddot, sdot, sdot_nw, p.ddt, dapart, ddpart, dbpart);
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
