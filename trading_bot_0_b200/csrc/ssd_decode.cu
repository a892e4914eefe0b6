// Streamed-rollout kernels: the single-timestep state update (in place on the caller's fp32
// state), per-stream state reset, and the small sequence-parallel prefix kernels.
//
// state_update is a pure HBM stream: every state element is read once and written once per
// step (2*H*P*N*4 bytes per stream) and the per-step vectors are tiny beside it.  Each thread
// moves 128-bit pieces of a state row; a row's dot product with C is finished with shuffles
// inside the lanes that share the row.
#include "common.cuh"
#include "ssd_internal.h"

namespace ssd {
namespace {

constexpr int DEC_THREADS = 128;

template <typename T> struct Vec4Load;
template <> struct Vec4Load<float> {
  static __device__ __forceinline__ float4 ld(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
};
template <> struct Vec4Load<__nv_bfloat16> {
  static __device__ __forceinline__ float4 ld(const __nv_bfloat16* p) {
    const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&r.x);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&r.y);
    const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
  }
};

__device__ __forceinline__ float ldf_shared(const float* p) { return *p; }
__device__ __forceinline__ float ldf_shared(const __nv_bfloat16* p) { return __bfloat162float(*p); }

// One block per (stream, head).  N is a power of two in [16, 256].
//   LPR = lanes that share a state row, V = float4 pieces per lane per row, RPW = rows per warp.
template <typename T, int N>
__global__ void __launch_bounds__(DEC_THREADS, 8) k_state_update(SsdStepDims d, SsdStepPtrs p) {
  pdl_wait();
  constexpr int LPR = (N / 4 < 32) ? N / 4 : 32;
  constexpr int V = N / (4 * LPR);
  constexpr int RPW = 32 / LPR;
  constexpr int RPB = RPW * (DEC_THREADS / 32);  // rows per block pass
  constexpr int UNROLL = 4;
  const int sh = blockIdx.x;
  const int s = sh / d.nheads, h = sh - s * d.nheads;
  const int grp = h / (d.nheads / d.ngroups);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lir = lane % LPR, riw = lane / LPR;
  const int P = d.headdim;

  // The state rows of the first pass are requested before anything else: the step's small vectors (dt, A, B, C, x) sit
  // behind a dependent exp, and a warp that waited for them first would request its state a memory round trip later.
  float* st = p.state + (size_t)sh * P * N;
  float4 sv[UNROLL][V];
  auto load_state = [&](int p0) {
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int pr = p0 + riw + u * RPB;
      if (pr < P) {
#pragma unroll
        for (int v = 0; v < V; ++v)
          sv[u][v] = *reinterpret_cast<const float4*>(st + (size_t)pr * N + 4 * (lir + v * LPR));
      }
    }
  };
  load_state(warp * RPW);

  const T* xs = (const T*)p.x + s * d.x_stride_s + (long long)h * P;
  const float dtv = dt_activation(ldf((const T*)p.dt + s * d.dt_stride_s + h), p.dt_bias ? __ldg(p.dt_bias + h) : 0.f, d.dt_softplus);
  const float a = expf(dtv * __ldg(p.A + h));
  const float Dh = p.D ? __ldg(p.D + h) : 0.f;
  const T* Bp = (const T*)p.Bm + s * d.b_stride_s + (long long)grp * N;
  const T* Cp = (const T*)p.Cm + s * d.c_stride_s + (long long)grp * N;
  float4 Bv[V], Cv[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int n = 4 * (lir + v * LPR);
    Bv[v] = Vec4Load<T>::ld(Bp + n);
    Cv[v] = Vec4Load<T>::ld(Cp + n);
  }
  const T* zs = p.z ? (const T*)p.z + s * d.z_stride_s + (long long)h * P : nullptr;
  T* ys = (T*)p.y + s * d.y_stride_s + (long long)h * P;

  for (int p0 = warp * RPW; p0 < P; p0 += RPB * UNROLL) {  // warp-uniform trip count
    const int pbase = p0 + riw;
    if (p0 != warp * RPW) load_state(p0);
    float xv[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int pr = pbase + u * RPB;
      if (pr < P) xv[u] = ldf(xs + pr);
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int pr = pbase + u * RPB;
      float acc = 0.f;
      if (pr < P) {
        const float dx = dtv * xv[u];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          float4 t = sv[u][v];
          t.x = fmaf(a, t.x, dx * Bv[v].x);
          t.y = fmaf(a, t.y, dx * Bv[v].y);
          t.z = fmaf(a, t.z, dx * Bv[v].z);
          t.w = fmaf(a, t.w, dx * Bv[v].w);
          *reinterpret_cast<float4*>(st + (size_t)pr * N + 4 * (lir + v * LPR)) = t;
          acc = fmaf(t.x, Cv[v].x, acc);
          acc = fmaf(t.y, Cv[v].y, acc);
          acc = fmaf(t.z, Cv[v].z, acc);
          acc = fmaf(t.w, Cv[v].w, acc);
        }
      }
#pragma unroll
      for (int o = LPR / 2; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (pr < P && lir == 0) {
        float yv = acc + Dh * xv[u];
        if (zs) {
          const float zv = ldf(zs + pr);
          yv *= zv * sigmoidf_(zv);
        }
        stf(ys + pr, yv);
      }
    }
  }
}

// The same update with the state staged through shared memory.  The work is cut into tiles of one head's state (R * RPB rows
// of N floats: 8 KB, 16 KB at N = 128, wherever the head is that large); a persistent block keeps the next DEC_STAGES - 1 tiles on the way with
// 16-byte cp.async copies, so the bytes in flight per SM are set by the ring (8 blocks x 2 tiles x 8 KB), not by the
// registers a thread can hold.  Bound: HBM, every state byte read and written once.  Measured at 8192 streams x 8 heads of
// 32 x 64: 2 stages (12 blocks per SM) 0.213 ms, 3 stages (8 blocks) 0.175 ms, 4 stages (6 blocks) 0.193 ms, 6 stages
// (4 blocks) 0.223 ms; the register kernel 0.205 ms.  The gate travels in the ring like x (read by the row's lane when it was
// needed it cost 0.03 ms: 0.199 -> 0.168), the row sums are folded together (fold_rows), and at 24 heads of 64 x 128 (1024
// streams) 16 KB tiles took 0.250 ms, 8 KB tiles 0.258, the register kernel 0.254 (gated 0.248, 0.261, 0.274).
constexpr int DEC_STAGES = 3;

// How 128 threads sit on a tile: LPR lanes share a state row, V float4 pieces per lane per row, R rows per thread.
template <int N, int R_>
struct Tile {
  static constexpr int LPR = (N / 4 < 32) ? N / 4 : 32, V = N / (4 * LPR), RPW = 32 / LPR, RPB = RPW * (DEC_THREADS / 32), R = R_;
  static constexpr int ROWS = R * RPB, BYTES = ROWS * N * 4;
};

// The state copies of one tile (as it lies in global memory).
template <class Tl, int N>
__device__ __forceinline__ void tile_request(unsigned char* sm, const float* gst, int row0, int lir) {
#pragma unroll
  for (int u = 0; u < Tl::R; ++u)
#pragma unroll
    for (int v = 0; v < Tl::V; ++v) {
      const int off = (row0 + u * Tl::RPB) * N + 4 * (lir + v * Tl::LPR);
      cp_async16(sm + off * 4, gst + off, true);
    }
}

// One tile: new state to global memory, `out(row, y)` called by one lane of every row.  sx: the tile's x, sB / sC: the group's
// vectors, all in shared memory; a: the step's decay.
template <class Tl, typename T, int N, class Out>
__device__ __forceinline__ void tile_update(const unsigned char* sm, float* gst, const T* sx, const T* sB, const T* sC, float dtv, float a,
                                            float Dh, int row0, int lir, Out out) {
  float Bv[Tl::V][4], Cv[Tl::V][4];
#pragma unroll
  for (int v = 0; v < Tl::V; ++v)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      Bv[v][j] = ldf_shared(sB + 4 * (lir + v * Tl::LPR) + j);
      Cv[v][j] = ldf_shared(sC + 4 * (lir + v * Tl::LPR) + j);
    }
  float acc[Tl::R];
#pragma unroll
  for (int u = 0; u < Tl::R; ++u) {
    const int pr = row0 + u * Tl::RPB;
    const float dx = dtv * ldf_shared(sx + pr);
    acc[u] = 0.f;
#pragma unroll
    for (int v = 0; v < Tl::V; ++v) {
      const int off = pr * N + 4 * (lir + v * Tl::LPR);
      float4 t = *reinterpret_cast<const float4*>(sm + off * 4);
      t.x = fmaf(a, t.x, dx * Bv[v][0]);
      t.y = fmaf(a, t.y, dx * Bv[v][1]);
      t.z = fmaf(a, t.z, dx * Bv[v][2]);
      t.w = fmaf(a, t.w, dx * Bv[v][3]);
      *reinterpret_cast<float4*>(gst + off) = t;
      acc[u] = fmaf(t.x, Cv[v][0], acc[u]);
      acc[u] = fmaf(t.y, Cv[v][1], acc[u]);
      acc[u] = fmaf(t.z, Cv[v][2], acc[u]);
      acc[u] = fmaf(t.w, Cv[v][3], acc[u]);
    }
  }
  int u;
  const float y = fold_rows<Tl::LPR, Tl::R>(acc, lir, u);
  const int pr = row0 + u * Tl::RPB;
  if (lir % (Tl::LPR / Tl::R) == 0) out(pr, fmaf(Dh, ldf_shared(sx + pr), y));
}

// A block's walk over (stream, tile of the stream) with a fixed stride, without divisions in the loop.
struct TileWalk {
  int s, r, ds, dr, per;   // per = tiles of a stream
  __device__ __forceinline__ TileWalk(long long first, long long stride, int per_) : per(per_) {
    s = (int)(first / per_); r = (int)(first - (long long)s * per_);
    ds = (int)(stride / per_); dr = (int)(stride - (long long)ds * per_);
  }
  __device__ __forceinline__ void next() {
    s += ds; r += dr;
    if (r >= per) { r -= per; ++s; }
  }
};

template <typename T, int N, int R, bool GATED>
__global__ void __launch_bounds__(DEC_THREADS) k_state_update_ring(SsdStepDims d, SsdStepPtrs p, int tph) {   // tph: tiles per head
  pdl_wait();
  using Tl = Tile<N, R>;
  constexpr int ES = (int)sizeof(T), X_B = Tl::ROWS * ES, BC_B = N * ES;
  constexpr int STAGE = Tl::BYTES + (GATED ? 2 : 1) * X_B + 2 * BC_B;   // ring slot: state, x, B, C, gate
  constexpr int NXP = X_B / 16, NBP = BC_B / 16;       // 16-byte pieces of x and of B (C); the host checked the divisibility
  extern __shared__ __align__(16) unsigned char dec_ring[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lir = lane % Tl::LPR, row0 = warp * Tl::RPW + lane / Tl::LPR;
  const int hpg = d.nheads / d.ngroups, per = d.nheads * tph;

  auto issue = [&](const TileWalk& w, int stage) {
    if (w.s < d.streams) {
      const int h = tph == 1 ? w.r : w.r / tph, t0 = (w.r - h * tph) * Tl::ROWS;
      unsigned char* sm = dec_ring + stage * STAGE;
      tile_request<Tl, N>(sm, p.state + ((long long)w.s * per + w.r) * (Tl::ROWS * N), row0, lir);
      for (int t = threadIdx.x; t < (GATED ? 2 : 1) * NXP + 2 * NBP; t += DEC_THREADS) {
        const char* src;
        if (t < NXP) src = (const char*)((const T*)p.x + w.s * d.x_stride_s + (long long)h * d.headdim + t0) + t * 16;
        else if (t < NXP + NBP) src = (const char*)((const T*)p.Bm + w.s * d.b_stride_s + (long long)(h / hpg) * N) + (t - NXP) * 16;
        else if (t < NXP + 2 * NBP) src = (const char*)((const T*)p.Cm + w.s * d.c_stride_s + (long long)(h / hpg) * N) + (t - NXP - NBP) * 16;
        else src = (const char*)((const T*)p.z + w.s * d.z_stride_s + (long long)h * d.headdim + t0) + (t - NXP - 2 * NBP) * 16;
        cp_async16(sm + Tl::BYTES + t * 16, src, true);
      }
    }
    cp_async_commit();   // a group per slot even when it is empty: the wait counts groups
  };
  auto load_dt = [&](const TileWalk& w) -> float {   // fetched one tile ahead
    return w.s < d.streams ? ldf((const T*)p.dt + w.s * d.dt_stride_s + (tph == 1 ? w.r : w.r / tph)) : 0.f;
  };

  TileWalk cur(blockIdx.x, gridDim.x, per), ahead = cur, nextw = cur;
#pragma unroll
  for (int k = 0; k < DEC_STAGES - 1; ++k) { issue(ahead, k); ahead.next(); }
  float dt_next = load_dt(nextw);
  int stage = 0;
  while (cur.s < d.streams) {
    cp_async_wait<DEC_STAGES - 2>();
    __syncthreads();     // every thread's pieces of this tile have landed; every thread is done with the previous slot
    issue(ahead, stage == 0 ? DEC_STAGES - 1 : stage - 1);
    ahead.next();
    const float dt_raw = dt_next;
    nextw.next();
    dt_next = load_dt(nextw);
    const int s = cur.s, h = tph == 1 ? cur.r : cur.r / tph;
    const unsigned char* sm = dec_ring + stage * STAGE;
    stage = stage + 1 == DEC_STAGES ? 0 : stage + 1;
    const float dtv = dt_activation(dt_raw, p.dt_bias ? __ldg(p.dt_bias + h) : 0.f, d.dt_softplus);
    const float a = expf(dtv * __ldg(p.A + h));
    const float Dh = p.D ? __ldg(p.D + h) : 0.f;
    const T* sx = reinterpret_cast<const T*>(sm + Tl::BYTES);
    const long long p0 = (long long)h * d.headdim + (cur.r - h * tph) * Tl::ROWS;
    const T* sz = sx + Tl::ROWS + 2 * N;
    T* ys = (T*)p.y + s * d.y_stride_s + p0;
    tile_update<Tl, T, N>(sm, p.state + ((long long)s * per + cur.r) * (Tl::ROWS * N), sx, sx + Tl::ROWS, sx + Tl::ROWS + N, dtv, a, Dh, row0,
                          lir, [&](int row, float yv) {
      if (GATED) {
        const float zv = ldf_shared(sz + row);
        yv *= zv * sigmoidf_(zv);
      }
      stf(ys + row, yv);
    });
    cur.next();
  }
  cp_async_wait<0>();
}

// The step of a rollout whose environments live on the host: x, dt, B and C lie in pinned host memory, one packed row per
// stream, and y goes back to pinned host memory, with no copy in front of or behind the kernel.  A block takes a unit of one
// stream and `hs` of its heads: the unit's part of the row is read over PCIe once, 16 bytes per thread and coalesced, a
// whole unit ahead of its use (registers, then one of two shared-memory slots), the state tiles stream through the ring
// as above, and y leaves in 16-byte stores once the unit is complete.  Bound: max(PCIe, HBM) plus one launch; 24 copy and
// kernel nodes on three streams took 80 us at 1024 streams of 8 x 32 x 64 where the bytes take 20.
template <typename T, int N, int R, int PT>
__global__ void __launch_bounds__(DEC_THREADS) k_state_update_host(SsdStepDims d, SsdStepPtrs p, T* __restrict__ y_host, int tph, int hs,
                                                                   int units) {
  pdl_wait();
  using Tl = Tile<N, R>;
  constexpr int ES = (int)sizeof(T);
  extern __shared__ __align__(16) unsigned char dec_ring[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lir = lane % Tl::LPR, row0 = warp * Tl::RPW + lane / Tl::LPR;
  const int H = d.nheads, P = d.headdim, hpg = H / d.ngroups, ups = H / hs;   // ups: units per stream
  const int x_b = hs * P * ES, dt_b = H * ES, bc_b = d.ngroups * N * ES, row_b = x_b + dt_b + 2 * bc_b;
  unsigned char* rows = dec_ring + DEC_STAGES * Tl::BYTES;   // two slots
  unsigned char* ybuf = rows + 2 * row_b;                    // hs * P values
  const int tiles = hs * tph;                                // of a unit

  uint4 reg[PT];
  auto row_request = [&](int u) {
    if (u >= units) return;
    const long long s = u / ups;
    const int h0 = (u - (int)s * ups) * hs;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
      int o = (threadIdx.x + j * DEC_THREADS) * 16;
      if (o >= row_b) break;
      const char* src;
      if (o < x_b) src = (const char*)((const T*)p.x + s * d.x_stride_s + (long long)h0 * P) + o;
      else if ((o -= x_b) < dt_b) src = (const char*)((const T*)p.dt + s * d.dt_stride_s) + o;
      else if ((o -= dt_b) < bc_b) src = (const char*)((const T*)p.Bm + s * d.b_stride_s) + o;
      else src = (const char*)((const T*)p.Cm + s * d.c_stride_s) + (o - bc_b);
      asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(reg[j].x), "=r"(reg[j].y), "=r"(reg[j].z), "=r"(reg[j].w) : "l"(src));
    }
  };
  auto row_store = [&](unsigned char* slot) {
#pragma unroll
    for (int j = 0; j < PT; ++j) {
      const int o = (threadIdx.x + j * DEC_THREADS) * 16;
      if (o < row_b) *reinterpret_cast<uint4*>(slot + o) = reg[j];
    }
  };

  // the walk of the state ring: tile `at` of unit `au`, two tiles ahead of the one being worked on
  int au = blockIdx.x, at = 0;
  auto issue = [&](int stage) {
    if (au < units) tile_request<Tl, N>(dec_ring + stage * Tl::BYTES, p.state + ((long long)au * tiles + at) * (Tl::ROWS * N), row0, lir);
    cp_async_commit();
    if (++at == tiles) { at = 0; au += gridDim.x; }
  };
  row_request(blockIdx.x);
#pragma unroll
  for (int k = 0; k < DEC_STAGES - 1; ++k) issue(k);
  int stage = 0, slot = 0;
  for (int u = blockIdx.x; u < units; u += gridDim.x, slot ^= 1) {
    unsigned char* row = rows + slot * row_b;   // its last readers were two units ago
    row_store(row);
    row_request(u + gridDim.x);
    const long long s = u / ups;
    const int h0 = (u - (int)s * ups) * hs;
    const T* sx = reinterpret_cast<const T*>(row);
    const T* sdt = reinterpret_cast<const T*>(row + x_b);
    const T* sB = reinterpret_cast<const T*>(row + x_b + dt_b);
    const T* sC = reinterpret_cast<const T*>(row + x_b + dt_b + bc_b);
    int hl = 0, tl = 0;
    for (int k = 0; k < tiles; ++k) {
      cp_async_wait<DEC_STAGES - 2>();
      __syncthreads();   // this tile and the row are in shared memory; the previous slot and the last unit's y are free
      issue(stage == 0 ? DEC_STAGES - 1 : stage - 1);
      const unsigned char* sm = dec_ring + stage * Tl::BYTES;
      stage = stage + 1 == DEC_STAGES ? 0 : stage + 1;
      const int h = h0 + hl;
      const float dtv = dt_activation(ldf_shared(sdt + h), p.dt_bias ? __ldg(p.dt_bias + h) : 0.f, d.dt_softplus);
      const float a = expf(dtv * __ldg(p.A + h));
      const float Dh = p.D ? __ldg(p.D + h) : 0.f;
      const int r0 = hl * P + tl * Tl::ROWS, gb = (h / hpg) * N;
      tile_update<Tl, T, N>(sm, p.state + ((long long)u * tiles + k) * (Tl::ROWS * N), sx + r0, sB + gb, sC + gb, dtv, a, Dh, row0, lir,
                            [&](int r, float yv) { stf(reinterpret_cast<T*>(ybuf) + r0 + r, yv); });
      if (++tl == tph) { tl = 0; ++hl; }
    }
    __syncthreads();   // y of the unit is complete
    for (int o = threadIdx.x * 16; o < x_b; o += DEC_THREADS * 16) {
      const uint4 v = *reinterpret_cast<const uint4*>(ybuf + o);
      const long long to = s * d.y_stride_s + (long long)h0 * P;
      *reinterpret_cast<uint4*>((char*)(y_host + to) + o) = v;
      if (p.y) *reinterpret_cast<uint4*>((char*)((T*)p.y + to) + o) = v;
    }
  }
  cp_async_wait<0>();
}

// Any other dstate: one warp per state row, lanes stride over n.
template <typename T>
__global__ void __launch_bounds__(DEC_THREADS) k_state_update_generic(SsdStepDims d, SsdStepPtrs p) {
  pdl_wait();
  const int sh = blockIdx.x;
  const int s = sh / d.nheads, h = sh - s * d.nheads;
  const int grp = h / (d.nheads / d.ngroups);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int P = d.headdim, N = d.dstate;
  const T* xs = (const T*)p.x + s * d.x_stride_s + (long long)h * P;
  const float dtv = dt_activation(ldf((const T*)p.dt + s * d.dt_stride_s + h), p.dt_bias ? __ldg(p.dt_bias + h) : 0.f, d.dt_softplus);
  const float a = expf(dtv * __ldg(p.A + h));
  const float Dh = p.D ? __ldg(p.D + h) : 0.f;
  const T* Bp = (const T*)p.Bm + s * d.b_stride_s + (long long)grp * N;
  const T* Cp = (const T*)p.Cm + s * d.c_stride_s + (long long)grp * N;
  float* st = p.state + (size_t)sh * P * N;
  for (int pr = warp; pr < P; pr += DEC_THREADS / 32) {
    const float xv = ldf(xs + pr), dx = dtv * xv;
    float acc = 0.f;
    for (int n = lane; n < N; n += 32) {
      float t = fmaf(a, st[(size_t)pr * N + n], dx * ldf(Bp + n));
      st[(size_t)pr * N + n] = t;
      acc = fmaf(t, ldf(Cp + n), acc);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      float yv = acc + Dh * xv;
      if (p.z) {
        const float zv = ldf((const T*)p.z + s * d.z_stride_s + (long long)h * P + pr);
        yv *= zv * sigmoidf_(zv);
      }
      stf((T*)p.y + s * d.y_stride_s + (long long)h * P + pr, yv);
    }
  }
}

__global__ void k_reset_rows(float* state, long long row_elems, const long long* idx, long long count,
                             long long streams) {
  pdl_wait();
  const long long r = blockIdx.y;
  if (r >= count) return;
  const long long s = idx[r];
  if (s < 0 || s >= streams) return;
  float4* row = reinterpret_cast<float4*>(state + s * row_elems);
  const long long n4 = row_elems / 4;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n4; e += (long long)gridDim.x * blockDim.x)
    row[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (blockIdx.x == 0)
    for (long long e = n4 * 4 + threadIdx.x; e < row_elems; e += blockDim.x) state[s * row_elems + e] = 0.f;
}

__global__ void k_total_logdecay(Geo g, const float* __restrict__ cs, float* __restrict__ out) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // b*H + h
  if (i >= g.B * g.H) return;
  float v = 0.f;
  for (int c = 0; c < g.nc; ++c) v += cs[((size_t)i * g.nc + c) * g.Q + g.Q - 1];
  out[i] = v;
}

// Exclusive prefix over ranks by Horner's rule:
//   direction +1: acc = init; for q = 0..rank-1:        acc = exp(ld_q)*acc + st_q
//   direction -1: acc = init; for q = world-1..rank+1:  acc = exp(ld_q)*acc + st_q
__global__ void k_sp_prefix(const float* __restrict__ gs, const float* __restrict__ gl, int world, int rank,
                            int direction, long long bh, long long elems, const float* __restrict__ init,
                            float* __restrict__ out) {
  pdl_wait();
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long r = blockIdx.y;  // b*H + h
  if (e >= elems) return;
  float acc = init ? init[r * elems + e] : 0.f;
  if (direction > 0) {
    for (int q = 0; q < rank; ++q) acc = expf(gl[q * bh + r]) * acc + gs[((size_t)q * bh + r) * elems + e];
  } else {
    for (int q = world - 1; q > rank; --q) acc = expf(gl[q * bh + r]) * acc + gs[((size_t)q * bh + r) * elems + e];
  }
  out[r * elems + e] = acc;
}

}  // namespace

// The ring kernel takes every head that is a whole number of tiles, with x / B / C rows that are whole, 16-byte aligned
// pieces; everything else takes the register kernels.
template <typename T, int N, int R, bool GATED>
static bool launch_ring(const SsdStepDims& d, const SsdStepPtrs& p, cudaStream_t s) {
  using Tl = Tile<N, R>;
  constexpr int ES = (int)sizeof(T), STAGE = Tl::BYTES + (GATED ? 2 : 1) * Tl::ROWS * ES + 2 * N * ES, smem = DEC_STAGES * STAGE;
  if (d.headdim % Tl::ROWS || (Tl::ROWS * ES) % 16 || (N * ES) % 16) return false;
  auto al = [&](const void* q, long long stride) { return ((uintptr_t)q % 16) == 0 && (stride * ES) % 16 == 0; };
  if (!al(p.x, d.x_stride_s) || !al(p.Bm, d.b_stride_s) || !al(p.Cm, d.c_stride_s) || ((uintptr_t)p.state % 16)) return false;
  if (GATED && !al(p.z, d.z_stride_s)) return false;
  const int tph = d.headdim / Tl::ROWS;
  const long long items = (long long)d.streams * d.nheads * tph;
  constexpr int per_sm = (227 * 1024) / (smem + 1024) < 16 ? (227 * 1024) / (smem + 1024) : 16;
  long long grid = (long long)sm_count() * per_sm;
  if (grid > items) grid = items;
  launch<k_state_update_ring<T, N, R, GATED>>((unsigned)grid, DEC_THREADS, smem, s, d, p, tph);
  return true;
}
// The larger of two tile sizes that divides the head; false: neither does (or an operand cannot be copied in 16-byte pieces).
template <typename T, int N>
static bool launch_ring_n(const SsdStepDims& d, const SsdStepPtrs& p, cudaStream_t s) {
  // rows per thread: 8 KB tiles, 16 KB at N = 128 (a row there takes a whole warp, so a tile of four rows per thread is half
  // address arithmetic)
  constexpr int R = N == 256 ? 2 : N == 128 ? 8 : 4;
  if (p.z) return launch_ring<T, N, R, true>(d, p, s) || launch_ring<T, N, R / 2, true>(d, p, s);
  return launch_ring<T, N, R, false>(d, p, s) || launch_ring<T, N, R / 2, false>(d, p, s);
}

template <typename T>
static int decode_t(const SsdStepDims& d, const SsdStepPtrs& p, cudaStream_t s) {
  const unsigned blocks = (unsigned)((long long)d.streams * d.nheads);
  bool ring = false;
  switch (d.dstate) {
    case 64: ring = launch_ring_n<T, 64>(d, p, s); break;
    case 128: ring = launch_ring_n<T, 128>(d, p, s); break;
    case 256: ring = launch_ring_n<T, 256>(d, p, s); break;
  }
  if (!ring) switch (d.dstate) {
    case 16: launch<k_state_update<T, 16>>(blocks, DEC_THREADS, 0, s, d, p); break;
    case 32: launch<k_state_update<T, 32>>(blocks, DEC_THREADS, 0, s, d, p); break;
    case 64: launch<k_state_update<T, 64>>(blocks, DEC_THREADS, 0, s, d, p); break;
    case 128: launch<k_state_update<T, 128>>(blocks, DEC_THREADS, 0, s, d, p); break;
    case 256: launch<k_state_update<T, 256>>(blocks, DEC_THREADS, 0, s, d, p); break;
    default: launch<k_state_update_generic<T>>(blocks, DEC_THREADS, 0, s, d, p); break;
  }
  SSD_CUDA_CHECK_LAUNCH("state_update");
  return SSD_OK;
}

// Host-memory step: false where the layout is not covered (segments of 16-byte pieces, whole tiles, no gate).
template <typename T, int N>
static bool launch_host(const SsdStepDims& d, const SsdStepPtrs& p, void* y_host, cudaStream_t s) {
  using Tl = Tile<N, 4>;
  constexpr int ES = (int)sizeof(T);
  const int H = d.nheads, P = d.headdim;
  if (P % Tl::ROWS || (P * ES) % 16 || (H * ES) % 16 || (N * ES) % 16 || p.z) return false;
  auto al = [&](const void* q, long long stride) { return ((uintptr_t)q % 16) == 0 && (stride * ES) % 16 == 0; };
  if (!al(p.x, d.x_stride_s) || !al(p.dt, d.dt_stride_s) || !al(p.Bm, d.b_stride_s) || !al(p.Cm, d.c_stride_s) || !al(p.y, d.y_stride_s) ||
      !al(y_host, d.y_stride_s) || ((uintptr_t)p.state % 16)) return false;
  const int tph = P / Tl::ROWS, fixed_b = (H + 2 * d.ngroups * N) * ES;
  if (H * P * ES + fixed_b > 2 * DEC_THREADS * 16) return false;   // two 16-byte pieces of a row per thread
  // Heads per unit: all of a stream's, so that its row crosses PCIe once; a few streams are split, while that gives no more
  // than two blocks per SM, because there the walk over the heads is what takes the time.
  int hs = H;
  for (int c = H; c >= 1; --c)
    if (H % c == 0 && (long long)d.streams * (H / c) <= 2 * sm_count()) hs = c;
  const long long units = (long long)d.streams * (H / hs);
  if (units > 0x7fffffffLL - 16 * sm_count()) return false;
  const int smem = DEC_STAGES * Tl::BYTES + 2 * (hs * P * ES + fixed_b) + hs * P * ES;
  const int per_sm = (227 * 1024) / (smem + 1024) < 8 ? (227 * 1024) / (smem + 1024) : 8;
  long long grid = (long long)sm_count() * per_sm;
  if (grid > units) grid = units;
  if (hs * P * ES + fixed_b <= DEC_THREADS * 16)
    launch<k_state_update_host<T, N, 4, 1>>((unsigned)grid, DEC_THREADS, smem, s, d, p, (T*)y_host, tph, hs, (int)units);
  else
    launch<k_state_update_host<T, N, 4, 2>>((unsigned)grid, DEC_THREADS, smem, s, d, p, (T*)y_host, tph, hs, (int)units);
  return true;
}

int decode_step_host(const SsdStepDims& d, const SsdStepPtrs& p, void* y_host, cudaStream_t s) {
  const bool bf = d.dtype == SSD_BF16;
  bool ok = false;
  if (d.dstate == 64) ok = bf ? launch_host<__nv_bfloat16, 64>(d, p, y_host, s) : launch_host<float, 64>(d, p, y_host, s);
  else if (d.dstate == 128) ok = bf ? launch_host<__nv_bfloat16, 128>(d, p, y_host, s) : launch_host<float, 128>(d, p, y_host, s);
  if (!ok) {
    set_error("state_update_host: needs dstate 64 or 128, headdim a multiple of an 8 KB state tile, rows of 16-byte aligned segments of at "
              "most 4 KB, no gate");
    return SSD_ERR_UNSUPPORTED;
  }
  SSD_CUDA_CHECK_LAUNCH("state_update_host");
  return SSD_OK;
}

int decode_step(const SsdStepDims& d, const SsdStepPtrs& p, cudaStream_t s) {
  return d.dtype == SSD_BF16 ? decode_t<__nv_bfloat16>(d, p, s) : decode_t<float>(d, p, s);
}

int reset_rows(float* state, long long row_elems, const long long* idx, long long count, long long streams,
               cudaStream_t s) {
  if (count == 0) return SSD_OK;
  const long long n4 = row_elems / 4;
  const unsigned gx = (unsigned)((n4 + 255) / 256 > 0 ? ((n4 + 255) / 256 < 64 ? (n4 + 255) / 256 : 64) : 1);
  for (long long off = 0; off < count; off += 65535) {
    const long long c = (count - off < 65535) ? count - off : 65535;
    launch<k_reset_rows>(dim3(gx, (unsigned)c), 256, 0, s, state, row_elems, idx + off, c, streams);
  }
  SSD_CUDA_CHECK_LAUNCH("state_reset_rows");
  return SSD_OK;
}

int sp_total_logdecay(const Geo& g, const float* cs, float* out, cudaStream_t s) {
  launch<k_total_logdecay>(cdiv(g.B * g.H, 128), 128, 0, s, g, cs, out);
  SSD_CUDA_CHECK_LAUNCH("sp_total_logdecay");
  return SSD_OK;
}

int sp_prefix_state(const float* gs, const float* gl, int world, int rank, int direction, long long bh,
                    long long elems, const float* init, float* out, cudaStream_t s) {
  launch<k_sp_prefix>(dim3((unsigned)((elems + 255) / 256), (unsigned)bh), 256, 0, s, gs, gl, world, rank, direction, bh,
                                                                                 elems, init, out);
  SSD_CUDA_CHECK_LAUNCH("sp_prefix_state");
  return SSD_OK;
}

}  // namespace ssd
