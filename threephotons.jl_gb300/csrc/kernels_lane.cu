// Stage (a) coupling, lane-owned form: the reference's triple products
//   T[(k1,k2,k3)][(l1,l2,l3)] = sum_j w_j Re(c_k1[l1,m1] c_k2[l2,m2] c_k3[l3,m3])
// (src/correlations.jl:157-176; src/cuda_kernel.cu:31-37), pair-factorised as
//   D[k1,k2][l3][m3] = sum_m1 w(l1 m1 l2 m2 l3 m3) c_k1[l1,m1] c_k2[l2,m2],  m2 = -m3 - m1
//   T[(k1,k2,k3)][lt] = Re sum_m3 D[k1,k2][l3][m3] c_k3[l3,m3]
// with D and T held in the registers of the lane that owns the shell pair (k1, k2).
//
// Units: the shell pairs with k3 in one block of 16 shells, sorted by k2 downwards, 32
// consecutive pairs a warp, one a lane, so the lanes of a warp need nearly the same k3 <= k2.
// A task is one unit and a run of up to NC orders l3 of one (l1, l2) block; its T accumulators
// (NC orders x 16 shells k3) stay in registers while the warp walks quads of four consecutive m3:
//   Phase 1: D of the quad's four m3 and the task's orders.  One of the two coefficient rows
//     of a product is the same for all four m3, the other slides by one m, so a step loads two
//     coefficients, forms four complex products and feeds one 16-byte 3j broadcast (the four
//     m3) per order into four packed FMAs.
//   Phase 2: T += Re(D c_k3) for the quad, packed over pairs of k3; c_k3 comes as 16-byte
//     broadcasts (all lanes read the same four shells).
// A warp needs no other warp, so warps take tasks from a counter, heaviest first.
//
// What bounds it: issue slots and the shared-memory port.  At L = 18, K = 26 a proposal of a real
// function is 11.4 M warp instructions (the folded rows 15.5 M) in 14.5 us, 62 % of the issue slots
// and 60 % of the port; 5.5 M of them go to the FMA pipe, where the operations it cannot do without
// (m3 >= 0 and the pairs, orders and shells that exist) take 3.2 us on 152 SMs.  Only coefficients
// and 3j values are shared, 80 KB a CTA with no D buffer, which lets 16 warps run with no barrier
// after the staging.
//
// Every accumulation runs in the order of the one-kernel pair coupling (k_couple_pair), so
// both give the same bits: m1 upwards in phase 1, m3 = 1 .. l3 then the doubled sum plus the
// m3 = 0 term in phase 2 (real functions), or m3 = -l3 .. l3 (general coefficients).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/tp3.h"
#include "internal.h"
#include "scalar.cuh"
#include "tables.h"
#include "tc_prims.cuh"

namespace tp3 {
namespace {

// Orders per task: 16 kLaneNC accumulator registers for T and 8 kLaneNC for D, 128 a thread in
// all, so 16 warps per SM.  All kLaneNC columns are always computed (columns outside the task
// are not used): with a loop per column count, or more instances for more shells k3, the code
// of an SM's warps left its instruction cache (29 of 34 stall cycles per issue with one
// instance per width of k3).  64 proposals at L = 18, K = 26: 0.93 ms at 3 orders and 16 warps,
// 1.02 at 4 and 12, 1.44 at 5 and 12 (spills), 1.30 at 5 with a loop per column count; the
// one-kernel pair coupling takes 2.51 ms and the folded rows at 13 warps 1.58.
constexpr int kLaneNC = 3;
constexpr int kLaneMaxWarps = 16;

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"((uint64_t)__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ float2 lds2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}

__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}

// Shared-memory addresses of one (proposal, block).
struct LaneView {
  uint32_t X;         // float2 rows, operand with one row per step
  uint32_t V;         // float2 rows, operand that slides by one row per m3
  uint32_t W;         // 3j values, float4 per (step, order): the quad's four m3
  uint32_t C3;        // c_k3 rows: (re x 4, im x 4) per quad of shells
  const LaneQuad* quads;
  int nq;
#ifdef TP3_DEBUG
  // what is staged: rows of X and V and of C3, 3j values (float4, from 8 before W on); C3 of block 0
  int xrows, vrows, wlen, c3rows;
  uint32_t c3first;
  int* err;
#endif
};

// One step of phase 1: the products of x with the window rows of the quad's four m3, each into
// its half of the packed accumulators.  SW: x is c_k2 and the window c_k1 (in the imaginary
// part the product with c_k1's imaginary part is the fused one).  FIRST: sets the accumulators.
template <int NC, bool SW, bool FIRST>
__device__ __forceinline__ void lane_step(const float2 x, const float2 v0, const float2 v1, const float2 v2,
                                          const float2 v3, uint32_t w, float2 (&R0)[NC], float2 (&I0)[NC],
                                          float2 (&R1)[NC], float2 (&I1)[NC]) {
  auto re = [&](const float2 v) { return fmaf(x.x, v.x, -(x.y * v.y)); };
  auto im = [&](const float2 v) { return SW ? fmaf(v.y, x.x, v.x * x.y) : fmaf(x.y, v.x, x.x * v.y); };
  const float2 xr0 = make_float2(re(v0), re(v1)), xr1 = make_float2(re(v2), re(v3));
  const float2 xi0 = make_float2(im(v0), im(v1)), xi1 = make_float2(im(v2), im(v3));
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const float4 wv = lds4(w + 16 * c);
    const float2 w0 = make_float2(wv.x, wv.y), w1 = make_float2(wv.z, wv.w);
    if (FIRST) {
      R0[c] = __fmul2_rn(w0, xr0);
      I0[c] = __fmul2_rn(w0, xi0);
      R1[c] = __fmul2_rn(w1, xr1);
      I1[c] = __fmul2_rn(w1, xi1);
    } else {
      R0[c] = __ffma2_rn(w0, xr0, R0[c]);
      I0[c] = __ffma2_rn(w0, xi0, I0[c]);
      R1[c] = __ffma2_rn(w1, xr1, R1[c]);
      I1[c] = __ffma2_rn(w1, xi1, I1[c]);
    }
  }
}

// Phase 1 of one quad: n steps (odd) over all NC columns; PS shells per coefficient row, rs
// bytes of 3j values per step.  The window rows run with the steps (SW: against m3).
template <int NC, int PS, bool SW>
__device__ __forceinline__ void lane_p1(uint32_t x, uint32_t v, int n, uint32_t w, uint32_t rs, float2 (&R0)[NC],
                                        float2 (&I0)[NC], float2 (&R1)[NC], float2 (&I1)[NC]) {
  constexpr int xs = 8 * (SW ? -PS : PS), vs = -xs;
  auto step = [&](const float2 xv, const float2 a, const float2 b, const float2 c, const float2 d, uint32_t wa, auto first) {
    if (SW)
      lane_step<NC, SW, decltype(first)::value>(xv, d, c, b, a, wa, R0, I0, R1, I1);
    else
      lane_step<NC, SW, decltype(first)::value>(xv, a, b, c, d, wa, R0, I0, R1, I1);
  };
  float2 a = lds2(v + vs), b = lds2(v + 2 * vs), c = lds2(v + 3 * vs);
  step(lds2(x), lds2(v), a, b, c, w, std::true_type());
  x += xs;
  v += 4 * vs;
  w += rs;
  int i = n - 1;
#pragma unroll 1
  for (; i >= 4; i -= 4) {
    const float2 d = lds2(v), e = lds2(v + vs), f = lds2(v + 2 * vs), g = lds2(v + 3 * vs);
    step(lds2(x), a, b, c, d, w, std::false_type());
    step(lds2(x + xs), b, c, d, e, w + rs, std::false_type());
    step(lds2(x + 2 * xs), c, d, e, f, w + 2 * rs, std::false_type());
    step(lds2(x + 3 * xs), d, e, f, g, w + 3 * rs, std::false_type());
    a = e; b = f; c = g;
    v += 4 * vs;
    x += 4 * xs;
    w += 4 * rs;
  }
#pragma unroll 1
  for (; i > 0; --i) {
    const float2 d = lds2(v);
    step(lds2(x), a, b, c, d, w, std::false_type());
    a = b; b = c; c = d;
    v += vs;
    x += xs;
    w += rs;
  }
}

// T of one order: acc (pairs of k3) += Re(D c_k3) for one m3 and the unit's 8 or 16 shells k3.
__device__ __forceinline__ void lane_p2(uint32_t row, float dr, float di, bool wide, float2 (&acc)[8]) {
  const float2 a = make_float2(dr, dr), b = make_float2(-di, -di);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (j == 2 && !wide) break;
    const float4 r = lds4(row + 32 * j), s = lds4(row + 32 * j + 16);
    acc[2 * j] = __ffma2_rn(a, make_float2(r.x, r.y), __ffma2_rn(b, make_float2(s.x, s.y), acc[2 * j]));
    acc[2 * j + 1] = __ffma2_rn(a, make_float2(r.z, r.w), __ffma2_rn(b, make_float2(s.z, s.w), acc[2 * j + 1]));
  }
}

// Where a task's T goes.
struct LaneOut {
  void *hi, *lo;       // split operand of the proposal (null: not written)
  float* T32;          // FP32 T of the proposal (null: not written)
  int KP, klp, ldT32;
  bool tf32, ltmaj, t32maj;
};

// One task: orders s_lo .. s_lo + w - 1 of the block for the 32 shell pairs of a unit; CR bytes
// per c_k3 row, slots / nslot: the unit's staging slots (build_lane_units).  SYM: real functions.
template <bool SYM, int NC, int PS, int CR>
__device__ __forceinline__ void lane_task(const LaneView& V, bool swap, int l3min, int s_lo, int w, int lt_base,
                                          bool wide, int k1, int k2, int len, int off, int nslot, float* stage,
                                          const uint32_t* __restrict__ slots, const LaneOut& o) {
  const int lane = threadIdx.x & 31;
  float2 acc[NC][8];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[c][j] = make_float2(0.f, 0.f);
  float2 R0[NC], I0[NC], R1[NC], I1[NC];
  // column c is order s_lo + c - (NC - w); it takes the m3 with (unsigned)(|m3| - m_lo) < cnt[c]
  // (none for the NC - w columns before the task's orders).  row[c]: address of its c_k3 row of
  // the quad's first m3, after the rows of the orders staged before it: from order 0 with m3 =
  // 0 .. l3 (real functions), or from s_lo with m3 = -l3 .. l3 (general coefficients)
  const int s_hi = s_lo + w, s_off = s_lo - (NC - w);
  int m_lo = SYM ? 1 : 0;  // the m3 = 0 term of real functions is added last
  uint32_t row[NC];
  int cnt[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int s = s_off + c, l3 = l3min + 2 * s, j = s - s_lo;
    cnt[c] = s < s_lo ? 0 : l3 - m_lo + 1;
    row[c] = V.C3 + CR * (SYM ? s * (l3min + s) : j * (2 * l3 - 2 * j - 1) + V.quads[0].m3 + l3);
  }
  const uint32_t xk = V.X + 8 * (swap ? k2 : k1), vk = V.V + 8 * (swap ? k1 : k2);
  float2* D0 = reinterpret_cast<float2*>(stage);  // real functions: D of m3 = 0, [NC][32]
#pragma unroll 1
  for (int qi = 0; qi <= V.nq; ++qi) {
    int m = 0;
    if (qi < V.nq) {
      const LaneQuad q = V.quads[qi];
      if (q.c0 >= s_hi) continue;
      m = q.m3;
#ifdef TP3_DEBUG
      {  // the first and last rows of either operand and 3j values
        const int sx = swap ? -1 : 1, x1 = q.x0 + sx * (q.n - 1), v1 = q.vb - sx * (q.n + 2);
        const int w0 = q.wofs + s_hi - NC - q.c0;
        const bool ok = min(q.x0, x1) >= 0 && max(q.x0, x1) < V.xrows && min(q.vb, v1) >= 0 &&
                        max(q.vb, v1) < V.vrows && w0 >= -8 && w0 + (q.n - 1) * q.rs + NC <= V.wlen && k1 < PS && k2 < PS;
        if (!TP3_DCHECK(ok, V.err)) continue;
      }
#endif
      // all NC columns; those outside the task or below the quad's orders are not used
      const uint32_t x = xk + 8 * PS * q.x0, v = vk + 8 * PS * q.vb, wt = V.W + 16 * (q.wofs + s_hi - NC - q.c0);
      if (swap)
        lane_p1<NC, PS, true>(x, v, q.n, wt, 16 * q.rs, R0, I0, R1, I1);
      else
        lane_p1<NC, PS, false>(x, v, q.n, wt, 16 * q.rs, R0, I0, R1, I1);
      if (SYM && m == 0) {
#pragma unroll
        for (int c = 0; c < NC; ++c) D0[c * 32 + lane] = make_float2(R0[c].x, I0[c].x);
      }
    } else {
      if (!SYM) break;
      // T = 2 sum_{m3 > 0} Re(D c) + Re(D[0] c[0])
      m_lo = 0;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int s = s_off + c;
        cnt[c] = s < s_lo ? 0 : 1;
        row[c] = V.C3 + CR * (s * (l3min + s));
        const float2 d = D0[c * 32 + lane];
        R0[c].x = d.x;
        I0[c].x = d.y;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[c][j].x *= 2.f;
          acc[c][j].y *= 2.f;
        }
      }
    }
#ifdef TP3_DEBUG
    {  // the c_k3 rows of the m3 that count
      bool ok = true;
      for (int k = 0; k < 4; ++k)
        for (int c = 0; c < NC; ++c) {
          const int t = (SYM ? m + k : abs(m + k)) - m_lo, at = (int)(row[c] - V.c3first) + k * CR;
          if ((unsigned)t < (unsigned)cnt[c]) ok = ok && at >= 0 && at + 32 * (wide ? 4 : 2) <= V.c3rows * CR;
        }
      if (!TP3_DCHECK(ok, V.err)) break;
    }
#endif
    // phase 2, two m3 at a time
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int ma = m + 2 * h, mb = ma + 1;
      const int t0 = (SYM ? ma : abs(ma)) - m_lo, t1 = (SYM ? mb : abs(mb)) - m_lo;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if ((unsigned)t0 < (unsigned)cnt[c]) lane_p2(row[c], h ? R1[c].x : R0[c].x, h ? I1[c].x : I0[c].x, wide, acc[c]);
        if ((unsigned)t1 < (unsigned)cnt[c])
          lane_p2(row[c] + CR, h ? R1[c].y : R0[c].y, h ? I1[c].y : I0[c].y, wide, acc[c]);
        row[c] += 2 * CR;
      }
    }
  }
  __syncwarp();
  // T leaves order by order through the warp's staging row, in which the unit's shell triples
  // are sorted by their index, an even one on an even position: a lane takes slots of two
#pragma unroll 1
  for (int c = NC - w; c < NC; ++c) {
    const int lt = lt_base + s_off + c;
#define TP3_LANE_PUT(C)                                                                               \
  case C:                                                                                             \
    _Pragma("unroll") for (int j = 0; j < 16; ++j) if (j < len) stage[off + j] =                      \
        (j & 1) ? acc[C][j >> 1].y : acc[C][j >> 1].x;                                                \
    break;
    switch (c) {
      TP3_LANE_PUT(0) TP3_LANE_PUT(1) TP3_LANE_PUT(2)
      default: break;
    }
#undef TP3_LANE_PUT
    __syncwarp();
    if (o.hi && o.ltmaj) {
      __nv_bfloat16* hrow = reinterpret_cast<__nv_bfloat16*>(o.hi) + (size_t)lt * o.klp;
      __nv_bfloat16* lrow = reinterpret_cast<__nv_bfloat16*>(o.lo) + (size_t)lt * o.klp;
      auto put = [&](const uint32_t sl, const float2 t) {
        const uint32_t at = (sl >> 2) * 2;
        const __nv_bfloat162 h = __floats2bfloat162_rn(t.x, t.y);
        const float2 hf = __bfloat1622float2(h);
        const __nv_bfloat162 l = __floats2bfloat162_rn(t.x - hf.x, t.y - hf.y);
        if ((sl & 3) == 3) {
          *reinterpret_cast<__nv_bfloat162*>(hrow + at) = h;
          *reinterpret_cast<__nv_bfloat162*>(lrow + at) = l;
        } else if (sl & 1) {
          hrow[at] = h.x;
          lrow[at] = l.x;
        } else if (sl & 2) {
          hrow[at + 1] = h.y;
          lrow[at + 1] = l.y;
        }
      };
#ifdef TP3_DEBUG
      bool rows_ok = lt < o.KP;
      for (int i = lane; i < nslot; i += 32)
        rows_ok = rows_ok && ((slots[i] & 3) == 0 || (int)(slots[i] >> 2) * 2 + ((slots[i] & 2) ? 1 : 0) < o.klp);
      if (!TP3_DCHECK(__all_sync(0xffffffffu, rows_ok), V.err)) break;
#endif
      const float2* st = reinterpret_cast<const float2*>(stage);
#pragma unroll 1
      for (int i = lane; i < nslot; i += 64) {
        const bool two = i + 32 < nslot;
        const uint32_t sa = __ldg(slots + i), sb = two ? __ldg(slots + i + 32) : 0u;
        const float2 ta = st[i], tb = st[two ? i + 32 : i];
        put(sa, ta);
        put(sb, tb);
      }
    }
    if (!o.ltmaj || o.T32) {
#pragma unroll 1
      for (int i = lane; i < 2 * nslot; i += 32) {
        const uint32_t sl = __ldg(slots + (i >> 1));
        if (!((sl >> (i & 1)) & 1)) continue;
        const int ki = 2 * (int)(sl >> 2) + (i & 1);
        const float t = stage[i];
        if (!TP3_DCHECK(ki < o.klp && lt < (o.T32 && !o.t32maj ? o.ldT32 : o.KP), V.err)) continue;
        if (o.hi && !o.ltmaj) {
          const size_t at = (size_t)ki * o.KP + lt;
          if (o.tf32) {
            uint32_t h;
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(t));
            reinterpret_cast<float*>(o.hi)[at] = __uint_as_float(h);
            reinterpret_cast<float*>(o.lo)[at] = t - __uint_as_float(h);
          } else {
            const __nv_bfloat16 h = __float2bfloat16_rn(t);
            reinterpret_cast<__nv_bfloat16*>(o.hi)[at] = h;
            reinterpret_cast<__nv_bfloat16*>(o.lo)[at] = __float2bfloat16_rn(t - __bfloat162float(h));
          }
        }
        if (o.T32) o.T32[o.t32maj ? (size_t)lt * o.klp + ki : (size_t)ki * o.ldT32 + lt] = t;
      }
    }
    __syncwarp();
  }
}

// Run i of n balanced runs of nl3 orders: first order and orders.
__host__ __device__ __forceinline__ void lane_run(int nl3, int n, int i, int& s_lo, int& w) {
  const int lo = nl3 / n, ex = nl3 - lo * n;
  s_lo = i * lo + (i < ex ? i : ex);
  w = lo + (i < ex ? 1 : 0);
}

// grid: (n, Z, n_pb); block 32 x warps; dynamic shared memory lane_smem_bytes.
// CTA (p, z, b) takes the tasks z, z + Z, .. of block order[b] of proposal p: Z > 1 spreads the
// tasks of a small batch over the SMs.  A real function's c_k3 rows and 3j values (m3 >= 0) are
// staged for all orders; general coefficients (both signs of m3, twice the rows and values) go in
// passes of up to kLaneNC orders, one run of orders for all units, and Z > 1 spreads the passes first.
// A pass per order computes kLaneNC columns for one: 64 general proposals at L = 18, K = 26 took
// 3.39 ms (the whole scoring) so and 1.85 in runs; four in TF32 mode at L = 12, K = 16 107 and 66 us,
// where the one-kernel coupling takes 95.  Proposals run fastest, so an SM's CTAs are mostly on
// one block and their warps in the same code.
template <int PS>
__global__ void __launch_bounds__(32 * kLaneMaxWarps, 1) k_couple_lane(
    const float2* __restrict__ ct, const float4* __restrict__ c3p, int K, int nc, const int* __restrict__ order,
    const int* __restrict__ coff, const LaneBlock* __restrict__ blks, const LaneQuad* __restrict__ quads,
    const int4* __restrict__ gcols, const float4* __restrict__ wtab, const uint32_t* __restrict__ utab,
    const uint32_t* __restrict__ slots, const int2* __restrict__ kofs, int crows, int wmax, int c3rows, int stage_len,
    const int* __restrict__ symflags, LaneOut out, const RagInfo* __restrict__ rag, int* __restrict__ err) {
  constexpr int ps = PS, c3row = PS / 2;
  extern __shared__ __align__(16) unsigned char lane_smem[];
  __shared__ LaneQuad s_quads[kLaneMaxQuads];
  __shared__ uint64_t s_bar;
  __shared__ int s_next[17];
  __shared__ int s_abort;
  grid_wait();
  grid_release();
  const int prop = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blk = order[blockIdx.z];
  const LaneBlock fb = blks[blk];
  int Kp = K;
  bool skip = false;
  int klen = 0;
  if (rag) {
    const RagInfo ri = after_wait(rag)[prop];
    Kp = ri.K;
    klen = ri.klen;
    skip = fb.l1 > ri.L || fb.l2 > ri.L;
  }
  const size_t pbase = (size_t)prop * out.klp * out.KP;
  if (out.hi) {
    out.hi = out.tf32 ? (void*)((float*)out.hi + pbase) : (void*)((__nv_bfloat16*)out.hi + pbase);
    out.lo = out.tf32 ? (void*)((float*)out.lo + pbase) : (void*)((__nv_bfloat16*)out.lo + pbase);
  }
  if (out.T32) out.T32 += (size_t)prop * out.klp * out.ldT32;
  if (skip) {
    // absent orders: the block's l-triples are zero for this proposal's scored rows
    for (int i = threadIdx.x + blockIdx.y * blockDim.x; i < klen * fb.nl3; i += blockDim.x * gridDim.y) {
      const int s = i / klen, ki = i - s * klen, lt = fb.lt_base + s;
      if (out.hi) {
        const size_t at = out.ltmaj ? (size_t)lt * out.klp + ki : (size_t)ki * out.KP + lt;
        if (out.tf32) {
          reinterpret_cast<float*>(out.hi)[at] = 0.f;
          reinterpret_cast<float*>(out.lo)[at] = 0.f;
        } else {
          reinterpret_cast<__nv_bfloat16*>(out.hi)[at] = __float2bfloat16_rn(0.f);
          reinterpret_cast<__nv_bfloat16*>(out.lo)[at] = __float2bfloat16_rn(0.f);
        }
      }
      if (out.T32) out.T32[out.t32maj ? (size_t)lt * out.klp + ki : (size_t)ki * out.ldT32 + lt] = 0.f;
    }
    return;
  }
  const bool sym = after_wait(symflags)[prop] != 0;
  const int2 ko = kofs[Kp];
  const int nu = ko.y;
  // tasks t = next * tstep + toff; general coefficients: passes pass0, pass0 + pstep, ..
  const int pstep = sym ? 1 : min((int)gridDim.y, fb.gp), pass0 = sym ? 0 : blockIdx.y % pstep;
  const int tstep = (gridDim.y - pass0 + pstep - 1) / pstep, toff = blockIdx.y / pstep;
  if (toff >= (sym ? nu * fb.nl3 : nu)) return;  // more CTAs than tasks
  float2* C1 = reinterpret_cast<float2*>(lane_smem);
  float2* C2 = C1 + (size_t)crows * ps;
  float4* W = reinterpret_cast<float4*>(C2 + (size_t)crows * ps) + 8;  // a rounded-up run may start before its row
  float4* C3 = W + wmax;
  float* stage = reinterpret_cast<float*>(C3 + (size_t)c3rows * c3row) + (size_t)warp * stage_len;
  const float2* ctp = ct + (size_t)prop * nc * ps;
  const float4* c3g = c3p + (size_t)prop * nc * c3row;
  const int n1r = 2 * fb.l1 + 1, n2r = 2 * fb.l2 + 1;
  // three zero rows at either end of C1 and C2: the union m range of a quad reaches up to
  // three rows past an end, where its 3j value is zero
  for (int i = threadIdx.x; i < 6 * ps; i += blockDim.x) {
    const int r = i / ps, k = i - r * ps;
    C1[(r < 3 ? r : n1r + r) * ps + k] = make_float2(0.f, 0.f);
    C2[(r < 3 ? r : n2r + r) * ps + k] = make_float2(0.f, 0.f);
  }
  if (threadIdx.x == 0) {
    mbar_init(&s_bar, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 17) s_next[threadIdx.x] = 0;
  __syncthreads();
#ifdef TP3_DEBUG
  if (!TP3_DCHECK(n1r + 6 <= crows && n2r + 6 <= crows && fb.c1 + n1r <= nc && fb.c2 + n2r <= nc &&
                      fb.lt_base + fb.nl3 <= out.KP && fb.gp <= 16 && Kp <= K,
                  err))
    return;
#endif
  LaneView V;
#ifdef TP3_DEBUG
  V.xrows = 6 + (fb.swap ? n2r : n1r);
  V.vrows = 6 + (fb.swap ? n1r : n2r);
  V.c3first = smem_u32(C3);
  V.err = err;
#endif
  V.X = smem_u32(fb.swap ? C2 : C1);
  V.V = smem_u32(fb.swap ? C1 : C2);
  V.W = smem_u32(W);
  V.C3 = smem_u32(C3);
  V.quads = s_quads;
  // real functions and general coefficients each in code of its own, both without spills: 64 real
  // proposals at L = 18, K = 26 score in 1.176 ms so and in 1.254 with one task for both
  auto passes = [&](auto real) {
    constexpr bool SYM = decltype(real)::value;
    uint32_t phase = 0;
    for (int pass = pass0; pass < (SYM ? 1 : fb.gp); pass += pstep, phase ^= 1u) {
      int4 g = make_int4(fb.q0, fb.nq, fb.w0, fb.wn);
      int p_lo = 0, p_w = fb.nl3;  // the orders staged
      if (!SYM) {
        g = gcols[blk * 16 + pass];
        lane_run(fb.nl3, fb.gp, pass, p_lo, p_w);
      }
#ifdef TP3_DEBUG
      V.wlen = g.w;
      V.c3rows = 0;
      bool in_layout = g.w <= wmax && g.y <= kLaneMaxQuads;
      for (int s = p_lo; s < p_lo + p_w; ++s) {
        const int l3 = fb.l3min + 2 * s;
        V.c3rows += SYM ? l3 + 1 : 2 * l3 + 1;
        in_layout = in_layout && coff[l3 >> 1] + 2 * l3 + 1 <= nc;
      }
      if (!TP3_DCHECK(in_layout && V.c3rows <= c3rows, err)) return;
#endif
      if (pass > pass0) {
        __syncthreads();  // the previous orders' reads are done
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      if (threadIdx.x == 0) {
        uint32_t bytes = (uint32_t)g.w * 16u;
        if (pass == pass0) bytes += (uint32_t)(n1r + n2r) * ps * 8u;
        int r = 0;
        for (int s = p_lo; s < p_lo + p_w; ++s) {
          const int l3 = fb.l3min + 2 * s;
          r += SYM ? l3 + 1 : 2 * l3 + 1;
        }
        bytes += (uint32_t)r * c3row * 16u;
        mbar_expect_tx(&s_bar, bytes);
        if (pass == pass0) {
          bulk_load(C1 + 3 * ps, ctp + (size_t)fb.c1 * ps, (uint32_t)n1r * ps * 8u, &s_bar);
          bulk_load(C2 + 3 * ps, ctp + (size_t)fb.c2 * ps, (uint32_t)n2r * ps * 8u, &s_bar);
        }
        bulk_load(W, wtab + g.z, (uint32_t)g.w * 16u, &s_bar);
        r = 0;
        for (int s = p_lo; s < p_lo + p_w; ++s) {
          const int l3 = fb.l3min + 2 * s, cnt = SYM ? l3 + 1 : 2 * l3 + 1;
          const int c0 = coff[l3 >> 1] + (SYM ? l3 : 0);
          bulk_load(C3 + (size_t)r * c3row, c3g + (size_t)c0 * c3row, (uint32_t)cnt * c3row * 16u, &s_bar);
          r += cnt;
        }
      }
      for (int i = threadIdx.x; i < g.y; i += blockDim.x) s_quads[i] = quads[g.x + i];
      __syncthreads();
      V.nq = g.y;
      if (!mbar_wait(&s_bar, phase, &s_abort, err)) {
        mbar_wait_limit(&s_bar, phase, kTimeoutCycles, err);  // copies still in flight land before the exit
        return;
      }
      const int nrun = SYM ? (fb.nl3 + kLaneNC - 1) / kLaneNC : 1;
      for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(&s_next[pass], 1);
        t = __shfl_sync(0xffffffffu, t, 0) * tstep + toff;
        const int u = t / nrun;
        if (u >= nu) break;
        int s_lo = p_lo, w = p_w;
        if (SYM) lane_run(fb.nl3, nrun, t - u * nrun, s_lo, w);
        const uint32_t e = utab[ko.x + u * 34 + lane];  // the lane's shell pair, see build_lane_units
        const uint32_t s0 = utab[ko.x + u * 34 + 32], s1 = utab[ko.x + u * 34 + 33];
        V.C3 = smem_u32(C3 + 8 * (s1 >> 17));
        if (!TP3_DCHECK((int)(e >> 24) + ((int)(e >> 12) & 0xfff) <= stage_len && 2 * (int)(s1 & 0xffff) <= stage_len &&
                            (int)(s1 >> 17) * 8 < c3row,
                        err))
          break;
        lane_task<SYM, kLaneNC, PS, 8 * PS>(V, fb.swap, fb.l3min, s_lo, w, fb.lt_base, (s1 >> 16) & 1, (int)e & 63,
                                            (int)(e >> 6) & 63, (int)(e >> 24), (int)(e >> 12) & 0xfff, (int)(s1 & 0xffff),
                                            stage, slots + s0, out);
        __syncwarp();
      }
    }
  };
  if (sym)
    passes(std::true_type());
  else
    passes(std::false_type());
}

__device__ __forceinline__ double flip(const double x, bool neg) {
  return neg ? __hiloint2double(__double2hiint(x) ^ (int)0x80000000, __double2loint(x)) : x;
}

// Coefficients for the lane-owned coupling: one cluster of kGatherCtas CTAs per proposal, four
// shells (a quad) a CTA and round, reads the FP64 values once, checks the real-function relation
// c[l,-m] = (-1)^m conj c[l,m] to 1e-10 of the shell's largest coefficient, and writes two FP32
// layouts with the shells contiguous: ct [nc][ps] (c_k1 and c_k2) and c3p [nc][c3row] (c_k3: four
// real parts, four imaginary parts per quad of shells).  sym = 1 when every shell satisfies the
// relation; m < 0 is then rebuilt from m >= 0 so that it holds exactly in FP32.
// grid: (kGatherCtas, n); block 256; dynamic shared memory ROUNDS x 4 (nc | 1) double2.
// Bound by the latency of one round of loads (device memory or the caller's host array).  FP64
// arithmetic is kept for shells that hold the relation only approximately: with it everywhere
// and one CTA a proposal (as in k_gather_sym) K = 26, L = 18 took 34 us.
constexpr int kGatherCtas = 8;
template <int ROUNDS>
__global__ void __cluster_dims__(kGatherCtas, 1, 1) __launch_bounds__(256)
    k_gather_lane(int K, int nc, int ncoef, const int* __restrict__ csean, const int* __restrict__ cm,
                  const int* __restrict__ cmir, const int* __restrict__ cl, const double2* __restrict__ coeff,
                  float2* __restrict__ ct, float* __restrict__ c3p, int* __restrict__ sym, const RagInfo* __restrict__ rag,
                  int* __restrict__ err) {
  cluster_started_arrive();
  grid_release();
  extern __shared__ __align__(16) double2 gl_smem[];
  __shared__ int s_ok[kGatherCtas];
  constexpr int ps = 32 * ROUNDS, c3row = ps / 2;
  const int prop = blockIdx.y, rank = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ld = nc | 1;
  const double2* cp = coeff + (size_t)prop * K * ncoef;
#ifdef TP3_DEBUG
  {  // the coefficient maps stay inside a shell's coefficients and the compact layout
    int maps_ok = K <= ps;
    for (int c = threadIdx.x; c < nc; c += 256)
      maps_ok &= csean[c] >= 0 && csean[c] < ncoef && cmir[c] >= 0 && cmir[c] < nc;
    if (!TP3_DCHECK(__syncthreads_and(maps_ok) != 0, err)) K = 0;  // nothing is read, zeros are written
  }
#endif
  for (int rd = 0; rd < ROUNDS; ++rd) {
    const int k0 = 4 * (rank + kGatherCtas * rd), nk = min(4, K - k0);
#pragma unroll 4
    for (int i = threadIdx.x; i < nk * nc; i += 256) {
      const int kk = i / nc, c = i - kk * nc;
      gl_smem[(4 * rd + kk) * ld + c] = cp[(size_t)(k0 + kk) * ncoef + csean[c]];
    }
  }
  __syncthreads();
  // exact, finite mirror images need no tolerance
  int exact = 1;
  for (int rd = 0; rd < ROUNDS; ++rd) {
    const int nk = min(4, K - 4 * (rank + kGatherCtas * rd));
    for (int i = threadIdx.x; i < nk * nc; i += 256) {
      const int kk = i / nc, c = i - kk * nc, m = cm[c];
      if (m < 0) continue;
      const double2* row = gl_smem + (4 * rd + kk) * ld;
      const double2 a = row[c];
      if (m == 0) {
        exact &= (__double_as_longlong(a.y) << 1) == 0;
      } else {
        const double2 b = row[cmir[c]];
        const bool odd = m & 1;
        exact &= __double_as_longlong(b.x) == __double_as_longlong(flip(a.x, odd)) &&
                 __double_as_longlong(b.y) == __double_as_longlong(flip(a.y, !odd)) &&
                 (__double2hiint(a.x) & 0x7ff00000) != 0x7ff00000 && (__double2hiint(a.y) & 0x7ff00000) != 0x7ff00000;
      }
    }
  }
  int ok = 1;
  if (!__syncthreads_and(exact) && warp < 4 * ROUNDS) {  // one warp a shell
    const double2* row = gl_smem + warp * ld;
    const bool live = 4 * (rank + kGatherCtas * (warp >> 2)) + (warp & 3) < K;
    double amax = 0.0;
    if (live)
      for (int c = lane; c < nc; c += 32) amax = fmax(amax, fabs(row[c].x) + fabs(row[c].y));
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const double tol = 1e-10 * amax;
    for (int c = lane; live && c < nc; c += 32) {
      const int m = cm[c];
      if (m < 0) continue;
      const double2 a = row[c];
      if (m == 0) {
        ok &= fabs(a.y) <= tol;
      } else {
        const double2 b = row[cmir[c]];
        const double sg = (m & 1) ? -1.0 : 1.0;
        ok &= fabs(b.x - sg * a.x) + fabs(b.y + sg * a.y) <= tol;
      }
    }
  }
  ok = __syncthreads_and(ok);
  cluster_wait();  // ranks past the shells come here at once, before the others may have started
  if (threadIdx.x < kGatherCtas) {  // to every CTA of the cluster
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.u32 [a], %2;\n\t}" ::"r"(
                     smem_u32(&s_ok[rank])),
                 "r"((uint32_t)threadIdx.x), "r"(ok)
                 : "memory");
  }
  cluster_sync();
  int s = 1;
#pragma unroll
  for (int i = 0; i < kGatherCtas; ++i) s &= s_ok[i];
  if (rank == 0 && threadIdx.x == 0) sym[prop] = s;
  int Lp = 1 << 30, Kp = K;
  if (rag) { Lp = rag[prop].L; Kp = rag[prop].K; }
  float2* ctp = ct + (size_t)prop * nc * ps;
  float* c3o = c3p + (size_t)prop * nc * (4 * c3row);
  for (int rd = 0; rd < ROUNDS; ++rd) {
    const int q = rank + kGatherCtas * rd;
#pragma unroll 2
    for (int i = threadIdx.x; i < 4 * nc; i += 256) {
      const int c = i >> 2, kk = i & 3, k = 4 * q + kk;
      const int m = cm[c];
      const bool mir = s && m < 0, odd = m & 1;
      float2 v = make_float2(0.f, 0.f);  // absent orders / shells
      if (cl[c] <= Lp && k < Kp) {
        const double2 a = gl_smem[(4 * rd + kk) * ld + (mir ? cmir[c] : c)];
        v = make_float2(narrow(flip(a.x, mir && odd)), (s && m == 0) ? 0.f : narrow(flip(a.y, mir && !odd)));
      }
      ctp[(size_t)c * ps + k] = v;
      if (m >= 0 || !s) {
        float* o = c3o + (size_t)c * (4 * c3row) + 8 * q + kk;
        o[0] = v.x;
        o[4] = v.y;
      }
    }
  }
}

// FP32 T [lt][ki] of a proposal -> the TF32 split operand's rows [ki][lt] (hi, lo), 64 x 32
// tiles through shared memory; the column beside an odd last one gets 0.  grid: (klp / 32, lt tiles, n); block (32, 8).
// Memory-bound: 6.6 MB read (mostly L2) and 13.6 MB written a proposal at L = 18, K = 26.
// Writing these rows from the coupling itself costs a sector per value and array.
__global__ void __launch_bounds__(256) k_split_rows(const float* __restrict__ T, int n_lt, int klp, int KP, int ldT32,
                                                    float* __restrict__ hi, float* __restrict__ lo) {
  __shared__ float tile[64][33];
  grid_wait();
  grid_release();
  const int ki0 = blockIdx.x * 32, lt0 = blockIdx.y * 64;
  const float* src = after_wait(T) + (size_t)blockIdx.z * klp * ldT32 + ki0 + threadIdx.x;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int r = threadIdx.y + 8 * j;
    tile[r][threadIdx.x] = lt0 + r < n_lt ? src[(size_t)(lt0 + r) * klp] : 0.f;
  }
  __syncthreads();
  const int lt = lt0 + 2 * threadIdx.x;
  if (lt >= n_lt) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int r = threadIdx.y + 8 * j;
    const float2 t = make_float2(tile[2 * threadIdx.x][r], tile[2 * threadIdx.x + 1][r]);
    uint32_t h0, h1;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h0) : "f"(t.x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h1) : "f"(t.y));
    const float2 h = make_float2(__uint_as_float(h0), __uint_as_float(h1));
    const size_t at = ((size_t)blockIdx.z * klp + ki0 + r) * KP + lt;
    *reinterpret_cast<float2*>(hi + at) = h;
    *reinterpret_cast<float2*>(lo + at) = make_float2(t.x - h.x, t.y - h.y);
  }
}

constexpr int kGatherMaxSmem = 8 * 1025 * 16;  // two rounds of four shells, nc <= 1024

}  // namespace

// ---- host side ----------------------------------------------------------------

std::string build_lane_tables(const std::vector<PairBlock>& pbs, const std::vector<int>& coff, const Wigner3jTable& w3j,
                              std::vector<LaneBlock>& blks, std::vector<LaneQuad>& quads, std::vector<int4>& gcols,
                              std::vector<float4>& w, int& crows, int& wmax, int& c3rows) {
  blks.clear(); quads.clear(); gcols.clear(); w.clear();
  crows = wmax = c3rows = 0;
  std::string bad;
  // one quad (m3 .. m3 + 3) of orders s0 .. s1 - 1: its rows and, when put, 3j values; steps run
  // over the m of the shorter row, the other row slides with m3
  auto quad_of = [&](const PairBlock& pb, int m3, int s0, int s1, bool put) {
    const int l1 = pb.l1, l2 = pb.l2, a = std::min(l1, l2), b = std::max(l1, l2);
    const bool swap = l1 > l2;
    LaneQuad q{};
    q.m3 = m3;
    q.c0 = s0;
    q.rs = s1 - s0;
    int lo = std::max(-a, -b - m3 - 3), hi = std::min(a, b - m3);
    if ((hi - lo) & 1) ++hi;  // an odd number of steps (the form of the loop); the extra one is zero
    q.n = hi - lo + 1;
    // without swap: m1 = lo .. hi, window row k holds c_k2[-(m3 + k) - m1]; with swap: m2 =
    // hi .. lo, window row k holds c_k1[-(m3 + 3 - k) - m2].  Arrays start at row 3.
    q.x0 = (swap ? hi + l2 : lo + l1) + 3;
    q.vb = (swap ? -(m3 + 3) - hi + l1 : -m3 - lo + l2) + 3;
    const int xl = swap ? 2 * l2 + 7 : 2 * l1 + 7, vl = swap ? 2 * l1 + 7 : 2 * l2 + 7;
    const int sx = swap ? -1 : 1, sv = -sx;
    const int x1 = q.x0 + sx * (q.n - 1), v1 = q.vb + sv * (q.n + 2);
    if (q.n < 1 || std::min(q.x0, x1) < 0 || std::max(q.x0, x1) >= xl || std::min(q.vb, v1) < 0 || std::max(q.vb, v1) >= vl)
      bad = "lane tables: a quad leaves the staged rows";
    for (int i = 0; put && i < q.n; ++i)
      for (int s = s0; s < s1; ++s) {
        const int l3 = pb.l3min + 2 * s;
        float v[4];
        for (int k = 0; k < 4; ++k) {
          const int mm3 = m3 + k;
          const int m1 = swap ? -mm3 - (hi - i) : lo + i, m2 = -mm3 - m1;
          const bool in = std::abs(mm3) <= l3 && std::abs(m1) <= l1 && std::abs(m2) <= l2;
          v[k] = in ? (float)w3j(l1, l2, l3, m1, m2, mm3) : 0.f;
        }
        w.push_back(make_float4(v[0], v[1], v[2], v[3]));
      }
    return q;
  };
  // the quads from m3 (a multiple of 4) up of orders sa .. sb - 1, each with the orders that reach
  // it; returns their 3j values (float4)
  auto run_of = [&](const PairBlock& pb, int m3, int sa, int sb, bool put) {
    int len = 0, count = 0;
    for (; m3 <= pb.l3min + 2 * (sb - 1); m3 += 4, ++count) {
      const int least = m3 > 0 ? m3 : std::max(0, -(m3 + 3));  // least |m3| of the quad
      int s0 = sa;
      while (pb.l3min + 2 * s0 < least) ++s0;
      LaneQuad q = quad_of(pb, m3, s0, sb, put);
      q.wofs = len;
      len += q.n * q.rs;
      if (put) quads.push_back(q);
    }
    if (count > kLaneMaxQuads) bad = "lane tables: more quads than the kernel stages";
    return len;
  };
  // general coefficients: m3 from -l3 of the run's largest order, rows of both signs
  auto gen_run = [&](const PairBlock& pb, int sa, int sb, bool put) {
    return run_of(pb, -((pb.l3min + 2 * (sb - 1) + 3) / 4) * 4, sa, sb, put);
  };
  auto gen_rows = [&](const PairBlock& pb, int sa, int sb) {
    int r = 0;
    for (int s = sa; s < sb; ++s) r += 2 * (pb.l3min + 2 * s) + 1;
    return r;
  };
  for (const PairBlock& pb : pbs) {
    LaneBlock fb{};
    fb.l1 = pb.l1; fb.l2 = pb.l2; fb.l3min = pb.l3min; fb.nl3 = pb.nl3; fb.lt_base = pb.lt_base;
    fb.c1 = coff[pb.l1 >> 1]; fb.c2 = coff[pb.l2 >> 1];
    fb.swap = pb.l1 > pb.l2;
    fb.q0 = (int)quads.size();
    fb.w0 = (int)w.size();
    fb.wn = run_of(pb, 0, 0, pb.nl3, true);
    fb.nq = (int)quads.size() - fb.q0;
    blks.push_back(fb);
    crows = std::max(crows, 2 * std::max(pb.l1, pb.l2) + 7);
    wmax = std::max(wmax, fb.wn);
    int rows = 0;
    for (int s = 0; s < pb.nl3; ++s) {
      rows += pb.l3min + 2 * s + 1;
      wmax = std::max(wmax, gen_run(pb, s, s + 1, false));
      c3rows = std::max(c3rows, gen_rows(pb, s, s + 1));
    }
    c3rows = std::max(c3rows, rows);
  }
  // general coefficients: as few balanced runs of up to kLaneNC orders as fit the shared memory that
  // real functions and single orders take, so that the warps of an SM stay as many
  for (size_t i = 0; i < pbs.size(); ++i) {
    const PairBlock& pb = pbs[i];
    int gp = (pb.nl3 + kLaneNC - 1) / kLaneNC;
    auto fits = [&] {
      for (int r = 0; r < gp; ++r) {
        int s0, n;
        lane_run(pb.nl3, gp, r, s0, n);
        if (gen_rows(pb, s0, s0 + n) > c3rows || gen_run(pb, s0, s0 + n, false) > wmax) return false;
      }
      return true;
    };
    while (!fits()) ++gp;
    blks[i].gp = gp;
    for (int r = 0; r < 16; ++r) {
      int4 g = make_int4((int)quads.size(), 0, (int)w.size(), 0);
      if (r < gp) {
        int s0, n;
        lane_run(pb.nl3, gp, r, s0, n);
        g.w = gen_run(pb, s0, s0 + n, true);
        g.y = (int)quads.size() - g.x;
      }
      gcols.push_back(g);
    }
  }
  return bad;
}

// Units of every K' <= K: (offset in utab, units) in kofs[K'], 34 entries a unit: per lane
// shells of the block | staging offset | k2 | k1 (bits 24, 12, 6, 0; no shells: no pair), then
// the first slot and slots | (more than eight shells) << 16 | k3 block << 17.  A slot is two
// staging positions: half the even shell triple's index << 2 | which of the two are the unit's.
void build_lane_units(int K, std::vector<uint32_t>& utab, std::vector<uint32_t>& slots, std::vector<int2>& kofs,
                      int& stage) {
  utab.clear(); slots.clear();
  kofs.assign(K + 1, make_int2(0, 0));
  stage = kLaneNC * 64;  // the m3 = 0 values of a task
  for (int Kp = 1; Kp <= K; ++Kp) {
    kofs[Kp].x = (int)utab.size();
    for (int blk = 0; 16 * blk < Kp; ++blk) {
      std::vector<std::pair<int, int>> pr;  // (k1, k2)
      for (int k2 = Kp - 1; k2 >= 16 * blk; --k2)
        for (int k1 = k2; k1 < Kp; ++k1) pr.push_back({k1, k2});
      for (int p0 = 0; p0 < (int)pr.size(); p0 += 32, ++kofs[Kp].y) {
        const int n = std::min(32, (int)pr.size() - p0);
        auto shells = [&](int i) { return std::min(16, pr[p0 + i].second + 1 - 16 * blk); };
        std::vector<int> order(n), off(n);
        for (int i = 0; i < n; ++i) order[i] = i;
        std::sort(order.begin(), order.end(), [&](int a, int b) { return pr[p0 + a] < pr[p0 + b]; });
        const size_t s0 = slots.size();
        int pos = 0, next = -1, used[32] = {0};
        for (int i : order) {
          const int k1 = pr[p0 + i].first, k2 = pr[p0 + i].second;
          const int ki0 = k1 * (k1 + 1) * (k1 + 2) / 6 + k2 * (k2 + 1) / 2 + 16 * blk;
          if (ki0 != next) {
            pos = ((pos + 1) & ~1) + (ki0 & 1);
            int best = pos;
            for (int d = 2; d <= 8; d += 2)
              if (used[(pos + d) & 31] < used[best & 31]) best = pos + d;
            while (s0 + best / 2 > slots.size()) slots.push_back(0);
            pos = best;
          }
          ++used[pos & 31];
          off[i] = pos;
          next = ki0 + shells(i);
          for (int ki = ki0; ki < next; ++ki, ++pos) {
            if (s0 + pos / 2 == slots.size()) slots.push_back((uint32_t)(ki / 2) << 2);
            slots[s0 + pos / 2] |= 1u << (ki & 1);
          }
        }
        const int ns = (int)(slots.size() - s0);
        stage = std::max(stage, 2 * ns);
        for (int i = 0; i < 32; ++i)
          utab.push_back(i < n ? (uint32_t)shells(i) << 24 | (uint32_t)off[i] << 12 | (uint32_t)pr[p0 + i].second << 6 |
                                     (uint32_t)pr[p0 + i].first
                               : 0u);
        utab.push_back((uint32_t)s0);
        utab.push_back((uint32_t)ns | (shells(0) > 8 ? 1u << 16 : 0u) | (uint32_t)blk << 17);
      }
    }
  }
  stage = (stage + 3) / 4 * 4;
}

size_t lane_smem_bytes(const LaneTables& lt, int nw) {
  return (size_t)2 * lt.crows * lt.ps * 8 + ((size_t)lt.wmax + 8) * 16 + (size_t)lt.c3rows * lt.c3row * 16 +
         (size_t)nw * lt.stage * 4;
}

// Tasks of a block of nl3 orders (real functions) and nu units.
int lane_tasks(int nu, int nl3) { return nu * ((nl3 + kLaneNC - 1) / kLaneNC); }

// Warps per CTA: registers hold 16 warps per SM (128 a thread), so the split into CTAs that
// brings most of them together; on a tie the smaller CTA, whose idle tail and staging wait the
// SM's other CTAs cover.
void lane_pick_warps(LaneTables& lt) {
  lt.nw = 0;
  int best = 0;
  for (int nw : {4, 8, 16}) {
    const size_t b = lane_smem_bytes(lt, nw) + 2048;
    if (b > (size_t)kCoupleMaxDynSmem) continue;
    const int ctas = (int)std::min<size_t>(kLaneMaxWarps / nw, (size_t)(228 * 1024) / b);
    if (ctas * nw > best) { best = ctas * nw; lt.nw = nw; lt.ctas = ctas; }
  }
  lt.ok = lt.nw > 0;
  lt.smem = lt.ok ? lane_smem_bytes(lt, lt.nw) : 0;
}

cudaError_t lane_configure() {
  cudaError_t e = cudaFuncSetAttribute(k_couple_lane<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kCoupleMaxDynSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_couple_lane<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kCoupleMaxDynSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_gather_lane<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGatherMaxSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_gather_lane<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGatherMaxSmem);
  return e;
}

cudaError_t launch_gather_lane(const DevTables& t, const TcTables& tc, int n, const double2* coeff, CoeffLayout lay,
                               float2* ct, float* c3p, int* sym, cudaStream_t s, const RagInfo* rag) {
  const size_t row = (size_t)(t.nc | 1) * sizeof(double2);
  auto go = [&](auto kernel, int rounds) {
    kernel<<<dim3(kGatherCtas, n), 256, 4 * rounds * row, s>>>(t.K, t.nc, lay.stride, lay.map, tc.cm, tc.cmir, tc.cl, coeff,
                                                               ct, c3p, sym, rag, tc.err);
  };
  if (tc.lane.ps == 32)
    go(k_gather_lane<1>, 1);
  else
    go(k_gather_lane<2>, 2);
  return cudaGetLastError();
}

cudaError_t launch_couple_lane(const DevTables& t, const TcTables& tc, int n, const float2* ct, const float* c3p,
                               const int* sym, void* Thi, void* Tlo, bool tf32, float* T32, bool t32maj, float* scratch,
                               cudaStream_t s, const RagInfo* rag) {
  const LaneTables& lt = tc.lane;
  // a batch whose (block, proposal) CTAs do not fill the SMs spreads each block's tasks over Z CTAs
  // of four warps until they do, blocks strictly heaviest first (one proposal at L18 K26: 45 us in
  // CTAs of eight warps over twice the slots, 35 so, 43 with four times the CTAs, which stage more)
  const int slots = 2 * tc.nsm * lt.ctas;
  int z = 1, nw = lt.nw;
  size_t smem = lt.smem;
  if ((long long)tc.n_pb * n < slots) {
    nw = 4;
    smem = lane_smem_bytes(lt, nw);
    const int maxz = std::max(1, (lt.tasks + nw - 1) / nw);
    while (z < maxz && (long long)tc.n_pb * n * z < slots) ++z;
  }
  // TF32 rows are split from order-major FP32 T by a kernel of its own
  const bool rows = tf32 && Thi && !T32;
  LaneOut o;
  o.hi = rows ? nullptr : Thi;
  o.lo = rows ? nullptr : Tlo;
  o.T32 = rows ? scratch : T32;
  o.KP = tc.KP; o.klp = t.klp; o.ldT32 = t.n_ltp;
  o.tf32 = tf32; o.ltmaj = t_order_major(tc, tf32); o.t32maj = rows || t32maj;
  auto go = [&](auto kernel) {
    return launch_after(kernel, dim3(n, z, tc.n_pb), 32 * nw, smem, s, 1, ct, reinterpret_cast<const float4*>(c3p), t.K,
                        t.nc, z > 1 ? lt.by_work : lt.by_form, tc.coff, lt.blks, lt.quads, lt.gcols, lt.w, lt.utab,
                        lt.slots, lt.kofs, lt.crows, lt.wmax, lt.c3rows, lt.stage, sym, o, rag, tc.err);
  };
  const cudaError_t e = lt.ps == 32 ? go(k_couple_lane<32>) : go(k_couple_lane<64>);
  if (e != cudaSuccess || !rows) return e;
  return launch_after(k_split_rows, dim3(t.klp / 32, (t.n_lt + 63) / 64, n), dim3(32, 8), 0, s, 1, scratch, t.n_lt, t.klp,
                      tc.KP, t.n_ltp, (float*)Thi, (float*)Tlo);
}

}  // namespace tp3
