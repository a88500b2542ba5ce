// lambda != 0 on the tensor-core path: the Fourier-pair operand of the angular stage,
//   H[ki][q] = sum over the basis entries j of pair q of T[ki][lt(j)] w_j Y1 Y2 Y3
// with the shells' Legendre factors (src/correlations.jl:137-148), as split rows.
//
// A pair q = (m2, m3) up to sign fixes m1, m2, m3, so an l-triple holds exactly two entries of
// it, j and its mirror -j (one for q = (0, 0)), and both have the same product P = w Y1 Y2 Y3.
// The sum k_build_H_split forms -- the even and the odd entries of q in two accumulators, added
// at the end -- therefore has two equal halves: one accumulator, doubled, gives the same bits at
// half the work.  For q = (0, 0) the two accumulators are two slots, added at the end.
//
// One CTA takes four consecutive shell triples and NP proposals.  A lane owns one of the four
// triples and four pairs (a quad of columns), its warp eight quads: a 16-byte read of T serves
// four accumulator columns, and w Y1 Y2 Y3 is formed once for the NP proposals.  Quads that need
// the same l-triples share a warp's list, and a CTA's warps draw the lists from a queue, longest
// first.  The sums keep the order of the l-triples, so the bits are k_build_H_split's.
// Bound by instruction issue and shared-memory latency at 16 warps a SM (128 registers: 48 sums,
// 12 values of T); the FMA pipe is 46 % busy.  12 proposals at L18 K26: 500 us.  A lane per pair
// with all four triples in it read T with 12 16-byte loads for 24 packed FMAs: 818 us.  Weights
// straight from L2 a pair of terms ahead: 607 us; by blocks through shared memory, 562; y1 and y2
// reloaded only when l1 or l2 changes, next entry read early, 32-bit addresses: 500.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "internal.h"
#include "tc_prims.cuh"

namespace tp3 {
namespace {

constexpr int kHfMaxSmem = 226 * 1024;
constexpr int kHfThreads = 512;  // most of a CTA; two CTAs of half as many where T fits twice

// Shared memory by 32-bit address: a generic pointer costs two registers and 64-bit sums.
__device__ __forceinline__ float lds1(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}

template <int NP>
__global__ void __launch_bounds__(kHfThreads, 1) k_build_H_pairs(
    const float* __restrict__ T32, int klp, int64_t Tstride, int n, int klength, int n_lt,
    const float* __restrict__ Ytab, int nc, int L, const int4* __restrict__ kl, const int2* __restrict__ lists,
    const int2* __restrict__ entries, const float4* __restrict__ wts, const int4* __restrict__ quad_m,
    const int* __restrict__ quad_q, int nunits, int KP, int tf32, void* __restrict__ Hhi, void* __restrict__ Hlo,
    int* __restrict__ err) {
  extern __shared__ __align__(16) float hf_smem[];
  __shared__ int next;
  const int ncp = nc + 2 * L;                   // L zeros on each side: a pair with |m| > l reads them
  float* Ts = hf_smem;                          // [n_lt][4][NP]
  float* Ys = Ts + (size_t)n_lt * 4 * NP;       // [3][ncp][4]
  int4* Ms = reinterpret_cast<int4*>(Ys + 12 * ncp);  // [nunits][8]
  const int ki0 = blockIdx.x * 4, p0 = blockIdx.y * NP;
  if (threadIdx.x == 0) next = blockDim.x / 32;
  for (int i = threadIdx.x; i < 12 * ncp; i += blockDim.x) {
    const int u = i & 3, r = (i >> 2) / ncp, c = (i >> 2) - r * ncp - L;
    const int4 k = __ldg(kl + min(ki0 + u, klength - 1));
    Ys[i] = c >= 0 && c < nc ? Ytab[(size_t)(r == 0 ? k.x : r == 1 ? k.y : k.z) * nc + c] : 0.f;
  }
  for (int i = threadIdx.x; i < nunits * 8; i += blockDim.x) Ms[i] = __ldg(quad_m + i);
  grid_wait();
  grid_release();
  T32 = after_wait(T32);
  // rows of T are padded to a multiple of 16 shell triples, so a group's 16 bytes are always there
  for (int i = threadIdx.x; i < n_lt * NP; i += blockDim.x) {
    const int lt = i / NP, p = i - lt * NP;
    const float4 v = p0 + p < n ? __ldg(reinterpret_cast<const float4*>(
                                      T32 + (int64_t)(p0 + p) * Tstride + (int64_t)lt * klp + ki0))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
    float* d = Ts + lt * 4 * NP + p;
    d[0] = v.x; d[NP] = v.y; d[2 * NP] = v.z; d[3 * NP] = v.w;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, u = lane & 3, pos = lane >> 2;
  float4* Ws = reinterpret_cast<float4*>(Ms + nunits * 8) + (threadIdx.x >> 5) * 34;  // [4][8] values, 4 entries
  int2* Es = reinterpret_cast<int2*>(Ws + 32);
  const uint32_t Tu = (uint32_t)__cvta_generic_to_shared(Ts + u * NP);
  const uint32_t Yu = (uint32_t)__cvta_generic_to_shared(Ys + 4 * L + u);
  for (int unit = threadIdx.x >> 5; unit < nunits;) {
    const int4* mq = Ms + unit * 8 + pos;  // byte offsets of m2 (low half) and m3 (high half)
    uint32_t y3p[4];
    {
      const int4 m = *mq;
      const uint32_t c = Yu + 32 * ncp;
      y3p[0] = c + (m.x >> 16); y3p[1] = c + (m.y >> 16); y3p[2] = c + (m.z >> 16); y3p[3] = c + (m.w >> 16);
    }
    float2 acc[4][NP / 2];
    float y1[4] = {0.f, 0.f, 0.f, 0.f}, y2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int p = 0; p < NP / 2; ++p) acc[s][p] = make_float2(0.f, 0.f);
    auto term = [&](const int2 en, const float4 w) {
#ifdef TP3_DEBUG
      {  // the l-triple and the quad's three Legendre rows
        const int4 m = *mq;
        const uint32_t y = (uint32_t)__cvta_generic_to_shared(Ys), end = 48u * ncp;
        bool ok = en.x >= 0 && (en.x >> 4) < n_lt;
        const int ms[4] = {m.x, m.y, m.z, m.w};
        for (int s = 0; s < 4; ++s) {
          const int m2 = (short)ms[s], m3 = ms[s] >> 16;
          ok = ok && Yu + ((en.y & 1023) << 4) - m2 - m3 - y < 16u * ncp &&
               Yu + 16 * ncp + ((en.y >> 6) & (1023 << 4)) + m2 - y < 32u * ncp &&
               Yu + 32 * ncp + ((en.y >> 16) & (1023 << 4)) + m3 - y < end;
        }
        if (!TP3_DCHECK(ok, err)) return;
      }
#endif
      if (en.y < 0) {  // another l2
        const int4 m = *mq;
        const uint32_t b = Yu + 16 * ncp + ((en.y >> 6) & (1023 << 4));
        y2[0] = lds1(b + (short)m.x); y2[1] = lds1(b + (short)m.y); y2[2] = lds1(b + (short)m.z); y2[3] = lds1(b + (short)m.w);
        if (en.y & 1 << 30) {  // and another l1; m1 = -m2 - m3
          const uint32_t a = Yu + ((en.y & 1023) << 4);
          y1[0] = lds1(a - (short)m.x - (m.x >> 16)); y1[1] = lds1(a - (short)m.y - (m.y >> 16));
          y1[2] = lds1(a - (short)m.z - (m.z >> 16)); y1[3] = lds1(a - (short)m.w - (m.w >> 16));
        }
      }
      const int c3 = (en.y >> 16) & (1023 << 4);
      const uint32_t t4 = Tu + en.x * NP;
      float4 t[NP / 4];
#pragma unroll
      for (int p = 0; p < NP / 4; ++p) t[p] = lds4(t4 + 16 * p);
      const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const float P = wv[s] * y1[s] * y2[s] * lds1(y3p[s] + c3);
        const float2 P2 = make_float2(P, P);
#pragma unroll
        for (int p = 0; p < NP / 4; ++p) {
          acc[s][2 * p] = __ffma2_rn(P2, make_float2(t[p].x, t[p].y), acc[s][2 * p]);
          acc[s][2 * p + 1] = __ffma2_rn(P2, make_float2(t[p].z, t[p].w), acc[s][2 * p + 1]);
        }
      }
    };
    // Lists come in blocks of four terms: their 3j values and entries are fetched a block ahead into
    // registers, 16 bytes a lane, and read from the warp's 544 bytes of shared memory.
    // The tables end with a spare block.
    const int2 ls = __ldg(lists + unit);
    const int2* ep = entries + ls.x + (lane & 3);
    const float4* wp = wts + ls.x * 8 + lane;
    int2 en = __ldg(ep);
    float4 wn = __ldg(wp);
#pragma unroll 1
    for (int e = ls.x; e < ls.y; e += 4) {
      __syncwarp();
      Ws[lane] = wn;
      if (lane < 4) Es[lane] = en;
      __syncwarp();
      ep += 4; wp += 32;
      en = __ldg(ep);
      wn = __ldg(wp);
      int2 cur = Es[0];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int2 nxt = Es[(i + 1) & 3];
        term(cur, Ws[i * 8 + pos]);
        cur = nxt;
      }
    }
    const int q = __ldg(quad_q + unit * 8 + pos);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      float v[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const float a = p & 1 ? acc[s][p >> 1].y : acc[s][p >> 1].x;
        v[s] = a + a;
      }
      // unit 0: column 0 and, beside it, the even entries of pair (0, 0)
      const float a0 = p & 1 ? acc[0][p >> 1].y : acc[0][p >> 1].x;
      const float b0 = __shfl_down_sync(0xffffffffu, a0, 4);
      if (unit == 0 && pos == 0) v[0] = b0 + a0;
      if (q < 0 || ki0 + u >= klength || p0 + p >= n || !TP3_DCHECK(q + 3 < KP, err)) continue;
      const size_t o = ((size_t)(p0 + p) * klp + ki0 + u) * KP + q;
      if (tf32) {
        float h[4], l[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          uint32_t x;
          asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(x) : "f"(v[s]));
          h[s] = __uint_as_float(x);
          l[s] = v[s] - h[s];
        }
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(Hhi) + o) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(Hlo) + o) = make_float4(l[0], l[1], l[2], l[3]);
      } else {
        __nv_bfloat162 h[2], l[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const __nv_bfloat16 x = __float2bfloat16_rn(v[2 * s]), y = __float2bfloat16_rn(v[2 * s + 1]);
          h[s] = __halves2bfloat162(x, y);
          l[s] = __halves2bfloat162(__float2bfloat16_rn(v[2 * s] - __bfloat162float(x)),
                                    __float2bfloat16_rn(v[2 * s + 1] - __bfloat162float(y)));
        }
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(Hhi) + o) =
            make_uint2(*reinterpret_cast<uint32_t*>(&h[0]), *reinterpret_cast<uint32_t*>(&h[1]));
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(Hlo) + o) =
            make_uint2(*reinterpret_cast<uint32_t*>(&l[0]), *reinterpret_cast<uint32_t*>(&l[1]));
      }
    }
    if (lane == 0) unit = atomicAdd(&next, 1);
    unit = __shfl_sync(0xffffffffu, unit, 0);
  }
}

size_t hf_smem_bytes(int np, int n_lt, int nc, int L, int nunits, int threads) {
  return ((size_t)n_lt * 4 * np + 12 * (size_t)(nc + 2 * L) + 32 * (size_t)nunits) * sizeof(float) + threads * 17;
}

// Proposals a CTA: the most of 12, 8, 4 that are needed and whose T fits: the more share w Y1 Y2 Y3, the
// better, up to a last pass that is mostly empty.  Whole calls at L = 18, K = 26, N = 16 by 12 / 8 / 4:
// 784 / 958 / 1097 us for 12 proposals, 1424 / 1550 / 2070 for 24, 2003 / 1995 / 2727 for 32 and
// 3895 / 3917 / 5353 for 64, but 1214 / 1044 / 1403 for 16 (as for 13 to 15), two passes either way.
int hf_pick(int n_lt, int nc, int L, int nunits, int n) {
  for (int np = n > 8 ? 12 : n > 4 ? 8 : 4; np; np -= 4)
    if (hf_smem_bytes(np, n_lt, nc, L, nunits, kHfThreads) <= (size_t)kHfMaxSmem) return np;
  return 0;
}

}  // namespace

std::string build_hform_tables(const std::vector<int>& coff, int n_lt, const int* lt_l1, const int* lt_l2,
                               const int* lt_l3, const std::vector<std::pair<int, int>>& pairs,
                               const std::vector<int>& qstart, const std::vector<int>& qlist,
                               const std::vector<int>& lt_of_j, const std::vector<float>& w, int KP,
                               std::vector<int2>& lists, std::vector<int2>& entries, std::vector<float>& wts,
                               std::vector<int>& quad_m, std::vector<int>& quad_q) {
  const int nq = (int)pairs.size(), nquads = KP / 4;
  if (nq == 0 || pairs[0] != std::make_pair(0, 0)) return "pair 0 is not (0, 0)";
  // the entry weight of every l-triple per column; column KP: the even entries of pair 0
  std::vector<std::vector<std::pair<int, float>>> sw(KP + 4);
  for (int e = qstart[0]; e < qstart[1]; ++e)
    sw[(e - qstart[0]) & 1 ? 0 : KP].push_back({lt_of_j[qlist[e]], w[qlist[e]]});
  for (int q = 1; q < nq; ++q) {
    if ((qstart[q + 1] - qstart[q]) & 1) return "a pair has an odd number of entries";
    for (int e = qstart[q]; e < qstart[q + 1]; e += 2) {
      const int a = qlist[e], b = qlist[e + 1];
      if (lt_of_j[a] != lt_of_j[b] || std::memcmp(&w[a], &w[b], 4) != 0) return "entries of a pair are not mirrored";
      sw[q].push_back({lt_of_j[a], w[a]});
    }
  }
  // the l-triples of a quad as bits; units grow from the quad with the fewest by the one that adds
  // the fewest, the last takes quad 0 and the even entries beside it
  const int nw = (n_lt + 63) / 64;
  std::vector<std::vector<uint64_t>> use(nquads + 1, std::vector<uint64_t>(nw, 0));
  std::vector<int> size(nquads + 1, 0);
  for (int q = 0; q < KP + 4; ++q)
    for (const auto& x : sw[q]) use[q / 4][x.first >> 6] |= 1ull << (x.first & 63);
  auto added = [&](const std::vector<uint64_t>& cur, int k) {
    int c = 0;
    for (int i = 0; i < nw; ++i) c += __builtin_popcountll(use[k][i] & ~cur[i]);
    return c;
  };
  std::vector<int> rem;
  for (int k = 1; k < nquads; ++k) rem.push_back(k);
  for (int k = 0; k <= nquads; ++k) size[k] = added(std::vector<uint64_t>(nw, 0), k);
  const int nunits = (nquads + 1 + 7) / 8;
  std::vector<std::vector<int>> units;
  for (int i = 0; i + 1 < nunits; ++i) {
    std::vector<int> un;
    std::vector<uint64_t> cur(nw, 0);
    while (un.size() < 8 && !rem.empty()) {
      size_t best = 0;
      int ba = INT_MAX;
      for (size_t j = 0; j < rem.size(); ++j) {
        const int a = added(cur, rem[j]);
        if (a < ba || (a == ba && !un.empty() && size[rem[j]] > size[rem[best]])) { ba = a; best = j; }
      }
      un.push_back(rem[best]);
      for (int x = 0; x < nw; ++x) cur[x] |= use[rem[best]][x];
      rem.erase(rem.begin() + best);
    }
    units.push_back(un);
  }
  units.push_back({0, nquads});
  units.back().insert(units.back().end(), rem.begin(), rem.end());
  std::reverse(units.begin(), units.end());
  auto unit_size = [&](const std::vector<int>& un) {
    std::vector<uint64_t> cur(nw, 0);
    int c = 0;
    for (int k : un) {
      c += added(cur, k);
      for (int x = 0; x < nw; ++x) cur[x] |= use[k][x];
    }
    return c;
  };
  std::stable_sort(units.begin() + 1, units.end(), [&](const auto& a, const auto& b) { return unit_size(a) > unit_size(b); });

  lists.clear(); entries.clear(); wts.clear();
  quad_m.assign((size_t)nunits * 32, 0);
  quad_q.assign((size_t)nunits * 8, -1);
  for (int i = 0; i < nunits; ++i) {
    std::vector<std::vector<float>> by(n_lt);
    for (size_t j = 0; j < units[i].size(); ++j) {
      const int k = units[i][j];
      if (k < nquads) quad_q[i * 8 + j] = k * 4;
      for (int s = 0; s < 4; ++s) {
        const int q = k * 4 + s, slot = (int)j * 4 + s;
        if (q < nq) {
          const int m2 = pairs[q].first, m3 = pairs[q].second;
          quad_m[i * 32 + slot] = ((16 * m2) & 0xffff) | 16 * m3 * 65536;
        }
        for (const auto& x : sw[q]) {
          if (by[x.first].empty()) by[x.first].assign(32, 0.f);
          by[x.first][slot] = x.second;
        }
      }
    }
    const int e0 = (int)entries.size();
    int q1 = -1, q2 = -1;
    for (int t = 0; t < n_lt; ++t)
      if (!by[t].empty()) {
        const int l1 = lt_l1[t], l2 = lt_l2[t], l3 = lt_l3[t];
        const int fresh = l1 != q1 ? INT_MIN | 1 << 30 : l2 != q2 ? INT_MIN : 0;
        entries.push_back(make_int2(
            16 * t, (coff[l1 / 2] + l1) | (coff[l2 / 2] + l2) << 10 | (coff[l3 / 2] + l3) << 20 | fresh));
        wts.insert(wts.end(), by[t].begin(), by[t].end());
        q1 = l1; q2 = l2;
      }
    while ((entries.size() - e0) & 3) {  // terms of weight 0 fill the last block
      entries.push_back(make_int2(entries.back().x, entries.back().y & ~(INT_MIN | 1 << 30)));
      wts.resize(wts.size() + 32, 0.f);
    }
    lists.push_back(make_int2(e0, (int)entries.size()));
  }
  entries.resize(entries.size() + 4, make_int2(0, 0));  // fetched ahead of the last block
  wts.resize(wts.size() + 128, 0.f);
  return "";
}

bool hform_fits(int n_lt, int nc, int L, int nunits) { return hf_pick(n_lt, nc, L, nunits, 1) > 0; }

cudaError_t hform_configure() {
  cudaError_t e;
  const cudaFuncAttribute ds = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if ((e = cudaFuncSetAttribute(k_build_H_pairs<4>, ds, kHfMaxSmem)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_build_H_pairs<8>, ds, kHfMaxSmem)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_build_H_pairs<12>, ds, kHfMaxSmem)) != cudaSuccess)
    return e;
  return cudaSuccess;
}

cudaError_t launch_build_H_pairs(const DevTables& t, const TcTables& tc, int n, const float* T32, void* Hhi, void* Hlo,
                                 bool tf32, cudaStream_t s) {
  const HformTables& h = tc.hf;
  const int np = hf_pick(t.n_lt, t.nc, h.L, h.nunits, n);
  // two CTAs a SM, where T fits twice: one stages while the other sums, and the lists, 18 of
  // uneven lengths at L = 18, spread better over 8 warps than over 16
  const bool two = 2 * (hf_smem_bytes(np, t.n_lt, t.nc, h.L, h.nunits, kHfThreads / 2) + 1024 + 64) <= 228 * 1024;
  const int threads = two ? kHfThreads / 2 : kHfThreads;
  const size_t smem = hf_smem_bytes(np, t.n_lt, t.nc, h.L, h.nunits, threads);
  auto go = [&](auto kernel) {
    return launch_after(
        kernel, dim3((t.klength + 3) / 4, (n + np - 1) / np), threads, smem, s, 1, T32, t.klp, (int64_t)t.klp * t.n_ltp, n, t.klength, t.n_lt, t.Ytab, t.nc, h.L, t.kl, h.lists, h.entries,
        reinterpret_cast<const float4*>(h.wts), reinterpret_cast<const int4*>(h.quad_m), h.quad_q, h.nunits, tc.KP,
        tf32 ? 1 : 0, Hhi, Hlo, tc.err);
  };
  switch (np) {
    case 12: return go(k_build_H_pairs<12>);
    case 8: return go(k_build_H_pairs<8>);
    case 4: return go(k_build_H_pairs<4>);
    default: return cudaErrorInvalidConfiguration;
  }
}

}  // namespace tp3
