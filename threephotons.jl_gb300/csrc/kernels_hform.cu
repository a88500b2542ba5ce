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
// One CTA takes up to four consecutive shells k3 of one pair (k1, k2) and NP proposals: a thread
// owns a slot (pair) and walks the l-triples, so w Y1 Y2 is formed once for the four shells and
// T comes as 16-byte broadcasts; only the l-triples some lane of the warp uses are listed.
// Bound by FP32 FMA and shared-memory broadcasts in balance (12 16-byte loads for 24 packed FMAs
// at NP = 12).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "internal.h"

namespace tp3 {
namespace {

constexpr int kHfThreads = 576;

template <int NP>
__global__ void __launch_bounds__(kHfThreads, 1) k_build_H_pairs(
    const float* __restrict__ T32, int klp, int64_t Tstride, int n, int n_lt, const float* __restrict__ Ytab, int nc,
    const int4* __restrict__ groups, const int2* __restrict__ lists, const int2* __restrict__ entries,
    const float* __restrict__ wts, const int* __restrict__ slot_m, int nslots, int nq, int KP, int tf32,
    void* __restrict__ Hhi, void* __restrict__ Hlo) {
  extern __shared__ __align__(16) float hf_smem[];
  float* Ts = hf_smem;                          // [n_lt][4][NP]
  float* Ys = Ts + (size_t)n_lt * 4 * NP;       // [6][nc]: k1, k2, then the four k3
  const int4 g = groups[blockIdx.x];            // first shell triple, shells, k1 | k2 << 8, first k3
  const int cnt = g.y, k1 = g.z & 255, k2 = g.z >> 8, p0 = blockIdx.y * NP;
  for (int i = threadIdx.x; i < 6 * nc; i += blockDim.x) {
    const int r = i / nc, c = i - r * nc;
    Ys[i] = Ytab[(size_t)(r == 0 ? k1 : r == 1 ? k2 : g.w + min(r - 2, cnt - 1)) * nc + c];
  }
  for (int i = threadIdx.x; i < n_lt * NP; i += blockDim.x) {
    const int lt = i / NP, p = i - lt * NP;
    const float* src = T32 + (int64_t)(p0 + p) * Tstride + (int64_t)lt * klp + g.x;
#pragma unroll
    for (int u = 0; u < 4; ++u) Ts[(lt * 4 + u) * NP + p] = p0 + p < n && u < cnt ? src[u] : 0.f;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int s0 = 0; s0 < nslots; s0 += blockDim.x) {
    const int slot = s0 + threadIdx.x;
    if (slot - lane >= nslots) break;  // whole warps
    const int mm = slot < nslots ? slot_m[slot] : 0;
    const int m1 = (mm << 24) >> 24, m2 = (mm << 16) >> 24, m3 = (mm << 8) >> 24;
    const float *y1 = Ys + m1, *y2 = Ys + nc + m2, *y3 = Ys + 2 * nc + m3;
    float2 acc[4][NP / 2];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int p = 0; p < NP / 2; ++p) acc[u][p] = make_float2(0.f, 0.f);
    const int2 ls = lists[slot >> 5];
    auto term = [&](const int2 en, const float w) {
      if (w == 0.f) return;
      const float y = w * y1[en.y & 1023] * y2[(en.y >> 10) & 1023];
      const float* yr = y3 + (en.y >> 20);
      const float4* t4 = reinterpret_cast<const float4*>(Ts + en.x * (4 * NP));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float P = y * yr[u * nc];
        const float2 P2 = make_float2(P, P);
#pragma unroll
        for (int p = 0; p < NP / 4; ++p) {
          const float4 t = t4[u * (NP / 4) + p];
          acc[u][2 * p] = __ffma2_rn(P2, make_float2(t.x, t.y), acc[u][2 * p]);
          acc[u][2 * p + 1] = __ffma2_rn(P2, make_float2(t.z, t.w), acc[u][2 * p + 1]);
        }
      }
    };
    // l-triples (index, centres of the three orders' rows) and 3j values are fetched two ahead;
    // the tables end with two spare entries
    int2 ea = __ldg(entries + ls.x), eb = __ldg(entries + ls.x + 1);
    float wa = __ldg(wts + (size_t)ls.x * 32 + lane), wb = __ldg(wts + (size_t)ls.x * 32 + 32 + lane);
    for (int e = ls.x; e < ls.y; e += 2) {
      const int f = min(e + 2, ls.y);
      const int2 ec = __ldg(entries + f), ed = __ldg(entries + f + 1);
      const float wc = __ldg(wts + (size_t)f * 32 + lane), wd = __ldg(wts + (size_t)f * 32 + 32 + lane);
      term(ea, wa);
      if (e + 1 < ls.y) term(eb, wb);
      ea = ec; eb = ed; wa = wc; wb = wd;
    }
    const int q = slot - 1;  // slots 0 and 1: the even and odd entries of q = 0
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const float a = p & 1 ? acc[u][p >> 1].y : acc[u][p >> 1].x;
        const float b = __shfl_up_sync(0xffffffffu, a, 1);
        const float v = slot == 1 ? b + a : a + a;
        if (slot < 1 || slot >= nslots || u >= cnt || p0 + p >= n) continue;
        const size_t o = ((size_t)(p0 + p) * klp + g.x + u) * KP + q;
        if (tf32) {
          uint32_t h;
          asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(v));
          reinterpret_cast<float*>(Hhi)[o] = __uint_as_float(h);
          reinterpret_cast<float*>(Hlo)[o] = v - __uint_as_float(h);
        } else {
          const __nv_bfloat16 h = __float2bfloat16_rn(v);
          reinterpret_cast<__nv_bfloat16*>(Hhi)[o] = h;
          reinterpret_cast<__nv_bfloat16*>(Hlo)[o] = __float2bfloat16_rn(v - __bfloat162float(h));
        }
      }
  }
  // pair columns past nq are zero
  const int pad = KP - nq;
  for (int i = threadIdx.x; i < cnt * NP * pad; i += blockDim.x) {
    const int c = i % pad, r = i / pad, u = r % cnt, p = p0 + r / cnt;
    if (p >= n) break;
    const size_t o = ((size_t)p * klp + g.x + u) * KP + nq + c;
    if (tf32) {
      reinterpret_cast<float*>(Hhi)[o] = 0.f;
      reinterpret_cast<float*>(Hlo)[o] = 0.f;
    } else {
      reinterpret_cast<__nv_bfloat16*>(Hhi)[o] = __float2bfloat16_rn(0.f);
      reinterpret_cast<__nv_bfloat16*>(Hlo)[o] = __float2bfloat16_rn(0.f);
    }
  }
}

template <int NP>
size_t hf_smem_bytes(int n_lt, int nc) { return ((size_t)n_lt * 4 * NP + 6 * (size_t)nc) * sizeof(float); }

// Proposals a CTA: the most of 12, 8, 4 that are needed and whose T fits.
int hf_pick(int n_lt, int nc, int n) {
  if (n > 8 && hf_smem_bytes<12>(n_lt, nc) <= (size_t)kPlainMaxSmem) return 12;
  if (n > 4 && hf_smem_bytes<8>(n_lt, nc) <= (size_t)kPlainMaxSmem) return 8;
  return hf_smem_bytes<4>(n_lt, nc) <= (size_t)kPlainMaxSmem ? 4 : 0;
}

}  // namespace

std::string build_hform_tables(const std::vector<int>& coff, int K, int n_lt, const int* lt_l1, const int* lt_l2,
                               const int* lt_l3, const std::vector<std::pair<int, int>>& pairs,
                               const std::vector<int>& qstart, const std::vector<int>& qlist,
                               const std::vector<int>& lt_of_j, const std::vector<float>& w, std::vector<int4>& groups,
                               std::vector<int2>& lists, std::vector<int2>& entries, std::vector<float>& wts,
                               std::vector<int>& slot_m) {
  const int nq = (int)pairs.size(), nslots = nq + 1;
  if (nq == 0 || pairs[0] != std::make_pair(0, 0)) return "pair 0 is not (0, 0)";
  // per slot the entry weight of every l-triple
  std::vector<std::vector<std::pair<int, float>>> sw(nslots);
  for (int e = qstart[0]; e < qstart[1]; ++e)
    sw[(e - qstart[0]) & 1].push_back({lt_of_j[qlist[e]], w[qlist[e]]});
  for (int q = 1; q < nq; ++q) {
    if ((qstart[q + 1] - qstart[q]) & 1) return "a pair has an odd number of entries";
    for (int e = qstart[q]; e < qstart[q + 1]; e += 2) {
      const int a = qlist[e], b = qlist[e + 1];
      if (lt_of_j[a] != lt_of_j[b] || std::memcmp(&w[a], &w[b], 4) != 0) return "entries of a pair are not mirrored";
      sw[q + 1].push_back({lt_of_j[a], w[a]});
    }
  }
  groups.clear(); lists.clear(); entries.clear(); wts.clear();
  slot_m.assign(nslots, 0);
  for (int s = 2; s < nslots; ++s) {
    const int m2 = pairs[s - 1].first, m3 = pairs[s - 1].second;
    slot_m[s] = ((-m2 - m3) & 255) | (m2 & 255) << 8 | (m3 & 255) << 16;
  }
  for (int s0 = 0; s0 < nslots; s0 += 32) {
    std::vector<std::vector<float>> by(n_lt);
    for (int s = s0; s < std::min(nslots, s0 + 32); ++s)
      for (const auto& x : sw[s]) {
        if (by[x.first].empty()) by[x.first].assign(32, 0.f);
        by[x.first][s - s0] = x.second;
      }
    const int e0 = (int)entries.size();
    for (int t = 0; t < n_lt; ++t)
      if (!by[t].empty()) {
        const int l1 = lt_l1[t], l2 = lt_l2[t], l3 = lt_l3[t];
        entries.push_back(make_int2(t, (coff[l1 / 2] + l1) | (coff[l2 / 2] + l2) << 10 | (coff[l3 / 2] + l3) << 20));
        wts.insert(wts.end(), by[t].begin(), by[t].end());
      }
    lists.push_back(make_int2(e0, (int)entries.size()));
  }
  entries.resize(entries.size() + 2, make_int2(0, 0));  // fetched ahead of the last term
  wts.resize(wts.size() + 64, 0.f);
  for (int k1 = 0; k1 < K; ++k1)
    for (int k2 = 0; k2 <= k1; ++k2)
      for (int k3 = 0; k3 <= k2; k3 += 4)
        groups.push_back(make_int4(k1 * (k1 + 1) * (k1 + 2) / 6 + k2 * (k2 + 1) / 2 + k3, std::min(4, k2 + 1 - k3),
                                   k1 | k2 << 8, k3));
  return "";
}

bool hform_fits(int n_lt, int nc) { return hf_pick(n_lt, nc, 1) > 0; }

cudaError_t hform_configure() {
  cudaError_t e;
  const cudaFuncAttribute ds = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if ((e = cudaFuncSetAttribute(k_build_H_pairs<4>, ds, kPlainMaxSmem)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_build_H_pairs<8>, ds, kPlainMaxSmem)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_build_H_pairs<12>, ds, kPlainMaxSmem)) != cudaSuccess)
    return e;
  return cudaSuccess;
}

cudaError_t launch_build_H_pairs(const DevTables& t, const TcTables& tc, int n, const float* T32, void* Hhi, void* Hlo,
                                 bool tf32, cudaStream_t s) {
  const HformTables& h = tc.hf;
  auto go = [&](auto kernel, int np, size_t smem) {
    kernel<<<dim3(h.ngroups, (n + np - 1) / np), kHfThreads, smem, s>>>(
        T32, t.klp, (int64_t)t.klp * t.n_ltp, n, t.n_lt, t.Ytab, t.nc, h.groups, h.lists, h.entries, h.wts, h.slot_m,
        t.nq + 1, t.nq, tc.KP, tf32 ? 1 : 0, Hhi, Hlo);
  };
  switch (hf_pick(t.n_lt, t.nc, n)) {
    case 12: go(k_build_H_pairs<12>, 12, hf_smem_bytes<12>(t.n_lt, t.nc)); break;
    case 8: go(k_build_H_pairs<8>, 8, hf_smem_bytes<8>(t.n_lt, t.nc)); break;
    case 4: go(k_build_H_pairs<4>, 4, hf_smem_bytes<4>(t.n_lt, t.nc)); break;
    default: return cudaErrorInvalidConfiguration;
  }
  return cudaGetLastError();
}

}  // namespace tp3
