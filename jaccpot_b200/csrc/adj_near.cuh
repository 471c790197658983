#pragma once
// Near-field adjoint, warp per leaf unit.  For the pair (k, l), d = x_k - x_l,
// q = (|d|^2 + eps^2)^-1/2, y = m_l w_k - m_k w_l:
//   dL/dx_k += G q^3 (3 q^2 (y . d) d - y)
//   dL/dm_k += G q^3 (w_l . d)
// which needs l in near(k) <=> k in near(l) (the lists are symmetric).
//
// A close pair's m_l w_k and m_k w_l are each up to a thousand times the result
// and nearly cancel where the cotangent varies slowly, so y is formed first, as
// the difference of two rounded products with what the second's rounding left
// out put back (Kahan): to about an ulp of y itself, whatever the masses, and
// exactly 0 for w = const and equal masses or for w = m times powers of two.  Summing
// the terms apart (m_k sum q^3 w_l - w_k sum q^3 m_l + ..., 26 operations a pair)
// left the rounding of the large sums in the small result.  Against FP64, Plummer
// sphere of 131,072, w = x, 2-norm / largest over max(rms, value): 3.0e-7 / 1.6e-6,
// 2.2e-4 / 1.0e-3 with the terms apart, 7.2e-5 / 1.6e-4 with each pair's three
// terms added in turn; w random 2.0e-7 / 2.1e-6, 3.4e-7 / 7.0e-6, 5.4e-7 / 6.8e-6.
//
// 35 FP32 operations and one rsqrt a pair; the sources come two to an instruction
// (f32x2), staged per coordinate as in k_leaf_units_flat.  Bound by the FMA pipe
// (70% busy at a Plummer sphere of 262k, 529 M pairs in 0.79 ms; L1 49%).  A
// gradient call at 1M, order 6: 7.55 ms, 7.13 with the terms apart, 10.9 with one
// lane per target and the three terms in turn.
#include "fmm_kernels.cuh"

namespace jb {

constexpr int kAdjChunk = 32;             // sources per chunk (item)
constexpr int kAdjSlot = kAdjChunk + 4;   // slot stride: the slots one load reads use distinct banks

// Four ring slots of sources per coordinate (x, y, z, m, w), the targets and
// their sums (dL/dx, dL/dm)/G.
struct alignas(16) AdjStage {
  float v[7][4][kAdjSlot];
  float4 tp[32], tw[32], sum[32];
};

// One target against NS staged sources (a multiple of 4) at position o of
// slot sl; SELF: source self_j is the target.
template <bool SELF>
__device__ __forceinline__ float4 adj_chunk(const AdjStage& st, int sl, int o, int ns, float4 t, float4 w, int self_j,
                                            float eps2) {
  const f32x2 TX = f2(t.x, t.x), TY = f2(t.y, t.y), TZ = f2(t.z, t.z), E2 = f2(eps2, eps2);
  const f32x2 NX = f2(-w.x, -w.x), NY = f2(-w.y, -w.y), NZ = f2(-w.z, -w.z);
  const f32x2 M = f2(t.w, t.w), NM = f2(-t.w, -t.w), M3 = f2(-3.f, -3.f);
  f32x2 X = f2(0.f, 0.f), Y = X, Z = X, D = X;
  // -y = m_k w_l - m_l w_k, one component
  auto minus_y = [&](f32x2 nw, f32x2 sm, f32x2 ws) {
    const f32x2 p = f2_mul(M, ws);
    return f2_sub(f2_fma(sm, nw, p), f2_fma(NM, ws, p));
  };
  auto pair2 = [&](f32x2 sx, f32x2 sy, f32x2 sz, f32x2 sm, f32x2 wx, f32x2 wy, f32x2 wz, int j0) {
    const f32x2 dx = f2_sub(TX, sx), dy = f2_sub(TY, sy), dz = f2_sub(TZ, sz);
    const f32x2 d2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_fma(dz, dz, E2)));
    float a, b;
    f2_split(d2, a, b);
    float qa = rsqrt_ftz(a), qb = rsqrt_ftz(b);
    if (SELF) {
      qa = j0 == self_j ? 0.f : qa;
      qb = j0 + 1 == self_j ? 0.f : qb;
    }
    const f32x2 q = f2(qa, qb), q2 = f2_mul(q, q), q3 = f2_mul(q2, q);
    const f32x2 yx = minus_y(NX, sm, wx), yy = minus_y(NY, sm, wy), yz = minus_y(NZ, sm, wz);
    const f32x2 g = f2_mul(f2_mul(q2, M3), f2_fma(yx, dx, f2_fma(yy, dy, f2_mul(yz, dz))));
    X = f2_fma(q3, f2_fma(g, dx, yx), X);
    Y = f2_fma(q3, f2_fma(g, dy, yy), Y);
    Z = f2_fma(q3, f2_fma(g, dz, yz), Z);
    D = f2_fma(q3, f2_fma(wx, dx, f2_fma(wy, dy, f2_mul(wz, dz))), D);
  };
  const ulonglong2* V[7];
#pragma unroll
  for (int k = 0; k < 7; ++k) V[k] = reinterpret_cast<const ulonglong2*>(&st.v[k][sl][o]);
#pragma unroll 4
  for (int i = 0; i < ns / 4; ++i) {
    const ulonglong2 x = V[0][i], y = V[1][i], z = V[2][i], m = V[3][i], wx = V[4][i], wy = V[5][i], wz = V[6][i];
    pair2(x.x, y.x, z.x, m.x, wx.x, wy.x, wz.x, 4 * i);
    pair2(x.y, y.y, z.y, m.y, wx.y, wy.y, wz.y, 4 * i + 2);
  }
  auto sum = [](f32x2 v) {
    float lo, hi;
    f2_split(v, lo, hi);
    return lo + hi;
  };
  return make_float4(sum(X), sum(Y), sum(Z), sum(D));
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

__device__ __forceinline__ float4 shfl_down4(float4 v, int o) {
  return make_float4(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o),
                     __shfl_down_sync(0xffffffffu, v.z, o), __shfl_down_sync(0xffffffffu, v.w, o));
}

__device__ __forceinline__ void adj_stage(AdjStage& s, int sl, int q, float4 p, float4 w) {
  s.v[0][sl][q] = p.x;
  s.v[1][sl][q] = p.y;
  s.v[2][sl][q] = p.z;
  s.v[3][sl][q] = p.w;
  s.v[4][sl][q] = w.x;
  s.v[5][sl][q] = w.y;
  s.v[6][sl][q] = w.z;
}

// The targets rg (at most 32, of the leaf lr) against the unit's sources.
// The chunk-major walk of leaf_unit_flat: item f = c * nt + t is target t
// against chunk c, 32 items a step, so every lane works.  A step of 17 to 32
// targets spans at most three chunks, and four ring slots hold them.  Fewer
// targets are taken G = 2 or 4 times, copy h of a target against the h-th part
// of each chunk, one chunk a step.
template <int G>
__device__ __forceinline__ void adj_unit(const float4* __restrict__ pos4, const float4* __restrict__ w4, int2 rg,
                                         int4 U, int2 aux, const int2* __restrict__ runs, AdjStage& S, int lane,
                                         float G_, float eps2, float4* __restrict__ out, float4* __restrict__ partial,
                                         int2 lr, int row) {
  constexpr int CH = kAdjChunk, PART = CH / G;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const int nt = rg.y - rg.x + 1, items = nt * G;
  const bool tgt = lane < nt;
  S.tp[lane] = tgt ? pos4[rg.x + lane] : zero4;
  S.tw[lane] = tgt ? w4[rg.x + lane] : zero4;
  S.sum[lane] = zero4;
  __syncwarp();
  // adds the items' sums, G lanes to a target, in lane order
  auto add_items = [&](float4 v, int nl) {
#pragma unroll
    for (int h = 1; h < G; ++h) {
      const float4 a = shfl_down4(v, h);
      if (lane % G == 0) v = add4(v, a);
    }
    if (lane % G == 0 && lane < nl) S.sum[lane / G] = add4(S.sum[lane / G], v);
  };
  if (aux.y & 1) {  // the leaf itself, 32 at a time, the diagonal excluded
    for (int b = lr.x; b <= lr.y; b += 32) {
      const bool ok = b + lane <= lr.y;
      __syncwarp();  // the previous chunk's reads are done
      adj_stage(S, 0, lane, ok ? pos4[b + lane] : JB_PAD4, ok ? w4[b + lane] : zero4);
      __syncwarp();
      const int t = min(lane / G, nt - 1), h = lane % G;
      add_items(adj_chunk<true>(S, 0, h * PART, PART, S.tp[t], S.tw[t], rg.x + t - b - h * PART, eps2), items);
    }
  }
  const int nsrc = U.w;
  if (nsrc > 0) {
    const int C = (nsrc + CH - 1) / CH;
    int r = U.y, rbase = 0;
    int2 run = runs[r];
    float4 np, nw;  // the next chunk's source of this lane, in flight
    auto fetch = [&](int f) {
      while (f >= rbase + run.y && r + 1 < U.z) {
        rbase += run.y;
        ++r;
        run = runs[r];
      }
      np = f < nsrc ? pos4[run.x + (f - rbase)] : JB_PAD4;
      nw = f < nsrc ? w4[run.x + (f - rbase)] : zero4;
    };
    fetch(lane);
    if (G > 1) {  // one chunk a step, all its items at once
      for (int c = 0; c < C; ++c) {
        __syncwarp();
        adj_stage(S, c & 1, lane, np, nw);
        if (c + 1 < C) fetch((c + 1) * CH + lane);
        __syncwarp();
        const int t = min(lane / G, nt - 1), h = lane % G;
        add_items(adj_chunk<false>(S, c & 1, h * PART, PART, S.tp[t], S.tw[t], -1, eps2), items);
      }
    } else {
      const int total = nt * C;
      int staged = 0;
      int c = (lane >= nt) ? 1 : 0, t = lane - c * nt;  // item f = lane
      for (int base = 0; base < total; base += 32) {
        const int need = min(__shfl_sync(0xffffffffu, c, 31), C - 1);
        __syncwarp();  // the previous step's reads and adds are done
        while (staged <= need) {
          adj_stage(S, staged & 3, lane, np, nw);
          if (++staged < C) fetch(staged * CH + lane);
        }
        __syncwarp();
        const float4 v = adj_chunk<false>(S, c & 3, 0, CH, S.tp[t], S.tw[t], -1, eps2);
        const float4 v2 = shfl_down4(v, nt);
        if (tgt && base + lane < total) {
          float4 a = add4(S.sum[t], v);
          if (lane + nt < 32 && base + lane + nt < total) a = add4(a, v2);  // lane + nt holds (t, c + 1)
          S.sum[t] = a;
        }
        t += 32 - nt;  // item f + 32
        c += 1;
        if (t >= nt) {
          t -= nt;
          c += 1;
        }
      }
    }
  }
  __syncwarp();
  if (tgt) {
    const float4 v = S.sum[lane];
    const float4 res = make_float4(G_ * v.x, G_ * v.y, G_ * v.z, G_ * v.w);
    if (aux.x < 0) out[rg.x + lane] = res;
    else partial[(size_t)aux.x * kMaxLeaf + row + lane] = res;
  }
}

static __global__ void __launch_bounds__(32 * kWarpsPerBlock) k_adj_near(
    const float4* __restrict__ pos4, const float4* __restrict__ w4, int num_internal, int num_units,
    const int4* __restrict__ units, const int2* __restrict__ aux, const int2* __restrict__ runs,
    const int2* __restrict__ ranges, float G, float eps2, float4* __restrict__ out, float4* __restrict__ partial) {
  __shared__ AdjStage sA[kWarpsPerBlock];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int u = blockIdx.x * kWarpsPerBlock + warp;
  if (u >= num_units) return;
  const int4 U = units[u];
  const int2 ax = aux[u];
  const int2 rg = ranges[num_internal + U.x];
  const int n = rg.y - rg.x + 1;
  if (n > kMaxLeaf) return;  // a split leaf's partial row holds kMaxLeaf targets (jb_validate_leaves)
  for (int row = 0; row < n; row += 32) {  // a leaf of more than 32 particles in two passes
    const int2 rt = make_int2(rg.x + row, min(rg.y, rg.x + row + 31));
    const int nt = rt.y - rt.x + 1;
    if (row > 0) __syncwarp();  // the first pass's reads of the stage are done
    if (nt <= 8) adj_unit<4>(pos4, w4, rt, U, ax, runs, sA[warp], lane, G, eps2, out, partial, rg, row);
    else if (nt <= 16) adj_unit<2>(pos4, w4, rt, U, ax, runs, sA[warp], lane, G, eps2, out, partial, rg, row);
    else adj_unit<1>(pos4, w4, rt, U, ax, runs, sA[warp], lane, G, eps2, out, partial, rg, row);
  }
}

}  // namespace jb
