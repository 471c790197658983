#pragma once
// Adjoint (vector-Jacobian product) of the evaluation pass at fixed topology:
// given w (one 3-vector per sorted particle), the gradient of
// L = sum_i w_i . a_i with respect to the sorted positions and masses, with the
// COM expansion centres differentiated too.  This is what the reference's
// differentiable_accelerations gives jax.grad (runtime/fmm_evaluate.py:542-731,
// :1175-1250; analytic near-field VJP nearfield/grad.py:726-869; analytic L2P
// VJP operators/real_p2m_l2p.py:402-491), written as hand-made reverse kernels.
//
// Reverse order:
//   near      P2P adjoint, gathered over the (symmetric) neighbour lists
//   leaf far  L2P adjoint: Lbar_leaf = -G sum_i (w_i . grad) U, and the
//             Hessian-vector product for the particle
//   L2L       Lbar_a = sum of M2M(c_a - c_leaf) Lbar_leaf over a's leaves, up the
//             tree (L2L(d)^T = M2M(d))
//   M2L       Mbar_u += sum_v M2L(c_v - c_u) Lbar_v (M2L is symmetric), and
//             the displacement derivative -D(order p+1 M2L) per pair
//   nodes     cbar_n = Lbar_n . D L_n - M_n . D Mbar_n + the pairs' terms, with
//             L_n and Mbar_n the node's own M2L sums
//   M2M       Mbar_leaf += L2L(c_leaf - c_a) Mbar_a over the leaf's ancestors with
//             far pairs, and the chain of the centres of mass
//   P2M       per particle: mass and position terms
// The far field is written as (leaf <- ancestors) both ways, as the forward's
// L2L straight to the leaves: shifting an expansion is exact, so the centres
// in between carry no derivative, and a node without far pairs none at all.
// The sweeps level by level (jb_adj_l2l_level, jb_adj_m2m_level, jb_adj_p2m with
// a leaf-far stage that fills cbar4) give the same gradients from complete
// locals at every node, with a launch per level: the C ABI's plain sequence,
// which Pass.vjp does not take and the tests check the other against.
// Transposes come for free: the real M2L matrix is symmetric and
// M2M(d)^T = L2L(d) for the same displacement (both checked in the tests).
// Every output element has one writer per launch (no atomics).
//
// cbar4[node] = (dL/dc_x, dL/dc_y, dL/dc_z, dL/dmu) accumulates over stages;
// xm4[i] = (dL/dx, dL/dy, dL/dz, dL/dm) per sorted particle.
#include "fmm_kernels.cuh"

#include <algorithm>

namespace jb {

struct ArrF {
  const float* f;
  __device__ __forceinline__ float operator()(int k) const { return f[k]; }
};

// ---------------------------------------------------------------------------
// Leaf far field (L2P adjoint): warp per leaf, lane = particle.
//   Lbar_leaf  = -G sum_i sum_a w_ia D_a^T U(delta_i)
//   deltabar_i = -G grad_delta ( (sum_a w_ia D_a F) . U(delta_i) )
//   xbar_i -= deltabar_i ;  cbar_leaf += sum_i deltabar_i        (delta = c - x)
// Without cbar4, xm4 is set to the particles' far terms alone.
// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_adj_leaf_far(
    const float4* __restrict__ pos4, const float4* __restrict__ w4, int num_nodes, int num_internal,
    const int2* __restrict__ ranges, const float4* __restrict__ centers, const float* __restrict__ locals, float G,
    float4* __restrict__ xm4, float* __restrict__ lbar, float4* __restrict__ cbar4) {
  constexpr int C = csize(P), CS = cstride(P), CP = C + 1;
  extern __shared__ float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* red = smem + warp * 32 * CP;
  float* sF = smem + kWarpsPerBlock * 32 * CP + warp * CS;
  const int node = num_internal + blockIdx.x * kWarpsPerBlock + warp;
  if (node >= num_nodes) return;
  const int2 rg = ranges[node];
  const float4 c = centers[node];
  for (int k = lane; k < CS; k += 32) sF[k] = locals[(size_t)node * CS + k];
  float* myred = red + lane * CP;
#pragma unroll
  for (int k = 0; k < C; ++k) myred[k] = 0.f;
  __syncwarp();
  float cb0 = 0.f, cb1 = 0.f, cb2 = 0.f;
  for (int i = rg.x + lane; i <= rg.y; i += 32) {
    const float4 q = pos4[i];
    const float4 wv = w4[i];
    float U[C];
    solid_harmonics<P>(c.x - q.x, c.y - q.y, c.z - q.z, U);
    float Gw[C];
#pragma unroll
    for (int k = 0; k < C; ++k) Gw[k] = 0.f;
    for_ladder<P>([&](int a, int row, int col, float val) {
      const float wa = (a == 0) ? wv.x : ((a == 1) ? wv.y : wv.z);
      myred[col] += (-G * wa * val) * U[row];
      Gw[row] += (wa * val) * sF[col];
    });
    float phi, g[3];
    l2p_eval<P>(ArrF{Gw}, U, &phi, g);
    const float dbx = -G * g[0], dby = -G * g[1], dbz = -G * g[2];
    float4 x = cbar4 ? xm4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    x.x -= dbx;
    x.y -= dby;
    x.z -= dbz;
    xm4[i] = x;
    cb0 += dbx;
    cb1 += dby;
    cb2 += dbz;
  }
  __syncwarp();
  float* out = lbar + (size_t)node * CS;
  for (int k = lane; k < CS; k += 32) {
    float s = 0.f;
    if (k < C) {
#pragma unroll 8
      for (int j = 0; j < 32; ++j) s += red[j * CP + k];
    }
    out[k] = s;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    cb0 += __shfl_xor_sync(0xffffffffu, cb0, o);
    cb1 += __shfl_xor_sync(0xffffffffu, cb1, o);
    cb2 += __shfl_xor_sync(0xffffffffu, cb2, o);
  }
  if (lane == 0 && cbar4) {
    float4 cb = cbar4[node];
    cb.x += cb0;
    cb.y += cb1;
    cb.z += cb2;
    cbar4[node] = cb;
  }
}

// ---------------------------------------------------------------------------
// L2L adjoint, one level (parents in [first, last)), thread per parent:
//   X = L2L(d)^T Lbar_c = M2M(d) Lbar_c,  d = c_p - c_c
//   Lbar_p = X_left + X_right ;  g = X . D F_p ;  cbar_p += g, cbar_c -= g
// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(128) k_adj_l2l_level(int first, int last, const int* __restrict__ left,
                                                       const int* __restrict__ right,
                                                       const float4* __restrict__ centers,
                                                       const float* __restrict__ locals, float* __restrict__ lbar,
                                                       float4* __restrict__ cbar4) {
  constexpr int C = csize(P), CS = cstride(P);
  const int i = first + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= last) return;
  const float4 cp = centers[i];
  const float* Fp = locals + (size_t)i * CS;
  float* Lp = lbar + (size_t)i * CS;
  float4 cbp = cbar4[i];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int ch = side ? right[i] : left[i];
    const float4 cc = centers[ch];
    float X[C];
    const float* src = lbar + (size_t)ch * CS;
#pragma unroll
    for (int k = 0; k < C; ++k) X[k] = src[k];
    m2m_pair<P>(X, cp.x - cc.x, cp.y - cc.y, cp.z - cc.z);
    if (side == 0) {
#pragma unroll
      for (int k = 0; k < C; ++k) Lp[k] = X[k];
#pragma unroll
      for (int k = C; k < CS; ++k) Lp[k] = 0.f;
    } else {
#pragma unroll
      for (int k = 0; k < C; ++k) Lp[k] += X[k];
    }
    float g[3];
    ladder_dot3<P>(ArrF{X}, ArrF{Fp}, g);
    cbp.x += g[0];
    cbp.y += g[1];
    cbp.z += g[2];
    float4 cbc = cbar4[ch];
    cbc.x -= g[0];
    cbc.y -= g[1];
    cbc.z -= g[2];
    cbar4[ch] = cbc;
  }
  cbar4[i] = cbp;
}

// The three rows W_a = D_a^T X of the ladders at column k (for_ladder,
// transposed): X . D_a F = sum_k W_a[k] F[k].
__device__ __forceinline__ void ladder_col(const float* X, int k, float& wx, float& wy, float& wz) {
  wx = wy = wz = 0.f;
  const int n = (int)sqrtf((float)k + 0.5f), m = k - n * n - n, q = n - 1, a = m < 0 ? -m : m;
  if (n == 0) return;
  const float* R = X + q * q + q;  // R[m'] = X at degree n - 1
  if (m == 0) {
    wz = R[0];
    if (q >= 1) wx = -R[1], wy = -R[-1];
    return;
  }
  const float cm = 0.5f * R[a - 1], sm = a >= 2 ? 0.5f * R[1 - a] : 0.f;
  const float cp = a + 1 <= q ? 0.5f * R[a + 1] : 0.f, sp = a + 1 <= q ? 0.5f * R[-a - 1] : 0.f;
  wz = a <= q ? R[m] : 0.f;
  wx = m > 0 ? cm - cp : sm - sp;
  wy = m > 0 ? -sm - sp : cm + cp;
}

// ---------------------------------------------------------------------------
// M2L displacement derivative per far pair e = (t <- s):
//   g_e = Lbar_t . d/dd [M2L_p(d) M_s] = -Lbar_t . D (M2L_{p+1}(d) M_s),  d = c_t - c_s
// (the order p+1 triangular M2L carries exactly the degree n+1 terms that
// the derivative of the truncated degree-n coefficient needs).
//
// Thread per pair, up to kAdjPairs rounds of 32 consecutive pairs a warp (fewer
// where there are too few pairs to fill the GPU with that many), the source
// rows fetched by the whole warp a round ahead (k_m2l_units_coop).  The pairs
// are in target order, so a warp's share a target or two: the warp forms
// W_a = D_a^T Lbar_t once in shared memory and a pair's dot is 3 (p+2)^2 FMAs on
// broadcast words.  With a thread reading its own rows and the ladder written
// out per pair (300 terms at p = 6) the kernel took 1.66 ms at a Plummer sphere
// of 1M (18.9 M pairs); this form takes 1.43 beside the near field's adjoint.
// ---------------------------------------------------------------------------
constexpr int kAdjPairs = 8;

template <int P>
__host__ __device__ constexpr size_t adj_pairs_smem() {
  return sizeof(float4) * kM2LThreads * row4(P) + sizeof(int) * kM2LThreads +
         sizeof(float) * (kM2LThreads / 32) * 3 * cstride(P + 1);
}

template <int P>
__global__ void __launch_bounds__(kM2LThreads, 4) k_adj_m2l_pairs(int64_t num_pairs, const int* __restrict__ pair_tgt,
                                                                  const int* __restrict__ far_src,
                                                                  const float* __restrict__ mult,
                                                                  const float* __restrict__ lbar,
                                                                  const float4* __restrict__ centers,
                                                                  float4* __restrict__ g4, int rounds) {
  constexpr int C = csize(P), CS = cstride(P), C1 = csize(P + 1), CS1 = cstride(P + 1), R4 = row4(P), NW = CS / 4;
  extern __shared__ float4 m2l_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float4* wrows = m2l_smem + warp * 32 * R4;
  float4* row = wrows + lane * R4;
  int* ids = reinterpret_cast<int*>(m2l_smem + kM2LThreads * R4) + 32 * warp;
  float* W = reinterpret_cast<float*>(m2l_smem + kM2LThreads * R4 + kM2LThreads / 4) + warp * 3 * CS1;
  const int64_t base = ((int64_t)blockIdx.x * (kM2LThreads / 32) + warp) * 32 * rounds;
  if (base >= num_pairs) return;
  int s = base + lane < num_pairs ? far_src[base + lane] : -1;
  warp_rows_fetch<NW, R4>(wrows, ids, lane, s, mult, CS);
  int have = -1;  // the target W belongs to
  for (int it = 0; it < rounds; ++it) {
    const int64_t e = base + 32 * it + lane;
    const bool ok = e < num_pairs;
    const int t = ok ? pair_tgt[e] : -1;
    const float4 ct = ok ? centers[t] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 cs = ok ? centers[s] : ct;
    float v[C1];
    cp_async_wait_all();
    __syncwarp();  // the copies every lane issued into the warp's rows have landed
#pragma unroll
    for (int k = 0; k < CS / 4; ++k) {
      const float4 q = ok ? row[k] : make_float4(0.f, 0.f, 0.f, 0.f);
      if (4 * k + 0 < C) v[4 * k + 0] = q.x;
      if (4 * k + 1 < C) v[4 * k + 1] = q.y;
      if (4 * k + 2 < C) v[4 * k + 2] = q.z;
      if (4 * k + 3 < C) v[4 * k + 3] = q.w;
    }
#pragma unroll
    for (int k = C; k < C1; ++k) v[k] = 0.f;
    __syncwarp();  // every row (and every id) read before the next copies
    s = (it + 1 < rounds && e + 32 < num_pairs) ? far_src[e + 32] : -1;
    warp_rows_fetch<NW, R4>(wrows, ids, lane, s, mult, CS);
    float f[C1];
#pragma unroll
    for (int k = 0; k < C1; ++k) f[k] = 0.f;
    m2l_kfold_acc<P + 1>(v, f, ct.x - cs.x, ct.y - cs.y, ct.z - cs.z);
    for (unsigned todo = __ballot_sync(0xffffffffu, ok); todo;) {
      const int now = __shfl_sync(0xffffffffu, t, __ffs(todo) - 1);
      if (now != have) {
        __syncwarp();  // the last target's W is read
        for (int k = lane; k < CS1; k += 32) {
          float wx = 0.f, wy = 0.f, wz = 0.f;
          if (k < C1) ladder_col(lbar + (size_t)now * CS, k, wx, wy, wz);
          W[k] = wx;
          W[CS1 + k] = wy;
          W[2 * CS1 + k] = wz;
        }
        have = now;
        __syncwarp();
      }
      if (t == now) {
        float g[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int k = 0; k < CS1 / 4; ++k) {
            const float4 w = reinterpret_cast<const float4*>(W + a * CS1)[k];
            if (4 * k + 0 < C1) g[a] = fmaf(w.x, f[4 * k + 0], g[a]);
            if (4 * k + 1 < C1) g[a] = fmaf(w.y, f[4 * k + 1], g[a]);
            if (4 * k + 2 < C1) g[a] = fmaf(w.z, f[4 * k + 2], g[a]);
            if (4 * k + 3 < C1) g[a] = fmaf(w.w, f[4 * k + 3], g[a]);
          }
        g4[e] = make_float4(-g[0], -g[1], -g[2], 0.f);
      }
      todo &= ~__ballot_sync(0xffffffffu, t == now);
    }
  }
  cp_async_wait_all();  // nothing in flight (the last fetch copies nothing)
}

// Centre gradients, warp per node u with far pairs: for every pair e = (u <- v)
// g_e belongs to u as target and the reverse pair (v <- u), index rev[e],
// contributes -g_rev(e) to u as source; then Lbar_u . D L_u - M_u . D Mbar_u.
// Writes cbar4 (zero where there are no far pairs).  A thread per node took
// 0.43 ms for the gather alone (Plummer 1M, 200 pairs a node).
template <int P>
__global__ void __launch_bounds__(128) k_adj_nodes(int num_nodes, const int64_t* __restrict__ far_off,
                                                   const int* __restrict__ rev, const float4* __restrict__ g4,
                                                   const float* __restrict__ mult, const float* __restrict__ lbar,
                                                   const float* __restrict__ locals, int num_internal,
                                                   const float* __restrict__ own_rows,
                                                   const float* __restrict__ mbar, float4* __restrict__ cbar4) {
  constexpr int C = csize(P), CS = cstride(P);
  const int u = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (u >= num_nodes) return;
  const int64_t e0 = far_off[u], e1 = far_off[u + 1];
  float x = 0.f, y = 0.f, z = 0.f;
  if (e1 > e0) {
    for (int64_t e = e0 + lane; e < e1; e += 32) {
      const float4 a = g4[e], b = g4[rev[e]];
      x += a.x - b.x;
      y += a.y - b.y;
      z += a.z - b.z;
    }
    const size_t o = (size_t)u * CS;
    const float* F = u < num_internal ? locals + o : own_rows + (size_t)(u - num_internal) * CS;
    for (int k = lane; k < C; k += 32) {
      float wx, wy, wz;
      ladder_col(lbar + o, k, wx, wy, wz);
      const float f = F[k];
      x = fmaf(wx, f, x), y = fmaf(wy, f, y), z = fmaf(wz, f, z);
      ladder_col(mult + o, k, wx, wy, wz);
      const float h = -mbar[o + k];
      x = fmaf(wx, h, x), y = fmaf(wy, h, y), z = fmaf(wz, h, z);
    }
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, q);
      y += __shfl_xor_sync(0xffffffffu, y, q);
      z += __shfl_xor_sync(0xffffffffu, z, q);
    }
  }
  if (lane == 0) cbar4[u] = make_float4(x, y, z, 0.f);
}

// ---------------------------------------------------------------------------
// M2M adjoint + COM chain, one level (parents in [first, last)), root first:
//   Mbar_c += M2M(d)^T Mbar_p = L2L(d) Mbar_p,  d = c_c - c_p
//   g = (M2M(d) M_c) . D Mbar_p ; cbar_c += g, cbar_p -= g
//   then cbar_c += (mu_c / mu_p) cbar_p, mubar_c = mubar_p + (c_c - c_p).cbar_p / mu_p
// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(128) k_adj_m2m_level(int first, int last, const int* __restrict__ left,
                                                       const int* __restrict__ right,
                                                       const float4* __restrict__ centers,
                                                       const float* __restrict__ mult, float* __restrict__ mbar,
                                                       float4* __restrict__ cbar4) {
  constexpr int C = csize(P), CS = cstride(P);
  const int i = first + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= last) return;
  const float4 cp = centers[i];
  const float* Mbp = mbar + (size_t)i * CS;
  float4 cbp = cbar4[i];
  int chs[2] = {left[i], right[i]};
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int ch = chs[side];
    const float4 cc = centers[ch];
    float Y[C];
#pragma unroll
    for (int k = 0; k < C; ++k) Y[k] = Mbp[k];
    l2l_pair<P>(Y, cc.x - cp.x, cc.y - cp.y, cc.z - cp.z);
    float* Mbc = mbar + (size_t)ch * CS;
#pragma unroll
    for (int k = 0; k < C; ++k) Mbc[k] += Y[k];
    const float* Mc = mult + (size_t)ch * CS;
#pragma unroll
    for (int k = 0; k < C; ++k) Y[k] = Mc[k];
    m2m_pair<P>(Y, cc.x - cp.x, cc.y - cp.y, cc.z - cp.z);
    float g[3];
    ladder_dot3<P>(ArrF{Y}, ArrF{Mbp}, g);
    float4 cbc = cbar4[ch];
    cbc.x += g[0];
    cbc.y += g[1];
    cbc.z += g[2];
    cbar4[ch] = cbc;
    cbp.x -= g[0];
    cbp.y -= g[1];
    cbp.z -= g[2];
  }
  cbar4[i] = cbp;
  const float inv = cp.w > 0.f ? 1.f / cp.w : 0.f;
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int ch = chs[side];
    const float4 cc = centers[ch];
    const float f = cc.w * inv;
    float4 cbc = cbar4[ch];
    cbc.x += f * cbp.x;
    cbc.y += f * cbp.y;
    cbc.z += f * cbp.z;
    cbc.w = cbp.w + ((cc.x - cp.x) * cbp.x + (cc.y - cp.y) * cbp.y + (cc.z - cp.z) * cbp.z) * inv;
    cbar4[ch] = cbc;
  }
}

// ---------------------------------------------------------------------------
// P2M + leaf COM adjoint, warp per leaf, lane = particle, y = x - c:
//   gM = grad_y (Mbar . U(y)) ; cbar_tot = cbar_leaf - sum_j m_j gM_j
//   mbar_j += Mbar . U(y) + mubar + y . cbar_tot / mu
//   xbar_j += m_j gM + (m_j / mu) cbar_tot
// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_adj_p2m(const float4* __restrict__ pos4, int num_nodes,
                                                                  int num_internal, const int2* __restrict__ ranges,
                                                                  const float4* __restrict__ centers,
                                                                  const float* __restrict__ mbar,
                                                                  const float4* __restrict__ cbar4,
                                                                  float4* __restrict__ xm4) {
  constexpr int C = csize(P), CS = cstride(P);
  __shared__ float sM[kWarpsPerBlock][CS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int node = num_internal + blockIdx.x * kWarpsPerBlock + warp;
  if (node >= num_nodes) return;
  const int2 rg = ranges[node];
  const float4 c = centers[node];
  const float4 cb = cbar4[node];
  for (int k = lane; k < CS; k += 32) sM[warp][k] = mbar[(size_t)node * CS + k];
  __syncwarp();
  // pass 1: centre term
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
  for (int i = rg.x + lane; i <= rg.y; i += 32) {
    const float4 q = pos4[i];
    float U[C];
    solid_harmonics<P>(q.x - c.x, q.y - c.y, q.z - c.z, U);
    float phi, g[3];
    l2p_eval<P>(SmemF{sM[warp]}, U, &phi, g);
    s0 = fmaf(q.w, g[0], s0);
    s1 = fmaf(q.w, g[1], s1);
    s2 = fmaf(q.w, g[2], s2);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  const float tx = cb.x - s0, ty = cb.y - s1, tz = cb.z - s2;
  const float inv = c.w > 0.f ? 1.f / c.w : 0.f;
  // pass 2: particle terms
  for (int i = rg.x + lane; i <= rg.y; i += 32) {
    const float4 q = pos4[i];
    const float yx = q.x - c.x, yy = q.y - c.y, yz = q.z - c.z;
    float U[C];
    solid_harmonics<P>(yx, yy, yz, U);
    float phi, g[3];
    l2p_eval<P>(SmemF{sM[warp]}, U, &phi, g);
    float4 x = xm4[i];
    x.x += q.w * g[0] + q.w * inv * tx;
    x.y += q.w * g[1] + q.w * inv * ty;
    x.z += q.w * g[2] + q.w * inv * tz;
    x.w += phi + cb.w + (yx * tx + yy * ty + yz * tz) * inv;
    xm4[i] = x;
  }
}

// P2M adjoint with the chain of the centres of mass already summed per leaf
// (k_l2l_leaves<P, true>): with t = cbar_leaf / mu_leaf + chain.xyz, y = x - c_leaf,
//   dL/dx = far4 + m (grad_y (Mbar . U(y)) + t),  dL/dm = Mbar . U(y) + chain.w + y . t
// added to the near field's xm4.
template <int P>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_adj_particles(
    const float4* __restrict__ pos4, int num_nodes, int num_internal, const int2* __restrict__ ranges,
    const float4* __restrict__ centers, const float* __restrict__ mbar, const float4* __restrict__ cbar4,
    const float4* __restrict__ chain4, const float4* __restrict__ far4, float4* __restrict__ xm4) {
  constexpr int C = csize(P), CS = cstride(P);
  __shared__ float sM[kWarpsPerBlock][CS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int node = num_internal + blockIdx.x * kWarpsPerBlock + warp;
  if (node >= num_nodes) return;
  const int2 rg = ranges[node];
  const float4 c = centers[node], cb = cbar4[node], ch = chain4[node];
  for (int k = lane; k < CS; k += 32) sM[warp][k] = mbar[(size_t)node * CS + k];
  __syncwarp();
  const float inv = c.w > 0.f ? 1.f / c.w : 0.f;
  // a leaf without mass: its centre is the particles' mean, whatever their masses
  const float on = c.w > 0.f ? 1.f : 0.f;
  const float tx = on * fmaf(cb.x, inv, ch.x), ty = on * fmaf(cb.y, inv, ch.y), tz = on * fmaf(cb.z, inv, ch.z);
  for (int i = rg.x + lane; i <= rg.y; i += 32) {
    const float4 q = pos4[i], f = far4[i];
    const float yx = q.x - c.x, yy = q.y - c.y, yz = q.z - c.z;
    float U[C];
    solid_harmonics<P>(yx, yy, yz, U);
    float phi, g[3];
    l2p_eval<P>(SmemF{sM[warp]}, U, &phi, g);
    float4 x = xm4[i];
    x.x += f.x + q.w * (g[0] + tx);
    x.y += f.y + q.w * (g[1] + ty);
    x.z += f.z + q.w * (g[2] + tz);
    x.w += phi + ch.w + (yx * tx + yy * ty + yz * tz);
    xm4[i] = x;
  }
}

// ---------------------------------------------------------------------------
template <int P>
struct RunAdj {
  static int leaf_far(const float* pos4, const float* w4, int num_nodes, int num_internal, const int* ranges,
                      const float* centers, const float* locals, float G, float* xm4, float* lbar, float* cbar4,
                      cudaStream_t st);
  static int l2l_level(int first, int last, const int* left, const int* right, const float* centers,
                       const float* locals, float* lbar, float* cbar4, cudaStream_t st);
  static int m2l_pairs(int64_t num_pairs, const int* pair_tgt, const int* far_src, const float* mult,
                       const float* lbar, const float* centers, float* g4, cudaStream_t st);
  static int nodes(int num_nodes, const int64_t* far_off, const int* rev, const float* g4, const float* mult,
                   const float* lbar, const float* locals, int num_internal, const float* own_rows, const float* mbar,
                   float* cbar4, cudaStream_t st);
  static int l2l_hops(int num_hops, const int64_t* off, const int* items, const float* centers, float* lbar,
                      cudaStream_t st);
  static int leaves(int num_units, const int* units, const int* anc, const int* parent, const float* centers,
                    const float* cbar4, float* mbar, float* chain4, cudaStream_t st);
  static int particles(const float* pos4, int num_nodes, int num_internal, const int* ranges, const float* centers,
                       const float* mbar, const float* cbar4, const float* chain4, const float* far4, float* xm4,
                       cudaStream_t st);
  static int m2m_level(int first, int last, const int* left, const int* right, const float* centers,
                       const float* mult, float* mbar, float* cbar4, cudaStream_t st);
  static int p2m(const float* pos4, int num_nodes, int num_internal, const int* ranges, const float* centers,
                 const float* mbar, const float* cbar4, float* xm4, cudaStream_t st);
};

template <int P>
int RunAdj<P>::leaf_far(const float* pos4, const float* w4, int num_nodes, int num_internal, const int* ranges,
                        const float* centers, const float* locals, float G, float* xm4, float* lbar, float* cbar4,
                        cudaStream_t st) {
  const int L = num_nodes - num_internal;
  if (L <= 0) return JB_OK;
  const size_t sm = sizeof(float) * kWarpsPerBlock * (32 * (csize(P) + 1) + cstride(P));
  cudaFuncSetAttribute(k_adj_leaf_far<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_adj_leaf_far<P><<<blocks_for(L, kWarpsPerBlock), 32 * kWarpsPerBlock, sm, st>>>(
      reinterpret_cast<const float4*>(pos4), reinterpret_cast<const float4*>(w4), num_nodes, num_internal,
      reinterpret_cast<const int2*>(ranges), reinterpret_cast<const float4*>(centers), locals, G,
      reinterpret_cast<float4*>(xm4), lbar, reinterpret_cast<float4*>(cbar4));
  return launch_status();
}

template <int P>
int RunAdj<P>::l2l_level(int first, int last, const int* left, const int* right, const float* centers,
                         const float* locals, float* lbar, float* cbar4, cudaStream_t st) {
  if (last <= first) return JB_OK;
  k_adj_l2l_level<P><<<blocks_for(last - first, 128), 128, 0, st>>>(
      first, last, left, right, reinterpret_cast<const float4*>(centers), locals, lbar,
      reinterpret_cast<float4*>(cbar4));
  return launch_status();
}

template <int P>
int RunAdj<P>::m2l_pairs(int64_t num_pairs, const int* pair_tgt, const int* far_src, const float* mult,
                         const float* lbar, const float* centers, float* g4, cudaStream_t st) {
  if (num_pairs <= 0) return JB_OK;
  cudaFuncSetAttribute(k_adj_m2l_pairs<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)adj_pairs_smem<P>());
  const int rounds = (int)std::min<int64_t>(kAdjPairs, 1 + num_pairs / kM2LResident);
  k_adj_m2l_pairs<P><<<blocks_for(num_pairs, kM2LThreads * rounds), kM2LThreads, adj_pairs_smem<P>(), st>>>(
      num_pairs, pair_tgt, far_src, mult, lbar, reinterpret_cast<const float4*>(centers),
      reinterpret_cast<float4*>(g4), rounds);
  return launch_status();
}

template <int P>
int RunAdj<P>::nodes(int num_nodes, const int64_t* far_off, const int* rev, const float* g4, const float* mult,
                     const float* lbar, const float* locals, int num_internal, const float* own_rows, const float* mbar,
                     float* cbar4, cudaStream_t st) {
  k_adj_nodes<P><<<blocks_for(num_nodes, 4), 128, 0, st>>>(num_nodes, far_off, rev, reinterpret_cast<const float4*>(g4),
                                                           mult, lbar, locals, num_internal, own_rows, mbar,
                                                           reinterpret_cast<float4*>(cbar4));
  return launch_status();
}

template <int P>
int RunAdj<P>::l2l_hops(int num_hops, const int64_t* off, const int* items, const float* centers, float* lbar,
                        cudaStream_t st) {
  return launch_hops<P, true>(num_hops, off, items, nullptr, centers, lbar, st);
}

template <int P>
int RunAdj<P>::leaves(int num_units, const int* units, const int* anc, const int* parent, const float* centers,
                      const float* cbar4, float* mbar, float* chain4, cudaStream_t st) {
  return launch_l2l_leaves<P, true>(num_units, units, anc, centers, mbar, cbar4, chain4, parent, st);
}

template <int P>
int RunAdj<P>::particles(const float* pos4, int num_nodes, int num_internal, const int* ranges, const float* centers,
                         const float* mbar, const float* cbar4, const float* chain4, const float* far4, float* xm4,
                         cudaStream_t st) {
  const int L = num_nodes - num_internal;
  if (L <= 0) return JB_OK;
  k_adj_particles<P><<<blocks_for(L, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, st>>>(
      reinterpret_cast<const float4*>(pos4), num_nodes, num_internal, reinterpret_cast<const int2*>(ranges),
      reinterpret_cast<const float4*>(centers), mbar, reinterpret_cast<const float4*>(cbar4),
      reinterpret_cast<const float4*>(chain4), reinterpret_cast<const float4*>(far4), reinterpret_cast<float4*>(xm4));
  return launch_status();
}

template <int P>
int RunAdj<P>::m2m_level(int first, int last, const int* left, const int* right, const float* centers,
                         const float* mult, float* mbar, float* cbar4, cudaStream_t st) {
  if (last <= first) return JB_OK;
  k_adj_m2m_level<P><<<blocks_for(last - first, 128), 128, 0, st>>>(
      first, last, left, right, reinterpret_cast<const float4*>(centers), mult, mbar,
      reinterpret_cast<float4*>(cbar4));
  return launch_status();
}

template <int P>
int RunAdj<P>::p2m(const float* pos4, int num_nodes, int num_internal, const int* ranges, const float* centers,
                   const float* mbar, const float* cbar4, float* xm4, cudaStream_t st) {
  const int L = num_nodes - num_internal;
  if (L <= 0) return JB_OK;
  k_adj_p2m<P><<<blocks_for(L, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, st>>>(
      reinterpret_cast<const float4*>(pos4), num_nodes, num_internal, reinterpret_cast<const int2*>(ranges),
      reinterpret_cast<const float4*>(centers), mbar, reinterpret_cast<const float4*>(cbar4),
      reinterpret_cast<float4*>(xm4));
  return launch_status();
}

}  // namespace jb
