// Far-field stages of the evaluator, FP32 SIMT: moment gather, P2M, L2P (fused with the near/far combine and the unsort to user order).
//
// Layouts (K = states of the call):
//   mom [ns][K]            float4 (mx, my, mz, 0), Morton-sorted, scaled by 1/scale^3
//   M, L [node][coef][K]   node = (8^level - 1)/7 + morton(ix, iy, iz)
//   near [nt][K]           float4 (phi, Hx, Hy, Hz), Morton-sorted
// Each expansion coefficient is written by exactly one thread (no atomics),
// so results are deterministic run to run.
#include <cuda_runtime.h>

#include "far_kernels.hpp"
#include "kernels.cuh"

namespace cdfmm_b200 {

namespace {

// Calls f(nu, kn) for a tile of nu points and kn states, both <= 32: as
// compile-time constants for the full tiles (32 points, 32 or 16 states),
// whose index arithmetic is then shifts and whose loops unroll.  (With
// divisions at run time they ran at half of HBM.  N = 1,048,576, K = 64:
// gather 607 -> 498 us, L2P and unsort 1793 -> 1660 us;
// tiles of 8 states measured the same either way.)
template <class F> __device__ __forceinline__ void with_tile(int nu, int kn, F f) {
  using std::integral_constant;
  if (nu == 32 && kn == 32)
    f(integral_constant<int, 32>{}, integral_constant<int, 32>{});
  else if (nu == 32 && kn == 16)
    f(integral_constant<int, 32>{}, integral_constant<int, 16>{});
  else
    f(nu, kn);
}

// ---------------------------------------------------------------------------
// moments: user order [K][ns][3] (f32 / f64) -> sorted [ns][K] float4 / scale^3
// (upstream src/far_field.cpp:248-275, src/cuda_fmm.cu:56-64).  A CTA takes
// 32 consecutive user indices and 32 states at a time through a shared tile:
// the reads are contiguous runs of each state's user array, the writes
// contiguous runs of each sorted row (inv = user -> sorted index).
template <typename T>
__global__ void __launch_bounds__(256) gather_moments_kernel(const T *__restrict__ user, const int *__restrict__ inv,
                                                             int ns, int K, double inv_scale, float inv_scale3_f,
                                                             bool paired, float4 *__restrict__ mom, int k0,
                                                             int krow) {
  __shared__ float tile[32][32 * 3 + 1]; // [user][state * 3 + component]
  const int u0 = blockIdx.x * 32;
  for (int kc = 0; kc < K; kc += 32)
    with_tile(min(32, ns - u0), min(32, K - kc), [&](auto nu, auto kn) {
#pragma unroll 4
      for (int e = threadIdx.x; e < kn * nu * 3; e += 256) {
        const int k = e / (nu * 3);
        const int r = e - k * (nu * 3);
        const int t = r / 3;
        const T v = user[(static_cast<long long>(kc + k) * ns + u0) * 3 + r];
        float f;
        if constexpr (sizeof(T) == 8)
          f = static_cast<float>(static_cast<double>(v) * inv_scale * inv_scale * inv_scale); // m / s / s / s in FP64
        else
          f = static_cast<float>(v) * inv_scale3_f;
        tile[t][3 * k + (r - 3 * t)] = f;
      }
      __syncthreads();
      if (paired) {
        // state pairs (k, k+1) as (x_k, x_k1, y_k, y_k1), (z_k, z_k1, 0, 0); a
        // missing partner (K odd) is zero
        const int row = krow;
#pragma unroll 2
        for (int e = threadIdx.x; e < nu * ((kn + 1) / 2); e += 256) {
          const int t = e / ((kn + 1) / 2);
          const int k = 2 * (e - t * ((kn + 1) / 2));
          const bool b = k + 1 < kn;
          float4 *dst = mom + static_cast<long long>(inv[u0 + t]) * row + k0 + kc + k;
          dst[0] = make_float4(tile[t][3 * k], b ? tile[t][3 * k + 3] : 0.0F, tile[t][3 * k + 1],
                               b ? tile[t][3 * k + 4] : 0.0F);
          dst[1] = make_float4(tile[t][3 * k + 2], b ? tile[t][3 * k + 5] : 0.0F, 0.0F, 0.0F);
        }
      } else {
#pragma unroll 2
        for (int e = threadIdx.x; e < nu * kn; e += 256) {
          const int t = e / kn;
          const int k = e - t * kn;
          mom[static_cast<long long>(inv[u0 + t]) * krow + k0 + kc + k] =
              make_float4(tile[t][3 * k], tile[t][3 * k + 1], tile[t][3 * k + 2], 0.0F);
        }
      }
      __syncthreads();
    });
}

// Sorted results res[nt][K] (phi, Hx, Hy, Hz) -> user order: field[K][nt][3]
// and potential[K][nt] (layout 0) or field[K][nt][4] (layout 1).  A CTA takes
// 32 consecutive user indices and 32 states through a shared tile: the reads
// are contiguous runs of each sorted row (inv = user -> sorted), the writes
// contiguous runs of each state's user array.
__global__ void __launch_bounds__(256) unsort_results_kernel(const float4 *__restrict__ res, const int *__restrict__ inv,
                                                             int nt, int K, unsigned output, int layout,
                                                             float *__restrict__ field, float *__restrict__ potential,
                                                             int k_begin, int k_end) {
  __shared__ float4 tile[32][33];
  const int u0 = blockIdx.x * 32;
  const bool want_phi = (output & 1u) != 0u;
  const bool want_h = (output & 2u) != 0u;
  for (int kc = k_begin; kc < k_end; kc += 32)
    with_tile(min(32, nt - u0), min(32, k_end - kc), [&](auto nu, auto kn) {
#pragma unroll 4
      for (int e = threadIdx.x; e < nu * kn; e += 256) {
        const int t = e / kn;
        const int k = e - t * kn;
        tile[t][k] = res[static_cast<long long>(inv[u0 + t]) * K + kc + k];
      }
      __syncthreads();
      if (layout == 1) {
#pragma unroll 4
        for (int e = threadIdx.x; e < kn * nu; e += 256) {
          const int k = e / nu;
          const int t = e - k * nu;
          reinterpret_cast<float4 *>(field)[static_cast<long long>(kc + k) * nt + u0 + t] = tile[t][k];
        }
      } else {
        if (want_h) {
#pragma unroll 4
          for (int e = threadIdx.x; e < kn * nu * 3; e += 256) {
            const int k = e / (nu * 3);
            const int r = e - k * (nu * 3);
            const int t = r / 3;
            const int c = r - 3 * t;
            field[(static_cast<long long>(kc + k) * nt + u0) * 3 + r] =
                reinterpret_cast<const float *>(&tile[t][k])[1 + c];
          }
        }
        if (want_phi && potential != nullptr) {
#pragma unroll 4
          for (int e = threadIdx.x; e < kn * nu; e += 256) {
            const int k = e / nu;
            const int t = e - k * nu;
            potential[static_cast<long long>(kc + k) * nt + u0 + t] = tile[t][k].x;
          }
        }
      }
      __syncthreads();
    });
}

// Position gradient of L = sum_k w_k . H_k (reverse mode; no counterpart in
// the reference), far part.  H_k = -grad phi_k, so dL/dx_j = -sum_k sum_c
// w_kc d_c d_j phi_k, and from phi = sum_b L_b dx^b/b! (the exact derivative
// of the evaluated polynomial) the Hessian at the target is
//   S_cj[k] = sum_{|mu| <= p-2} x^mu/mu! L_{mu + e_c + e_j}[k]   (6 unique c <= j),
// so g_j -= sum_k sum_c w_kc S_cj[k].  Per leaf
// the leaf's locals (a state block) and the monomials of 32 targets are
// staged in shared memory; a thread owns a register tile of 2 targets x 4
// states x 6 Hessian components (a small GEMM over the monomials), contracts
// it with the weights and adds its 2 targets' partial gradients into shared
// memory; then the list-1 part (gpart, one partial per state group) is added
// and the result written in user order.
constexpr int kL2pTargets = 32;
constexpr int kL2pGradThreads = 128;

__global__ void __launch_bounds__(kL2pGradThreads) l2p_grad_kernel(
    const float *__restrict__ L, const float4 *__restrict__ tgt_rel, const int *__restrict__ tgt_off,
    const int *__restrict__ tgt_perm, const float4 *__restrict__ W, const float4 *__restrict__ gpart, int G, int n,
    int p, int K, int leaf_node_base, float inv_scale, float *__restrict__ out, int Kb) {
  extern __shared__ float4 l2pg_smem[];
  const int Kbp = (Kb + 3) & ~3;
  const int q = max(p - 2, 0);
  const int nm2 = p >= 2 ? basis_size_d(p - 2) : 0;
  float *sL = reinterpret_cast<float *>(l2pg_smem);               // [n][Kcp]
  float *mono = sL + n * Kbp;                                      // [nm2][kL2pTargets]
  float *gsum = mono + nm2 * kL2pTargets;                          // [kL2pTargets][3]
  short *sidx = reinterpret_cast<short *>(gsum + 3 * kL2pTargets); // [nm2][6] ranks of mu + e_c + e_j
  const int tid = threadIdx.x;
  const int leaf = blockIdx.x;
  const int t0 = tgt_off[leaf];
  const int t1 = tgt_off[leaf + 1];
  if (t0 == t1) return;
  for (int m = tid; m < nm2; m += kL2pGradThreads) {
    int a = 0, b = 0, c = 0;
    for (int aa = 0; aa <= q; ++aa)
      for (int bb = 0; aa + bb <= q; ++bb)
        for (int cc = 0; aa + bb + cc <= q; ++cc)
          if (rank3(aa, bb, cc) == m) {
            a = aa;
            b = bb;
            c = cc;
          }
    sidx[6 * m + 0] = static_cast<short>(rank3(a + 2, b, c));         // xx
    sidx[6 * m + 1] = static_cast<short>(rank3(a + 1, b + 1, c));     // xy
    sidx[6 * m + 2] = static_cast<short>(rank3(a + 1, b, c + 1));     // xz
    sidx[6 * m + 3] = static_cast<short>(rank3(a, b + 2, c));         // yy
    sidx[6 * m + 4] = static_cast<short>(rank3(a, b + 1, c + 1));     // yz
    sidx[6 * m + 5] = static_cast<short>(rank3(a, b, c + 2));         // zz
  }
  const float *src = L + static_cast<long long>(leaf_node_base + leaf) * n * K;
  for (int tc = t0; tc < t1; tc += kL2pTargets) {
    const int tn = min(kL2pTargets, t1 - tc);
    __syncthreads(); // previous chunk's gsum and mono reads are done
    if (tid < 3 * kL2pTargets) gsum[tid] = 0.0F;
    if (nm2 > 0) {
      const int t = tid & (kL2pTargets - 1);
      const float4 d = t < tn ? tgt_rel[tc + t] : make_float4(0.0F, 0.0F, 0.0F, 0.0F);
      monomials_part(d.x, d.y, d.z, q, mono + t, kL2pTargets, tid / kL2pTargets, t >= tn);
    }
    for (int kblk = 0; kblk < K; kblk += Kb) {
      const int Kc = min(Kb, K - kblk);
      const int Kcp = (Kc + 3) & ~3;
      const int Kq = Kcp >> 2;
      __syncthreads(); // previous block's sL reads are done
      if ((K & 3) == 0 && (kblk & 3) == 0 && (Kc & 3) == 0) {
        const int nq = Kcp >> 2;
        for (int e = tid; e < n * nq; e += kL2pGradThreads) {
          const int b = e / nq;
          cp_async16(reinterpret_cast<float4 *>(sL) + e, src + static_cast<long long>(b) * K + kblk + 4 * (e - b * nq));
        }
        cp_async_commit();
        cp_async_wait<0>();
      } else {
        for (int e = tid; e < n * Kcp; e += kL2pGradThreads) {
          const int b = e / Kcp;
          const int k = e - b * Kcp;
          sL[e] = k < Kc ? src[static_cast<long long>(b) * K + kblk + k] : 0.0F;
        }
      }
      __syncthreads();
      if (nm2 == 0) continue;
      const int tiles = ((tn + 1) >> 1) * Kq;
      for (int tile = tid; tile < tiles; tile += kL2pGradThreads) {
        const int tp = tile / Kq;
        const int kq = tile - tp * Kq;
        float hs[2][4][6];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v)
#pragma unroll
            for (int h = 0; h < 6; ++h) hs[u][v][h] = 0.0F;
        const float *mq = mono + 2 * tp;
        const float *lq = sL + 4 * kq;
        for (int m = 0; m < nm2; ++m) {
          const float2 mo = *reinterpret_cast<const float2 *>(mq + m * kL2pTargets);
#pragma unroll
          for (int h = 0; h < 6; ++h) {
            const float4 l = *reinterpret_cast<const float4 *>(lq + sidx[6 * m + h] * Kcp);
            hs[0][0][h] = fmaf(mo.x, l.x, hs[0][0][h]);
            hs[0][1][h] = fmaf(mo.x, l.y, hs[0][1][h]);
            hs[0][2][h] = fmaf(mo.x, l.z, hs[0][2][h]);
            hs[0][3][h] = fmaf(mo.x, l.w, hs[0][3][h]);
            hs[1][0][h] = fmaf(mo.y, l.x, hs[1][0][h]);
            hs[1][1][h] = fmaf(mo.y, l.y, hs[1][1][h]);
            hs[1][2][h] = fmaf(mo.y, l.z, hs[1][2][h]);
            hs[1][3][h] = fmaf(mo.y, l.w, hs[1][3][h]);
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int t = 2 * tp + u;
          float g0 = 0.0F, g1 = 0.0F, g2 = 0.0F;
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const int kl = 4 * kq + v;
            const float4 w = (t < tn && kl < Kc) ? W[static_cast<long long>(tc + t) * K + kblk + kl]
                                                 : make_float4(0.0F, 0.0F, 0.0F, 0.0F);
            g0 = fmaf(w.x, hs[u][v][0], fmaf(w.y, hs[u][v][1], fmaf(w.z, hs[u][v][2], g0)));
            g1 = fmaf(w.x, hs[u][v][1], fmaf(w.y, hs[u][v][3], fmaf(w.z, hs[u][v][4], g1)));
            g2 = fmaf(w.x, hs[u][v][2], fmaf(w.y, hs[u][v][4], fmaf(w.z, hs[u][v][5], g2)));
          }
          if (t < tn) {
            atomicAdd(&gsum[3 * t], -g0);
            atomicAdd(&gsum[3 * t + 1], -g1);
            atomicAdd(&gsum[3 * t + 2], -g2);
          }
        }
      }
    }
    __syncthreads();
    for (int t = tid; t < tn; t += kL2pGradThreads) {
      const int i = tc + t;
      float g0 = gsum[3 * t], g1 = gsum[3 * t + 1], g2 = gsum[3 * t + 2];
      for (int gi = 0; gi < G; ++gi) {
        const float4 v = gpart[static_cast<long long>(i) * G + gi];
        g0 += v.x;
        g1 += v.y;
        g2 += v.z;
      }
      const int u = tgt_perm[i];
      out[3 * static_cast<long long>(u)] = g0 * inv_scale;
      out[3 * static_cast<long long>(u) + 1] = g1 * inv_scale;
      out[3 * static_cast<long long>(u) + 2] = g2 * inv_scale;
    }
  }
}

// The same for fewer than 4 states (plain rows): a thread per (state, user
// point).  (The tiles above leave 160 of 256 threads idle at one state: N = 1M
// 52 us.)
template <typename T>
__global__ void __launch_bounds__(256) gather_few_kernel(const T *__restrict__ user, const int *__restrict__ inv, int ns,
                                                         int K, double inv_scale, float inv_scale3_f,
                                                         float4 *__restrict__ mom, int k0, int krow) {
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= static_cast<long long>(ns) * K) return;
  const int k = static_cast<int>(e / ns), u = static_cast<int>(e - static_cast<long long>(k) * ns);
  const T *v = user + 3 * e;
  float m[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if constexpr (sizeof(T) == 8)
      m[c] = static_cast<float>(static_cast<double>(v[c]) * inv_scale * inv_scale * inv_scale);
    else
      m[c] = static_cast<float>(v[c]) * inv_scale3_f;
  }
  mom[static_cast<long long>(inv[u]) * krow + k0 + k] = make_float4(m[0], m[1], m[2], 0.0F);
}

} // namespace

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------

void launch_gather_moments(const void *user, int dtype, const int *inv, int ns, int K,
                           double scale, float4 *mom, cudaStream_t s, bool paired, int k0, int k_total) {
  if (ns == 0) return;
  if (k_total < 0) k_total = K;
  const int krow = paired ? (k_total + 1) & ~1 : k_total;
  const int blocks = (ns + 31) / 32;
  const double invs = 1.0 / scale;
  const float inv3f = static_cast<float>(invs * invs * invs);
  if (K < 4 && !paired) {
    const unsigned few = static_cast<unsigned>((static_cast<long long>(ns) * K + 255) / 256);
    if (dtype == 1)
      gather_few_kernel<double><<<few, 256, 0, s>>>(static_cast<const double *>(user), inv, ns, K, invs, inv3f, mom, k0,
                                                    krow);
    else
      gather_few_kernel<float><<<few, 256, 0, s>>>(static_cast<const float *>(user), inv, ns, K, invs, inv3f, mom, k0,
                                                   krow);
    return;
  }
  if (dtype == 1)
    gather_moments_kernel<double><<<blocks, 256, 0, s>>>(static_cast<const double *>(user), inv, ns, K, invs, inv3f,
                                                         paired, mom, k0, krow);
  else
    gather_moments_kernel<float><<<blocks, 256, 0, s>>>(static_cast<const float *>(user), inv, ns, K, invs, inv3f,
                                                        paired, mom, k0, krow);
}

void launch_unsort(const float4 *res, const int *tgt_inv, int nt, int K, unsigned output, int layout, float *field,
                   float *potential, cudaStream_t s, int k_begin, int k_end) {
  if (nt == 0 || k_end <= k_begin) return;
  unsort_results_kernel<<<(nt + 31) / 32, 256, 0, s>>>(res, tgt_inv, nt, K, output, layout, field, potential, k_begin,
                                                       k_end);
}

void launch_l2p_grad(const float *L, const float4 *tgt_rel, const int *tgt_off, const int *tgt_perm,
                     const float4 *W, const float4 *gpart, int G, int n, int p, int K, int nt, int depth,
                     float inv_scale, float *out, cudaStream_t s) {
  if (nt == 0) return;
  const int leaves = 1 << (3 * depth);
  const int nm2 = p >= 2 ? basis_size_d(p - 2) : 0;
  auto smem_of = [&](int Kb) {
    return sizeof(float) * (static_cast<size_t>(n) * ((Kb + 3) & ~3) + static_cast<size_t>(nm2) * kL2pTargets +
                            3 * kL2pTargets) +
           sizeof(short) * 6 * static_cast<size_t>(nm2) + 16;
  };
  int Kb = std::min(K, 64);
  while (Kb > 4 && smem_of(Kb) > 48 * 1024) Kb = (Kb + 1) / 2;
  l2p_grad_kernel<<<leaves, kL2pGradThreads, smem_of(Kb), s>>>(L, tgt_rel, tgt_off, tgt_perm, W, gpart, G, n, p, K,
                                                              level_offset_d(depth), inv_scale, out, Kb);
}

void configure_far_kernels(size_t max_smem) {
  allow_dynamic_smem(l2p_grad_kernel, max_smem);
}

} // namespace cdfmm_b200
