// krylov.cu -- Arnoldi / least-squares kernels of restarted GMRES(m) and
// FGMRES (src/core/gmres.cpp:34-160, src/core/fgmres.cpp:28-144; replaces the
// host-driven cuBLAS loop of src/gpu/gmres_gpu.cu:10-138).
//
// Basis storage: raw_k (k <= m) are the columns of a (m+1) x ldv array; the
// orthonormal vector is v_k = vscale[k] * raw_k, so a new vector never needs
// a separate normalisation pass.
//
// One Arnoldi step orthogonalises w = raw_{j+1} against raw_0..raw_j by
// classical Gram-Schmidt applied twice (CGS2), in three streaming passes:
//   A  h1 = V^T w                          (dot products, one pass)
//   B  w' = w - V h1 ; h2 = V^T w'          (update and second dots, one pass)
//   C  w'' = w' - V h2 ; ||w''||           (update and norm, one pass)
// Every pass reduces per block, per cluster, and in the last cluster to finish
// (cluster_reduce); after the last pass that block also writes the Hessenberg
// column, applies the Givens rotations (the reference's, src/core/
// gmres.cpp:9-30) and tests convergence, so no value travels to the host
// inside a cycle.  These ends of a pass are chains of FP64 operations on one
// SM (~75 cycles each when dependent, ~400-560 for a root or a quotient), so
// they are arranged for depth: matrix-vector products take a lane per row and
// four sums per lane, the earlier rotations run as a parallel prefix.
#include <algorithm>

#include "dev_common.cuh"
#include "kernels.h"

namespace sg {

namespace {

constexpr int KT = 256;    // threads of the Krylov kernels
constexpr int BS_T = 256;  // threads of the back substitution (loads; one warp solves)

// State the end of an Arnoldi step reads, brought to shared memory in one round
// of loads: the column h(0..j),
// the earlier rotations, g(j..j+1) and the stopping-test scalars.
struct FinalizeIn {
    double hc[SG_MMAX + 2], csv[SG_MMAX], snv[SG_MMAX], gv[2];
    double tol, bnorm, est_scale;
    int tol_kind, hist_len, total_iter;
};

// global -> shared without a register in between: the issuing warp goes on
template <class T>
__device__ __forceinline__ void cp_async(T* dst, const T* src) {
    static_assert(sizeof(T) == 4 || sizeof(T) == 8, "cp.async sizes");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"((int)sizeof(T))
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// all threads of the block: starts to load everything but hc (the caller's
// column); the caller waits (cp_async_wait, then a barrier)
__device__ __forceinline__ void finalize_load(FinalizeIn& f, const SolveState* st, int j) {
    for (int i = threadIdx.x; i < j; i += blockDim.x) {
        cp_async(&f.csv[i], &st->cs[i]);
        cp_async(&f.snv[i], &st->sn[i]);
    }
    if (threadIdx.x == 0) {
        cp_async(&f.gv[0], &st->g[j]);
        cp_async(&f.gv[1], &st->g[j + 1]);
        cp_async(&f.tol, &st->tol);
        cp_async(&f.bnorm, &st->bnorm);
        cp_async(&f.est_scale, &st->est_scale);
        cp_async(&f.tol_kind, &st->tol_kind);
        cp_async(&f.hist_len, &st->hist_len);
        cp_async(&f.total_iter, &st->total_iter);
    }
}

// One warp: completes Arnoldi step j from a = rotate_column and ss =
// ||w''||^2: normalisation, the new rotation, residual estimate and stopping
// test.  Returns the new vector's scale 1/||w''|| when the cycle goes on, 0
// when it stops here (breakdown, convergence, last step); nrm = ||w''||.
__device__ double finalize_warp(SolveState* st, const FinalizeIn& f, int j, int m, double a,
                                double ss, double* hist, int hist_cap, double& nrm) {
    const int lane = threadIdx.x & 31;
    double* Hc = st->H + (size_t)j * (m + 1);
    nrm = sqrt(ss);
    if (!(nrm >= 1e-30)) {
        // breakdown (src/core/gmres.cpp:297-300): this column is used as is
        __syncwarp();
        for (int i = lane; i <= j + 1; i += 32) Hc[i] = i <= j ? f.hc[i] : nrm;
        if (lane == 0) {
            if (!isfinite(nrm)) {
                st->nonfinite = 1;
                st->done = 1;
            }
            st->breakdown = 1;
            st->kcount = j + 1;
            st->cycle_active = 0;
        }
        return 0.0;
    }
    const double vs = 1.0 / nrm;
    double c, sn;
    rot_compute(c, sn, a, nrm);
    const double g0 = f.gv[0], g1 = f.gv[1];
    const double gj = c * g0 - sn * g1, gn = sn * g0 + c * g1;
    const double res = fabs(gn);
    // the stopping tests: the reference's rule, or the estimated true residual
    // (which the restart verifies in FP64)
    const bool conv = f.tol_kind == SG_TOL_REF_ABS && res < f.tol;
    const bool bad = !isfinite(res);
    const bool stop = conv || bad || j + 1 >= m ||
                      (f.tol_kind == SG_TOL_TRUE_REL && res * f.est_scale <= 0.5 * f.tol * f.bnorm);
    if (lane == 0) {
        st->vscale[j + 1] = vs;
        Hc[j] = c * a - sn * nrm;
        Hc[j + 1] = sn * a + c * nrm;
        st->cs[j] = c;
        st->sn[j] = sn;
        st->g[j] = gj;
        st->g[j + 1] = gn;
        if (hist && f.hist_len < hist_cap) hist[f.hist_len] = res;
        st->hist_len = f.hist_len + 1;
        st->last_res = res;
        st->total_iter = f.total_iter + 1;
        st->kcount = j + 1;
        st->j = j + 1;
        if (conv) {
            st->converged = 1;
            st->done = 1;
        }
        if (bad) {
            st->nonfinite = 1;
            st->done = 1;
        }
        if (stop) st->cycle_active = 0;
    }
    return stop ? 0.0 : vs;
}

// Completes Arnoldi step j once ||w''||^2 is known (all threads of the last
// block; the column is hsum(0..j)).
__device__ void arnoldi_finalize(SolveState* st, int j, int m, double ss, double* hist,
                                 int hist_cap) {
    __shared__ FinalizeIn f;
    for (int i = threadIdx.x; i <= j; i += blockDim.x) cp_async(&f.hc[i], &st->hsum[i]);
    finalize_load(f, st, j);
    cp_async_wait();
    __syncthreads();
    if (threadIdx.x < 32) {
        double nrm;
        const double a = rotate_column(f.hc, f.csv, f.snv, st->H + (size_t)j * (m + 1), j);
        finalize_warp(st, f, j, m, a, ss, hist, hist_cap, nrm);
    }
}

template <class T>
struct Vec;
template <>
struct Vec<double> {
    static constexpr int N = 2;
    using V = double2;
};
template <>
struct Vec<float> {
    static constexpr int N = 4;
    using V = float4;
};

template <class T>
__device__ __forceinline__ void vload(const T* p, T (&o)[Vec<T>::N]);
template <>
__device__ __forceinline__ void vload<double>(const double* p, double (&o)[2]) {
    const double2 v = ld_stream(reinterpret_cast<const double2*>(p));
    o[0] = v.x; o[1] = v.y;
}
template <>
__device__ __forceinline__ void vload<float>(const float* p, float (&o)[4]) {
    const float4 v = ld_stream(reinterpret_cast<const float4*>(p));
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
template <class T>
__device__ __forceinline__ void vstore(T* p, const T (&o)[Vec<T>::N]);
template <>
__device__ __forceinline__ void vstore<double>(double* p, const double (&o)[2]) {
    *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
}
template <>
__device__ __forceinline__ void vstore<float>(float* p, const float (&o)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
}

// ---- pass A (and generic second dots): s_k = raw_{k0+k} . w for k < kc.
// A row tile is 32 lanes x one 16-byte vector of elements.  The kc <= 32
// vectors of a launch are spread over a group of nwg warps that share a tile
// (vector k is held by warp k % nwg of the group, so a thread keeps at most 4
// accumulators); the block's 8 / nwg groups walk different tiles, so a step
// with few vectors still keeps every warp loading.
constexpr int KW = KT / 32;  // warps per block
constexpr int KPW = 4;       // basis vectors per warp
constexpr int DOTS_PER_SM = 4, UPD_PER_SM = 3;  // resident blocks of the two passes

// warps per tile group (the kernels' NWG): the fewest that hold kc vectors at
// KPW per warp
int warps_per_tile(int kc) { return kc <= KPW ? 1 : (kc <= 2 * KPW ? 2 : (kc <= 4 * KPW ? 4 : 8)); }

// acc + a . b.  FP64: one multiply-add per element (the scarce resource).  FP32:
// the four products by themselves first, then one addition to the sum -- four
// at the sum's size double a dot's error (128^3: 2.0e-6 of a lane's terms, not
// 1.1e-6) and save nothing, as the loads bound the pass.
template <class TV>
__device__ __forceinline__ TV dotv(const TV (&a)[Vec<TV>::N], const TV (&b)[Vec<TV>::N], TV acc);
template <>
__device__ __forceinline__ double dotv<double>(const double (&a)[2], const double (&b)[2],
                                               double acc) {
    return fma(a[1], b[1], fma(a[0], b[0], acc));
}
template <>
__device__ __forceinline__ float dotv<float>(const float (&a)[4], const float (&b)[4], float acc) {
    float s = a[0] * b[0];
#pragma unroll
    for (int e = 1; e < 4; ++e) s = fmaf(a[e], b[e], s);
    return acc + s;
}

// the warp sums of four values at once: each of the first two exchanges halves
// the values a lane holds (6 additions a lane instead of 20); the sum of value
// (lane >> 3) is in every lane of that eighth
template <class TV>
__device__ __forceinline__ TV warp_sum4(const TV (&v)[KPW]) {
    static_assert(KPW == 4, "two halvings");
    const int lane = threadIdx.x & 31;
    const bool h1 = lane & 16, h2 = lane & 8;
    TV a = h1 ? v[2] : v[0], b = h1 ? v[3] : v[1];
    a += __shfl_xor_sync(0xffffffffu, h1 ? v[0] : v[2], 16);
    b += __shfl_xor_sync(0xffffffffu, h1 ? v[1] : v[3], 16);
    TV r = h2 ? b : a;
    r += __shfl_xor_sync(0xffffffffu, h2 ? a : b, 8);
    r += __shfl_xor_sync(0xffffffffu, r, 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    return r;
}

// per-warp accumulators -> block sums bs[k] (k < kc): the warp trees run in
// the basis precision, the groups' sums of vector k are added in FP64 in
// group order (fixed: deterministic)
template <class TV>
__device__ __forceinline__ void group_sums(const TV (&acc)[KPW], int kc, int nwg, double* bs) {
    __shared__ double red[KW][KPW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double v = (double)warp_sum4<TV>(acc);
    if ((lane & 7) == 0) red[warp][lane >> 3] = v;
    __syncthreads();
    if ((int)threadIdx.x < kc) {
        const int k = threadIdx.x, slot = k % nwg, q = k / nwg;
        double v = red[slot][q];
        for (int g = 1; g < KW / nwg; ++g) v += red[g * nwg + slot][q];
        bs[k] = v;
    }
    __syncthreads();
}

// barrier among the nwg >= 2 warps of tile group grp < 4 (named barrier
// 1 + grp; immediate ids keep the block's barrier count at five)
__device__ __forceinline__ void group_sync(int grp, int nwg) {
    const int cnt = nwg * 32;
    switch (grp) {
    case 0: asm volatile("bar.sync 1, %0;" ::"r"(cnt) : "memory"); break;
    case 1: asm volatile("bar.sync 2, %0;" ::"r"(cnt) : "memory"); break;
    case 2: asm volatile("bar.sync 3, %0;" ::"r"(cnt) : "memory"); break;
    default: asm volatile("bar.sync 4, %0;" ::"r"(cnt) : "memory"); break;
    }
}

// ---- lagged CGS2 (restart < SG_LAGM, FP32 or FP64 basis).
// Step j orthogonalises z = B (vscale_j raw_j), where the stored raw_j still
// lacks its second projection: v_j = T(j,j) raw_j - sum_{k<j} c_k v_k.  By
// linearity B v_j = z - V_j g with g = H(0..j, 0..j-1) c (the Arnoldi relation
// B v_k = V H(:,k)), so the projections of z give the Hessenberg column after
// subtracting g, and the orthogonalised vector is the same.  Two passes:
//   A  d = S^T z over the stored vectors; p = T^T d; hsum = p - g;
//      update coefficients on the stored vectors u = T p
//   B  w' = z - S u; r = S^T w'; ||w'||^2; then h2 = T^T r, the column is
//      hsum + h2, ||w''||^2 = ||w'||^2 - ||h2||^2 (Pythagoras), and w' is
//      stored as raw_{j+1} with its pending correction c = h2 / ||w''||.
// In exact arithmetic this is CGS2; the stored vectors are never rewritten.

// What the ends of the two passes read from the state.  The first block of
// every cluster starts to copy it when the kernel starts (cp.async, waited
// for at the end: none of it changes during the kernel), so the block that
// gets there last finds it in shared memory.  T and H keep their zeros below
// the (sub)diagonal, so whole rows are summed.
struct LagIn {
    double T[SG_LAGM][SG_LAGM + 1];   // T(l, i) at [i][l]
    double Tt[SG_LAGM][SG_LAGM + 1];  // T(l, i) at [l][i]
    double H[SG_LAGM][SG_LAGM + 1];   // pass A: the unrotated Hessenberg, H(i, k) at [k][i]
    double c[SG_LAGM];                // pass A: the pending correction
    FinalizeIn f;                     // pass B
};
__device__ __forceinline__ void lag_prefetch(LagIn& in, const SolveState* st, int j, bool pass_b) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = warp; i <= j; i += KT / 32) {
        if (lane <= j) {
            cp_async(&in.T[i][lane], &st->lagT[lane + i * SG_LAGM]);
            cp_async(&in.Tt[lane][i], &st->lagT[lane + i * SG_LAGM]);
        }
        if (!pass_b && i < j && lane <= j) cp_async(&in.H[i][lane], &st->lagH[lane + i * SG_LAGM]);
    }
    if (pass_b) {
        for (int i = threadIdx.x; i <= j; i += KT) cp_async(&in.f.hc[i], &st->hsum[i]);
        finalize_load(in.f, st, j);
    } else if (warp == 0 && lane < j) {
        cp_async(&in.c[lane], &st->lagc[lane]);
    }
}

// pass A's end (all threads of the block that ends the pass; d = tot[0..j]): p = T^T d,
// hsum = p - g with g = H c, update coefficients u = T p
__device__ void lagged_pass_a(SolveState* st, int j, const double* d, const LagIn& in) {
    __shared__ double p_s[SG_LAGM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double g = 0.0;
    if (warp == 0) {
        const double p = lag_rows(in.Tt, d, j + 1);
        if (lane <= j) p_s[lane] = p;
    } else if (warp == 1) {
        if (lane <= j) g = lag_rows(in.H, in.c, j);
    }
    __syncthreads();
    if (lane > j) return;
    if (warp == 0) st->cfu[lane] = lag_rows(in.T, p_s, j + 1);
    if (warp == 1) st->hsum[lane] = p_s[lane] - g;
}

// pass B's end (all threads of that block; r = tot[0..j], ss =
// ||w'||^2): h2 = T^T r, the column hsum + h2, its rotations (warp 0), the new
// norm (warp 2), the step's end (warp 0), the new vector's pending correction
// and T column (warp 1).
//
// A remainder below a tenth of w' (Kahan's and Parlett's "twice is enough", B. N.
// Parlett, "The symmetric eigenvalue problem", 1980, 6.9) or below four
// roundings of w is rounding itself: w lies in the span of the vectors before.
// Left-preconditioned GMRES has converged then, and so has FGMRES where the
// column's diagonal stands above the noise (w' is all of it).  Else (directions
// that repeat, a preconditioner of low rank) the column is noise too, and to
// carry on multiplies it by the correction's size at every step -- residuals of
// 1e9 to 1e50 where three passes stay at 1 -- so the cycle ends without it.
__device__ void lagged_pass_b(SolveState* st, int j, int m, const double* r, double ss,
                              double* hist, int hist_cap, LagIn& in, bool flexible, double eps) {
    __shared__ double h2_s[SG_LAGM];
    __shared__ double s_vs, s_n2;
    __shared__ int s_noise;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double a = 0.0, tc = 0.0;
    if (warp == 0) {
        const double h2 = lag_rows(in.Tt, r, j + 1);
        if (lane <= j) {
            h2_s[lane] = h2;
            const double hs = in.f.hc[lane] + h2;  // the Hessenberg column
            in.f.hc[lane] = hs;
            st->hsum[lane] = hs;
            st->lagH[lane + j * SG_LAGM] = hs;
        }
    }
    __syncthreads();
    if (warp == 0) {
        a = rotate_column(in.f.hc, in.f.csv, in.f.snv, st->H + (size_t)j * (m + 1), j);
    } else if (warp == 1) {
        if (lane <= j) tc = lag_rows(in.T, h2_s, j + 1);
    } else if (warp == 2) {
        const double h2 = lane <= j ? h2_s[lane] : 0.0;
        double nrm2 = ss - warp_sum(h2 * h2);
        if (!(nrm2 > 0.0)) nrm2 = isfinite(nrm2) ? 0.0 : nrm2;
        if (lane == 0) s_n2 = nrm2;
        if (flexible) {
            const double h = lane <= j ? in.f.hc[lane] : 0.0;
            const double col = warp_sum(h * h);
            if (lane == 0) s_noise = nrm2 < 0.01 * ss || nrm2 < 16.0 * eps * eps * col;
        }
    }
    __syncthreads();
    if (warp == 0) {
        double nrm = 0.0, vs = 0.0;
        if (flexible && s_noise && a * a <= 1e4 * ss) {
            if (lane == 0) {
                st->kcount = j;
                st->cycle_active = 0;
            }
        } else {
            vs = finalize_warp(st, in.f, j, m, a, s_n2, hist, hist_cap, nrm);
        }
        if (lane == 0) {
            st->lagH[j + 1 + j * SG_LAGM] = nrm;
            s_vs = j + 1 < SG_LAGM ? vs : 0.0;
        }
    }
    __syncthreads();
    const double vs = s_vs;
    if (vs == 0.0 || warp != 1) return;
    // T(:, j+1) = T(j+1,j+1) e_{j+1} - T(:, 0..j) c with c = h2 vs
    if (lane <= j) {
        st->lagc[lane] = h2_s[lane] * vs;
        st->lagT[lane + (j + 1) * SG_LAGM] = -tc * vs;
    } else if (lane == j + 1) {
        st->lagT[lane + (j + 1) * SG_LAGM] = vs;
    }
}

template <class TV, int NWG>
__global__ void __launch_bounds__(KT, DOTS_PER_SM)
k_dots(const TV* __restrict__ raw, size_t ldv, int n, int k0, int kc, const TV* __restrict__ w,
       SolveState* st, int second, int lagged, double* partials, unsigned* counter) {
    if (!st->cycle_active) return;
    constexpr int VN = Vec<TV>::N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int nwg = NWG, ngrp = KW / NWG;
    const int grp = warp / nwg, slot = warp % nwg;
    __shared__ LagIn lag_in;
    if (lagged && cluster_rank() == 0) lag_prefetch(lag_in, st, kc - 1, false);
    TV acc[KPW];
#pragma unroll
    for (int q = 0; q < KPW; ++q) acc[q] = (TV)0;
    const int nvec = n / VN;
    const int stride = gridDim.x * ngrp * 32;
    // two tiles per round: all their loads are in flight before the first
    // product (a step with few vectors has only a few rounds per thread, each
    // a full memory latency); the tiles are still added in ascending order
    int u = (blockIdx.x * ngrp + grp) * 32 + lane;
    for (; u + stride < nvec; u += 2 * stride) {
        TV w0[VN], w1[VN], v0[KPW][VN], v1[KPW][VN];
        vload<TV>(w + (size_t)u * VN, w0);
        vload<TV>(w + (size_t)(u + stride) * VN, w1);
#pragma unroll
        for (int q = 0; q < KPW; ++q) {
            const int k = slot + nwg * q;
            if (k < kc) {
                vload<TV>(raw + (size_t)(k0 + k) * ldv + (size_t)u * VN, v0[q]);
                vload<TV>(raw + (size_t)(k0 + k) * ldv + (size_t)(u + stride) * VN, v1[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < KPW; ++q) {
            const int k = slot + nwg * q;
            if (k < kc) {
                acc[q] = dotv<TV>(v0[q], w0, acc[q]);
                acc[q] = dotv<TV>(v1[q], w1, acc[q]);
            }
        }
    }
    if (u < nvec) {
        TV wv[VN];
        vload<TV>(w + (size_t)u * VN, wv);
#pragma unroll
        for (int q = 0; q < KPW; ++q) {
            const int k = slot + nwg * q;
            if (k < kc) {
                TV vv[VN];
                vload<TV>(raw + (size_t)(k0 + k) * ldv + (size_t)u * VN, vv);
                acc[q] = dotv<TV>(vv, wv, acc[q]);
            }
        }
    }
    if (blockIdx.x == 0 && grp == 0) {  // elements past the last full vector
        const int i = nvec * VN + lane;
        if (lane < n - nvec * VN) {
#pragma unroll
            for (int q = 0; q < KPW; ++q) {
                const int k = slot + nwg * q;
                if (k < kc) acc[q] += raw[(size_t)(k0 + k) * ldv + i] * w[i];
            }
        }
    }
    __shared__ double bs[KW * KPW], tot[KW * KPW];
    group_sums<TV>(acc, kc, nwg, bs);
    if (lagged) cp_async_wait();
    if (!cluster_reduce(partials, counter, bs, kc, tot)) return;
    if (lagged) {
        lagged_pass_a(st, kc - 1, tot, lag_in);
        return;
    }
    for (int k = threadIdx.x; k < kc; k += blockDim.x) {
        const double h = st->vscale[k0 + k] * tot[k];
        st->h[k0 + k] = h;
        st->hsum[k0 + k] = second ? st->hsum[k0 + k] + h : h;
    }
}

// ---- pass B fused (nk <= 32): w' = w - sum_k c_k raw_k ; s2_k = raw_k . w'.
// Each warp of a tile group forms the update of its own vectors for the
// tile.  A one-warp group holds every vector: w' = w - share directly.  In a
// larger group the shares meet in shared memory, the group's threads each
// form w' = w - (sum of the shares) for some elements of the
// tile (and store them), and every warp dots w' with the vector values it
// still holds.
template <class TV, int NWG>
__global__ void __launch_bounds__(KT, UPD_PER_SM)
k_upd_dots(const TV* __restrict__ raw, size_t ldv, int n, int nk, TV* __restrict__ w,
           SolveState* st, double* partials, unsigned* counter, int lagged, int m,
           double* hist, int hist_cap) {
    if (!st->cycle_active) return;
    constexpr int VN = Vec<TV>::N;
    constexpr int TE = 32 * VN;  // elements of a tile
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int nwg = NWG, ngrp = KW / NWG;
    const int grp = warp / nwg, slot = warp % nwg;
    constexpr int gsz = nwg * 32;  // threads of the group
    const int gt = slot * 32 + lane;
    __shared__ TV cf[KW * KPW];
    __shared__ TV upd[KW][TE];
    __shared__ TV wsh[KW / 2][TE];
    __shared__ LagIn lag_in;
    TV ss = (TV)0;  // ||w'||^2 (lagged): slot 0 of each group counts its elements
    TV acc[KPW];
#pragma unroll
    for (int q = 0; q < KPW; ++q) acc[q] = (TV)0;
    const int nvec = n / VN;
    const int ntiles = (nvec + 31) / 32;
    const int nfull = nvec * VN;  // elements covered by whole vectors
    // registers of the current tile and of the next one (loaded ahead): the
    // warp's vector values, and the w elements this thread turns into w'
    // (its lanes' elements in a one-warp group; else elements gt + r * gsz)
    TV vv[KPW][VN], nv[KPW][VN], we[VN], nwe[VN];
    // tiles are walked in reverse: pass A (k_dots) has just streamed the
    // basis in ascending order, so its last tiles are still in L2
    auto load_tile = [&](int tile_l, TV (&v)[KPW][VN], TV (&wl)[VN]) {
        const int tile = ntiles - 1 - tile_l;
        const int u = tile * 32 + lane;
        const bool ok = u < nvec;
#pragma unroll
        for (int q = 0; q < KPW; ++q) {
            const int k = slot + nwg * q;
            if (k < nk && ok) {
                vload<TV>(raw + (size_t)k * ldv + (size_t)u * VN, v[q]);
            } else {
#pragma unroll
                for (int e = 0; e < VN; ++e) v[q][e] = (TV)0;
            }
        }
        if (nwg == 1) {
            if (ok) {
                vload<TV>(w + (size_t)u * VN, wl);
            } else {
#pragma unroll
                for (int e = 0; e < VN; ++e) wl[e] = (TV)0;
            }
        } else {
#pragma unroll
            for (int r = 0; r < VN; ++r) {
                const int t = gt + r * gsz, i = tile * TE + t;
                wl[r] = (t < TE && i < nfull) ? w[i] : (TV)0;
            }
        }
    };
    const int gstride = gridDim.x * ngrp;
    int tile = blockIdx.x * ngrp + grp;
    // the first tile's loads, the coefficients' and the end's all in flight at once
    if (tile < ntiles) load_tile(tile, vv, we);
    if (lagged && cluster_rank() == 0) lag_prefetch(lag_in, st, nk - 1, true);
    for (int k = threadIdx.x; k < nk; k += blockDim.x)
        cf[k] = lagged ? (TV)st->cfu[k] : (TV)(st->h[k] * st->vscale[k]);
    __syncthreads();
    for (; tile < ntiles; tile += gstride) {
        const int next = tile + gstride;
        if (next < ntiles) load_tile(next, nv, nwe);
        // this warp's share of the update for its lanes' elements
        TV part[VN];
#pragma unroll
        for (int e = 0; e < VN; ++e) part[e] = (TV)0;
#pragma unroll
        for (int q = 0; q < KPW; ++q) {
            const int k = slot + nwg * q;
            if (k < nk) {
#pragma unroll
                for (int e = 0; e < VN; ++e) part[e] += cf[k] * vv[q][e];
            }
        }
        TV wn[VN];
        const int ptile = ntiles - 1 - tile;  // the physical tile
        if (nwg == 1) {
#pragma unroll
            for (int e = 0; e < VN; ++e) wn[e] = we[e] - ((TV)0 + part[e]);
            const int u = ptile * 32 + lane;
            if (u < nvec) vstore<TV>(w + (size_t)u * VN, wn);
#pragma unroll
            for (int e = 0; e < VN; ++e) ss += wn[e] * wn[e];
        } else {
#pragma unroll
            for (int e = 0; e < VN; ++e) upd[warp][lane * VN + e] = part[e];
            group_sync(grp, nwg);
            // w' = w - (sum of the shares), once per element
#pragma unroll
            for (int r = 0; r < VN; ++r) {
                const int t = gt + r * gsz;
                if (t < TE) {
                    TV sh[nwg];  // added pairwise: three deep for eight warps
#pragma unroll
                    for (int g = 0; g < nwg; ++g) sh[g] = upd[grp * nwg + g][t];
#pragma unroll
                    for (int o = 1; o < nwg; o *= 2)
#pragma unroll
                        for (int g = 0; g < nwg; g += 2 * o) sh[g] += sh[g + o];
                    const TV x = we[r] - sh[0];
                    wsh[grp][t] = x;
                    const int i = ptile * TE + t;
                    if (i < nfull) w[i] = x;
                }
            }
            group_sync(grp, nwg);
#pragma unroll
            for (int e = 0; e < VN; ++e) wn[e] = wsh[grp][lane * VN + e];
            if (slot == 0) {
#pragma unroll
                for (int e = 0; e < VN; ++e) ss += wn[e] * wn[e];
            }
        }
#pragma unroll
        for (int q = 0; q < KPW; ++q) {
            acc[q] = dotv<TV>(vv[q], wn, acc[q]);
        }
#pragma unroll
        for (int q = 0; q < KPW; ++q)
#pragma unroll
            for (int e = 0; e < VN; ++e) vv[q][e] = nv[q][e];
#pragma unroll
        for (int e = 0; e < VN; ++e) we[e] = nwe[e];
    }
    if (blockIdx.x == 0 && warp == 0) {  // tail elements: one warp, serial over k
        const int i = nfull + lane;
        if (lane < n - nfull) {
            TV wi = w[i];
            for (int k = 0; k < nk; ++k) wi -= cf[k] * raw[(size_t)k * ldv + i];
            w[i] = wi;
            ss += wi * wi;
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && grp == 0) {
        const int i = nfull + lane;
        if (lane < n - nfull) {
#pragma unroll
            for (int q = 0; q < KPW; ++q) {
                const int k = slot + nwg * q;
                if (k < nk) acc[q] += raw[(size_t)k * ldv + i] * w[i];
            }
        }
    }
    __shared__ double bs[KW * KPW], tot[KW * KPW];
    group_sums<TV>(acc, nk, nwg, bs);
    if (lagged) {
        // block sum of ||w'||^2 next to the dots (nk < SG_LAGM)
        __shared__ double red_ss[KW];
        if (slot == 0 || warp == 0) {
            const double v = (double)warp_sum(ss);
            if (lane == 0) red_ss[warp] = v;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = red_ss[0];
            for (int g = 1; g < ngrp; ++g) t += red_ss[g * nwg];
            bs[nk] = t;
        }
        cp_async_wait();
        __syncthreads();
        if (cluster_reduce(partials, counter, bs, nk + 1, tot))
            lagged_pass_b(st, nk - 1, m, tot, tot[nk], hist, hist_cap, lag_in, lagged == 2,
                          sizeof(TV) == 8 ? 0x1p-53 : 0x1p-24);
        return;
    }
    if (cluster_reduce(partials, counter, bs, nk, tot)) {
        for (int k = threadIdx.x; k < nk; k += blockDim.x) {
            const double h = st->vscale[k] * tot[k];
            st->h[k] = h;
            st->hsum[k] += h;
        }
    }
}

// ---- generic update: w -= sum_k c_k raw_k (any nk)
template <class TV>
__global__ void __launch_bounds__(KT)
k_upd(const TV* __restrict__ raw, size_t ldv, int n, int nk, TV* __restrict__ w,
      SolveState* st) {
    if (!st->cycle_active) return;
    __shared__ TV cf[SG_MMAX + 1];
    for (int k = threadIdx.x; k < nk; k += blockDim.x) cf[k] = (TV)(st->h[k] * st->vscale[k]);
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        TV wi = w[i];
        for (int k = 0; k < nk; ++k) wi -= cf[k] * raw[(size_t)k * ldv + i];
        w[i] = wi;
    }
}

// ---- pass C: w'' = w' - sum c_k raw_k ; ||w''||^2 -> Arnoldi finalize.
// 16-byte vectors of elements per thread, the k loop unrolled by 4 so four
// basis loads are in flight per thread.
template <class TV>
__global__ void __launch_bounds__(KT)
k_upd_norm(const TV* __restrict__ raw, size_t ldv, int n, int j, int m, TV* __restrict__ w,
           SolveState* st, double* partials, unsigned* counter, double* hist, int hist_cap) {
    if (!st->cycle_active) return;
    constexpr int VN = Vec<TV>::N;
    const int nk = j + 1;
    __shared__ TV cf[SG_MMAX + 1];
    for (int k = threadIdx.x; k < nk; k += blockDim.x) cf[k] = (TV)(st->h[k] * st->vscale[k]);
    __syncthreads();
    TV ss = (TV)0;
    const int nvec = n / VN;
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < nvec; u += gridDim.x * blockDim.x) {
        TV wv[VN];
        vload<TV>(w + (size_t)u * VN, wv);
        int k = 0;
        for (; k + 4 <= nk; k += 4) {
            TV a[4][VN];
#pragma unroll
            for (int q = 0; q < 4; ++q) vload<TV>(raw + (size_t)(k + q) * ldv + (size_t)u * VN, a[q]);
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int e = 0; e < VN; ++e) wv[e] -= cf[k + q] * a[q][e];
        }
        for (; k < nk; ++k) {
            TV a[VN];
            vload<TV>(raw + (size_t)k * ldv + (size_t)u * VN, a);
#pragma unroll
            for (int e = 0; e < VN; ++e) wv[e] -= cf[k] * a[e];
        }
        vstore<TV>(w + (size_t)u * VN, wv);
#pragma unroll
        for (int e = 0; e < VN; ++e) ss += wv[e] * wv[e];
    }
    for (int i = nvec * VN + blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        TV wi = w[i];
        for (int k = 0; k < nk; ++k) wi -= cf[k] * raw[(size_t)k * ldv + i];
        w[i] = wi;
        ss += wi * wi;
    }
    __shared__ double red[KT / 32];
    __shared__ double bs[1], tot[1];
    TV v1[1] = {ss};
    block_sum_multi<1>(v1, 1, red, bs);
    if (cluster_reduce(partials, counter, bs, 1, tot))
        arnoldi_finalize(st, j, m, tot[0], hist, hist_cap);
}

// ---- cycle start: beta = ||raw0||
template <class TV>
__global__ void __launch_bounds__(KT)
k_cycle_init(const TV* __restrict__ raw0, int n, SolveState* st, int m, int flexible,
             double* partials, unsigned* counter) {
    if (st->done) return;
    constexpr int VN = Vec<TV>::N;
    TV ss = (TV)0;  // per-thread sum in the basis precision
    const int nvec = n / VN;
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < nvec; u += gridDim.x * blockDim.x) {
        TV v[VN];
        vload<TV>(raw0 + (size_t)u * VN, v);
#pragma unroll
        for (int e = 0; e < VN; ++e) ss += v[e] * v[e];
    }
    if (blockIdx.x == 0 && (int)threadIdx.x < n - nvec * VN) {
        const TV t = raw0[nvec * VN + threadIdx.x];
        ss += t * t;
    }
    __shared__ double red[KT / 32];
    __shared__ double bs[1], tot[1];
    TV v1[1] = {ss};
    block_sum_multi<1>(v1, 1, red, bs);
    if (!cluster_reduce(partials, counter, bs, 1, tot)) return;
    const int ld = m + 1;
    for (int i = threadIdx.x; i < ld * m; i += blockDim.x) st->H[i] = 0.0;
    for (int i = threadIdx.x; i <= m; i += blockDim.x) st->g[i] = 0.0;
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double beta = sqrt(tot[0]);
    st->beta = beta;
    st->j = 0;
    st->kcount = 0;
    st->breakdown = 0;
    if (!isfinite(beta)) {
        st->nonfinite = 1;
        st->done = 1;
        st->cycle_active = 0;
        return;
    }
    if (st->tol_kind == SG_TOL_REF_ABS && beta < st->tol) {
        // src/core/gmres.cpp:264-269
        st->converged = 1;
        st->done = 1;
        st->cycle_active = 0;
        return;
    }
    if (!(beta > 0.0)) {
        st->done = 1;
        st->cycle_active = 0;
        return;
    }
    st->vscale[0] = 1.0 / beta;
    st->lagT[0] = 1.0 / beta;  // lagged CGS2: v_0 = raw_0 / beta
    st->g[0] = beta;
    st->est_scale = flexible ? 1.0 : st->rnorm / beta;
    st->cycle_active = 1;
}

// y = H^{-1} g on the k x k upper triangle of the rotated Hessenberg
// (src/core/gmres.cpp:131-137).  Up to SG_LAGM columns one warp solves it in
// shared memory column by column (y_i, then every lane updates its rows);
// longer triangles use one thread.  Lagged CGS2: also the coefficients on
// the stored vectors, cfu = T y.
__global__ void __launch_bounds__(BS_T) k_backsolve(SolveState* st, int m) {
    if (blockIdx.x != 0) return;
    const int k = st->kcount;
    const int ld = m + 1;
    const int tid = threadIdx.x, lane = tid & 31;
    if (k > SG_LAGM) {
        if (tid != 0) return;
        for (int i = k - 1; i >= 0; --i) {
            double yi = st->g[i];
            for (int l = i + 1; l < k; ++l) yi -= st->H[i + l * ld] * st->y[l];
            st->y[i] = yi / st->H[i + i * ld];
        }
        return;
    }
    // the whole block loads R (and T) with independent loads; one warp then
    // solves, the block forms T y
    __shared__ double Hs[SG_LAGM][SG_LAGM + 1], Ts[SG_LAGM][SG_LAGM + 1];
    __shared__ double gs[SG_LAGM], ys[SG_LAGM];
    const bool lagged = st->lagged != 0;
    for (int idx = tid; idx < k * k; idx += blockDim.x) {
        const int i = idx % k, l = idx / k;
        Hs[i][l] = i <= l ? st->H[i + l * ld] : 0.0;
        if (lagged) Ts[i][l] = i <= l ? st->lagT[i + l * SG_LAGM] : 0.0;
    }
    for (int i = tid; i < k; i += blockDim.x) gs[i] = st->g[i];
    __syncthreads();
    if (tid < 32) {
        for (int i = k - 1; i >= 0; --i) {
            const double yi = gs[i] / Hs[i][i];
            if (lane == 0) ys[i] = yi;
            for (int t = lane; t < i; t += 32) gs[t] -= Hs[t][i] * yi;
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = tid; i < k; i += blockDim.x) st->y[i] = ys[i];
    if (!lagged) return;
    // V y = S (T y): coefficients on the stored vectors
    for (int i = tid; i < k; i += blockDim.x) {
        double u = 0.0;
        for (int l = i; l < k; ++l) u += Ts[i][l] * ys[l];
        st->cfu[i] = u;
    }
}

// x += V y: the correction is formed in the basis precision (FP32 for the
// mixed solver: the inner solve's precision) and added to x in FP64.  A
// thread takes one 16-byte vector of elements and four basis vectors' loads
// at a time; per element the terms are summed in basis order.
template <class TV>
__global__ void __launch_bounds__(KT)
k_update_x(const TV* __restrict__ basis, size_t ldv, int n, double* __restrict__ x,
           SolveState* st) {
    const int k = st->kcount;
    if (k <= 0) return;
    constexpr int VN = Vec<TV>::N;
    __shared__ TV cf[SG_MMAX];
    for (int i = threadIdx.x; i < k; i += blockDim.x)
        cf[i] = st->lagged ? (TV)st->cfu[i] : (TV)(st->y[i] * st->vscale[i]);
    __syncthreads();
    const int nvec = n / VN;
    const int stride = gridDim.x * blockDim.x;
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < nvec; u += stride) {
        TV d[VN];
#pragma unroll
        for (int e = 0; e < VN; ++e) d[e] = (TV)0;
        int q = 0;
        for (; q + 4 <= k; q += 4) {
            TV a[4][VN];
#pragma unroll
            for (int r = 0; r < 4; ++r) vload<TV>(basis + (size_t)(q + r) * ldv + (size_t)u * VN, a[r]);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int e = 0; e < VN; ++e) d[e] += cf[q + r] * a[r][e];
        }
        for (; q < k; ++q) {
            TV a[VN];
            vload<TV>(basis + (size_t)q * ldv + (size_t)u * VN, a);
#pragma unroll
            for (int e = 0; e < VN; ++e) d[e] += cf[q] * a[e];
        }
#pragma unroll
        for (int e = 0; e < VN; ++e) x[(size_t)u * VN + e] += (double)d[e];
    }
    for (int i = nvec * VN + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        TV d = (TV)0;
        for (int q = 0; q < k; ++q) d += cf[q] * basis[(size_t)q * ldv + i];
        x[i] += (double)d;
    }
}

template <class TI, class TO>
__global__ void k_copy(const TI* __restrict__ x, TO* __restrict__ y, int n,
                       const int* __restrict__ active) {
    if (active && *active == 0) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        y[i] = (TO)x[i];
}

__global__ void k_cycle_end(SolveState* st) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    st->cycles++;
    if (!st->done && st->total_iter >= st->max_iter) st->done = 1;
    st->cycle_active = st->done ? 0 : 1;
}

// ---- BLAS-1 of src/core/vector.h:11-44
// dot: per-thread sums in a fixed grid-stride order, block sums, then the
// last block adds the block partials in block order (deterministic).
__global__ void __launch_bounds__(KT)
k_dot(const double* __restrict__ x, const double* __restrict__ y, int n, double* partials,
      unsigned* counter, double* out) {
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        acc = fma(x[i], y[i], acc);
    __shared__ double red[KT / 32];
    __shared__ double bs[1], tot[1];
    double v1[1] = {acc};
    block_sum_multi<1>(v1, 1, red, bs);
    if (last_block_reduce(partials, counter, bs, 1, tot) && threadIdx.x == 0) *out = tot[0];
}

// y += alpha x, product and sum rounded separately (the reference's bits)
__global__ void k_axpy(double alpha, const double* __restrict__ x, double* __restrict__ y, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        y[i] = __dadd_rn(y[i], __dmul_rn(alpha, x[i]));
}

__global__ void k_scale(double alpha, double* __restrict__ x, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[i] = __dmul_rn(x[i], alpha);
}

int kgrid(sg_ctx* ctx, int n, int per_sm) {
    long long need = ((long long)n + KT - 1) / KT;
    long long cap = (long long)ctx->num_sms * per_sm;
    if (need > cap) need = cap;
    return need < 1 ? 1 : (int)need;
}

// Launches a reducing kernel over `need` blocks of work in clusters.  Up to 32
// blocks' worth runs as one cluster of up to eight blocks (its reduction stays
// in shared memory; up to four rounds of tiles cost less than the global
// round trip); a larger grid has clusters of four (two passes at 128^3 FP32
// take 70.8, 66.3, 63.6 and 64.3 us with clusters of 1, 2, 4 and 8), at most
// as many as are resident at once (the GPU's processor groups do not divide
// evenly, and a second wave of a few clusters would double the time: 84 us).
template <class... P, class... A>
void launch_clusters(sg_ctx* ctx, long long need, void (*kern)(P...), A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(KT);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL_SIZE;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (need <= 4 * CL_MAX) {
        unsigned c = 1;
        while (c < need && c < CL_MAX) c *= 2;
        at[0].val.clusterDim.x = c;
        cfg.gridDim = dim3(c);
    } else {
        int& cap = ctx->max_clusters[reinterpret_cast<const void*>(kern)];
        cfg.gridDim = dim3(CL_SIZE);
        if (cap == 0) {
            SG_CUDA(cudaOccupancyMaxActiveClusters(&cap, kern, &cfg));
            if (cap < 1) fail(SG_ERR_INTERNAL, "a reduction's clusters do not fit this GPU");
        }
        const long long ncl = (need + CL_SIZE - 1) / CL_SIZE;
        cfg.gridDim = dim3((unsigned)(CL_SIZE * std::min<long long>(ncl, cap)));
    }
    SG_CUDA(cudaLaunchKernelEx(&cfg, kern, P(args)...));
    count_launch(ctx);
}

// blocks that give every tile group of a pass over nk vectors one tile
template <class TV>
long long tile_blocks(int n, int nk) {
    const long long tiles = ((long long)n / Vec<TV>::N + 31) / 32;
    return (tiles * warps_per_tile(nk) + KW - 1) / KW;
}

}  // namespace

template <class TV>
void launch_cycle_init(sg_ctx* ctx, const TV* raw0, int n, SolveState* st, int m, bool flexible) {
    launch_clusters(ctx, n / (4 * KT) + 1, k_cycle_init<TV>, raw0, n, st, m,
                    flexible ? 1 : 0, ctx->partials.p, ctx->counter.p);
}

// the kernel for nk vectors
template <class TV>
static auto dots_kernel(int nk) {
    switch (warps_per_tile(nk)) {
    case 1: return k_dots<TV, 1>;
    case 2: return k_dots<TV, 2>;
    case 4: return k_dots<TV, 4>;
    default: return k_dots<TV, 8>;
    }
}
template <class TV>
static auto upd_dots_kernel(int nk) {
    switch (warps_per_tile(nk)) {
    case 1: return k_upd_dots<TV, 1>;
    case 2: return k_upd_dots<TV, 2>;
    case 4: return k_upd_dots<TV, 4>;
    default: return k_upd_dots<TV, 8>;
    }
}

template <class TV>
static void dots_any(sg_ctx* ctx, const TV* raw, size_t ldv, int n, int nk, const TV* w,
                     SolveState* st, int second, int lagged = 0) {
    for (int k0 = 0; k0 < nk; k0 += KW * KPW) {
        const int kc = nk - k0 < KW * KPW ? nk - k0 : KW * KPW;
        launch_clusters(ctx, tile_blocks<TV>(n, kc), dots_kernel<TV>(kc), raw, ldv, n,
                        k0, kc, w, st, second, lagged, ctx->partials.p, ctx->counter.p);
    }
}

template <class TV>
void launch_cgs2(sg_ctx* ctx, TV* raw, size_t ldv, int n, int j, int m, SolveState* st,
                 int lagged) {
    const int nk = j + 1;
    TV* w = raw + (size_t)(j + 1) * ldv;
    if (lagged) {
        // two passes (see lagged_pass_a / lagged_pass_b); m < SG_LAGM <= 32
        if (m >= SG_LAGM || nk > KW * KPW) fail(SG_ERR_INTERNAL, "lagged CGS2 needs m < %d", SG_LAGM);
        dots_any<TV>(ctx, raw, ldv, n, nk, w, st, 0, 1);
        launch_clusters(ctx, tile_blocks<TV>(n, nk), upd_dots_kernel<TV>(nk), raw, ldv,
                        n, nk, w, st, ctx->partials.p, ctx->counter.p, lagged, m, ctx->hist_d,
                        ctx->hist_cap);
        return;
    }
    // pass A
    dots_any<TV>(ctx, raw, ldv, n, nk, w, st, 0);
    // pass B
    if (nk <= KW * KPW) {
        launch_clusters(ctx, tile_blocks<TV>(n, nk), upd_dots_kernel<TV>(nk), raw, ldv,
                        n, nk, w, st, ctx->partials.p, ctx->counter.p, 0, m, (double*)nullptr, 0);
    } else {
        k_upd<TV><<<kgrid(ctx, n, 4), KT, 0, ctx->stream>>>(raw, ldv, n, nk, w, st);
        SG_CUDA(cudaGetLastError());
        count_launch(ctx);
        dots_any<TV>(ctx, raw, ldv, n, nk, w, st, 1);
    }
    // pass C
    launch_clusters(ctx, n / (Vec<TV>::N * KT) + 1, k_upd_norm<TV>, raw, ldv,
                    n, j, m, w, st, ctx->partials.p, ctx->counter.p, ctx->hist_d, ctx->hist_cap);
}

void launch_backsolve(sg_ctx* ctx, SolveState* st, int m) {
    k_backsolve<<<1, BS_T, 0, ctx->stream>>>(st, m);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

template <class TV>
void launch_update_x(sg_ctx* ctx, const TV* basis, size_t ldv, int n, double* x, SolveState* st) {
    k_update_x<TV><<<kgrid(ctx, n, 4), KT, 0, ctx->stream>>>(basis, ldv, n, x, st);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

template <class TI, class TO>
void launch_copy(sg_ctx* ctx, const TI* x, TO* y, int n, const int* active) {
    k_copy<TI, TO><<<kgrid(ctx, n, 4), KT, 0, ctx->stream>>>(x, y, n, active);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

// grid of the dot-product reduction: at most 1024 blocks
int dot_grid(int num_sms, int n) {
    long long need = ((long long)n + KT - 1) / KT;
    long long cap = (long long)num_sms * 2;
    if (cap > 1024) cap = 1024;
    if (need > cap) need = cap;
    return need < 1 ? 1 : (int)need;
}

void launch_dot(sg_ctx* ctx, const double* x, const double* y, int n, double* out_dev) {
    k_dot<<<dot_grid(ctx->num_sms, n), KT, 0, ctx->stream>>>(x, y, n, ctx->partials.p,
                                                              ctx->counter.p, out_dev);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

void launch_dot_scratch(cudaStream_t stream, const double* x, const double* y, int n,
                        int blocks, double* partials, unsigned* counter, double* out_dev) {
    k_dot<<<blocks, KT, 0, stream>>>(x, y, n, partials, counter, out_dev);
    SG_CUDA(cudaGetLastError());
}

void launch_axpy(sg_ctx* ctx, double alpha, const double* x, double* y, int n) {
    k_axpy<<<kgrid(ctx, n, 8), KT, 0, ctx->stream>>>(alpha, x, y, n);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

void launch_scale(sg_ctx* ctx, double alpha, double* x, int n) {
    k_scale<<<kgrid(ctx, n, 8), KT, 0, ctx->stream>>>(alpha, x, n);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

void launch_cycle_end(sg_ctx* ctx, SolveState* st) {
    k_cycle_end<<<1, 32, 0, ctx->stream>>>(st);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

template void launch_cycle_init<double>(sg_ctx*, const double*, int, SolveState*, int, bool);
template void launch_cycle_init<float>(sg_ctx*, const float*, int, SolveState*, int, bool);
template void launch_cgs2<double>(sg_ctx*, double*, size_t, int, int, int, SolveState*, int);
template void launch_cgs2<float>(sg_ctx*, float*, size_t, int, int, int, SolveState*, int);
template void launch_update_x<double>(sg_ctx*, const double*, size_t, int, double*, SolveState*);
template void launch_update_x<float>(sg_ctx*, const float*, size_t, int, double*, SolveState*);
template void launch_copy<double, double>(sg_ctx*, const double*, double*, int, const int*);
template void launch_copy<double, float>(sg_ctx*, const double*, float*, int, const int*);
template void launch_copy<float, float>(sg_ctx*, const float*, float*, int, const int*);
template void launch_copy<float, double>(sg_ctx*, const float*, double*, int, const int*);

}  // namespace sg
