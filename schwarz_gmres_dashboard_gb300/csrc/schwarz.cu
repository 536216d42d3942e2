// schwarz.cu -- device side of the preconditioners: Jacobi
// (src/precond/jacobi.h:10-27), ILU(0) (src/precond/ilu0.h:13-79), one-level
// ASM/RAS (src/precond/asm.h:34-60, src/precond/ras.h:45-70) and the
// piecewise-constant two-level coarse space (src/precond/coarse_space.h:26-78,
// src/precond/coarse_solve.h:15-67).  Replaces the host-staged GPU path of
// src/gpu/asm_gpu.h:108-165 and the single-thread sweep kernel of
// src/gpu/local_solve_kernel.cu:13-74.
//
// Every subdomain stays resident on the device.  One CTA owns one subdomain:
// it gathers its overlapped right-hand side from the global vector (the
// restriction that replaces the MPI halo exchange), runs the ILU(0) forward
// and backward sweeps in shared memory level by level (rows of one level are
// independent; one __syncthreads per level), and scatters its owned rows
// (RAS) or all rows with atomics (ASM), adding the coarse correction of its
// own part.  Factors are stored per level in ELL slices, so the threads of a
// level read them with coalesced loads.
#include <algorithm>

#include "dev_common.cuh"
#include "kernels.h"

namespace sg {

namespace {

constexpr int SWEEP_T = 512;

// ---------------------------------------------------------------- Jacobi
__global__ void k_jacobi_setup(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                               const double* __restrict__ v, double* inv, float* inv32) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        // CSRMatrix::diagonal (src/core/sparse_matrix.h:45-51): first match, else 0
        double d = 0.0;
        for (int e = rp[i]; e < rp[i + 1]; ++e)
            if (ci[e] == i) {
                d = v[e];
                break;
            }
        const double r = (fabs(d) > 1e-15) ? 1.0 / d : 1.0;
        inv[i] = r;
        inv32[i] = (float)r;
    }
}

template <class TI, class TO, class TD>
__global__ void k_jacobi(int n, const TD* __restrict__ inv, const TI* __restrict__ x,
                         TO* __restrict__ y, const int* __restrict__ active) {
    if (active && *active == 0) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (sizeof(TD) == 8) y[i] = (TO)__dmul_rn((double)inv[i], (double)x[i]);
        else y[i] = (TO)((float)inv[i] * (float)x[i]);
    }
}

// ---------------------------------------------------------------- ILU(0) set-up
__global__ void k_gather_vals(long long nz, const int* __restrict__ map,
                              const double* __restrict__ aval, double* __restrict__ lu) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nz;
         e += (long long)gridDim.x * blockDim.x)
        lu[e] = aval[map[e]];
}

// In-place ILU(0) of every subdomain, rows in forward-level order; the
// arithmetic of one row is src/precond/ilu0.h:313-333 step for step (same
// skip rule, same first-match search, product and difference rounded
// separately).
//
// A level is a chain of dependent loads: the row, the pivot rows' positions,
// their entries.  For rows of stencils (at most FAC_W entries, FAC_L of them
// below the diagonal, pivot rows with at most FAC_L entries above theirs) all
// pivot rows are fetched and matched before the first division, so a level
// costs three round trips and then only arithmetic; other rows fetch as they
// go.  64 subdomains of 64^3, 52 levels: 0.63 ms before, 0.45 now.
//
// A level of more rows than threads takes several rounds, so a subdomain that
// has an SM to itself takes FAC_T threads (one subdomain of 1600 x 1600, levels
// of up to 1,600 rows: a set-up of 102 ms with half of them, 82 so); two blocks of
// half the threads share one otherwise (1,000 subdomains of 128^3: 6.4 ms, 7.1
// with whole ones).
constexpr int FAC_T = 512;
constexpr int FAC_W = 9;
constexpr int FAC_L = 4;
__device__ __forceinline__ void factor_row(int i, const int* __restrict__ rp,
                                           const int* __restrict__ ci, const int* __restrict__ dg,
                                           double* v) {
    const int rs = rp[i], re = rp[i + 1];
    for (int jp = rs; jp < re; ++jp) {
        const int k = ci[jp];
        if (k >= i) break;
        const int dk = dg[k];
        if (dk < 0 || fabs(v[dk]) < 1e-30) continue;
        const double a = v[jp] / v[dk];
        v[jp] = a;
        const int ke = rp[k + 1];
        for (int kp = dk + 1; kp < ke; ++kp) {
            const int col = ci[kp];
            for (int ip = rs; ip < re; ++ip) {
                if (ci[ip] == col) {
                    v[ip] = __dsub_rn(v[ip], __dmul_rn(a, v[kp]));
                    break;
                }
            }
        }
    }
}

template <class TC, int T>
__global__ void __launch_bounds__(T, FAC_T / T)
k_factor(const SubInfo* __restrict__ info, const int* __restrict__ lrp,
         const int* __restrict__ lci, const int* __restrict__ ldiag,
         const TC* __restrict__ perm_f, const int* __restrict__ lev_f, double* lu) {
    __shared__ double s_v[FAC_W][T];  // each thread's row
    const SubInfo inf = info[blockIdx.x];
    const int* rp = lrp + inf.csr_row_off;
    const int* ci = lci + inf.csr_nz_off;
    double* v = lu + inf.csr_nz_off;
    const int* dg = ldiag + inf.row_off;
    const TC* pf = perm_f + inf.row_off;
    const int* lf = lev_f + inf.lev_off_f;
    const int tid = threadIdx.x;
    for (int l = 0; l < inf.nlev_f; ++l) {
        const int p0 = lf[l], p1 = lf[l + 1];
        for (int p = p0 + tid; p < p1; p += T) {
            const int i = pf[p];
            const int rs = rp[i], w = rp[i + 1] - rs;
            bool fast = w <= FAC_W;
            int c[FAC_W], dk[FAC_L], nk[FAC_L];
#pragma unroll
            for (int e = 0; e < FAC_W; ++e) {
                c[e] = fast && e < w ? ci[rs + e] : 0x7fffffff;
                s_v[e][tid] = fast && e < w ? v[rs + e] : 0.0;
            }
            // pivots: the entries before the first column >= i
            int np = 0;
#pragma unroll
            for (int e = 0; e < FAC_W; ++e) np += np == e && c[e] < i;
            fast = fast && np <= FAC_L;
#pragma unroll
            for (int t = 0; t < FAC_L; ++t) {
                const bool on = fast && t < np;
                dk[t] = on ? dg[c[t]] : -1;
                nk[t] = on && dk[t] >= 0 ? rp[c[t] + 1] - dk[t] - 1 : 0;
                fast = fast && nk[t] <= FAC_L;
            }
            if (!fast) {
                factor_row(i, rp, ci, dg, v);
                continue;
            }
            double d[FAC_L], u[FAC_L][FAC_L];
            unsigned at[FAC_L];  // entry of this row that each pivot row's entry meets, 8 bits each
#pragma unroll
            for (int t = 0; t < FAC_L; ++t) {
                d[t] = dk[t] >= 0 ? v[dk[t]] : 0.0;
                at[t] = 0;
#pragma unroll
                for (int q = 0; q < FAC_L; ++q) {
                    const bool on = q < nk[t];
                    u[t][q] = on ? v[dk[t] + 1 + q] : 0.0;
                    const int col = on ? ci[dk[t] + 1 + q] : -1;
                    unsigned m = FAC_W;
#pragma unroll
                    for (int e = FAC_W - 1; e >= 0; --e)
                        if (c[e] == col) m = e;
                    at[t] |= m << (8 * q);
                }
            }
#pragma unroll
            for (int t = 0; t < FAC_L; ++t) {
                // |d| as an integer: the order is the same and the FP64 pipe is left alone
                const long long mag = __double_as_longlong(d[t]) & 0x7fffffffffffffffll;
                if (dk[t] < 0 || mag < __double_as_longlong(1e-30)) continue;
                const double a = s_v[t][tid] / d[t];
                s_v[t][tid] = a;
#pragma unroll
                for (int q = 0; q < FAC_L; ++q) {
                    const unsigned m = at[t] >> (8 * q) & 0xff;
                    if (m < FAC_W) s_v[m][tid] = __dsub_rn(s_v[m][tid], __dmul_rn(a, u[t][q]));
                }
            }
#pragma unroll
            for (int e = 0; e < FAC_W; ++e)
                if (e < w) v[rs + e] = s_v[e][tid];
        }
        __syncthreads();
    }
}

template <class TF>
__device__ __forceinline__ TF cvt_factor(double v);
template <>
__device__ __forceinline__ double cvt_factor<double>(double v) { return v; }
template <>
__device__ __forceinline__ float cvt_factor<float>(double v) { return (float)v; }
template <>
__device__ __forceinline__ uint16_t cvt_factor<uint16_t>(double v) {
    return __bfloat16_as_ushort(__float2bfloat16_rn((float)v));
}

// Factored local CSR -> level-major ELL slices of type TF.
template <class TF, class TC>
__global__ void __launch_bounds__(SWEEP_T, 2)
k_pack(const SubInfo* __restrict__ info, const int* __restrict__ lrp,
       const int* __restrict__ lci, const int* __restrict__ ldiag,
       const double* __restrict__ lu, const TC* __restrict__ perm_f,
       const TC* __restrict__ perm_b, TC* lcol, TF* lval, TC* ucol, TF* uval, TF* udiag) {
    const SubInfo inf = info[blockIdx.x];
    const int n = inf.n;
    const int* rp = lrp + inf.csr_row_off;
    const int* ci = lci + inf.csr_nz_off;
    const double* v = lu + inf.csr_nz_off;
    const int* dg = ldiag + inf.row_off;
    for (int p = threadIdx.x; p < n; p += blockDim.x) {
        const int r = perm_f[inf.row_off + p];
        int k = 0;
        for (int e = rp[r]; e < rp[r + 1] && k < inf.wl; ++e) {
            const int c = ci[e];
            if (c >= r) break;
            lcol[inf.fl_off + (long long)k * n + p] = (TC)c;
            lval[inf.fl_off + (long long)k * n + p] = cvt_factor<TF>(v[e]);
            ++k;
        }
        for (; k < inf.wl; ++k) {
            lcol[inf.fl_off + (long long)k * n + p] = (TC)n;
            lval[inf.fl_off + (long long)k * n + p] = cvt_factor<TF>(0.0);
        }
        const int rb = perm_b[inf.row_off + p];
        k = 0;
        for (int e = dg[rb] + 1; e < rp[rb + 1] && k < inf.wu; ++e) {
            ucol[inf.fu_off + (long long)k * n + p] = (TC)ci[e];
            uval[inf.fu_off + (long long)k * n + p] = cvt_factor<TF>(v[e]);
            ++k;
        }
        for (; k < inf.wu; ++k) {
            ucol[inf.fu_off + (long long)k * n + p] = (TC)n;
            uval[inf.fu_off + (long long)k * n + p] = cvt_factor<TF>(0.0);
        }
        udiag[inf.row_off + p] = cvt_factor<TF>(v[dg[rb]]);
    }
}

// ---------------------------------------------------------------- sweeps
// One triangular sweep of a subdomain held in shared memory `t`.  Rows of a
// level are independent; a __syncthreads separates levels.  The factor
// entries, columns and row index of the next level are loaded into registers
// before the current level is computed, so the global-memory latency of level
// l+1 overlaps the arithmetic and the barrier of level l.  The per-row order
// of the subtractions (and the final division of the backward sweep) is the
// reference's (src/precond/ilu0.h:62-76).
constexpr int SWEEP_WP = 4;  // ELL widths up to this are prefetched

template <class TS, class TF, class TC, bool BACK>
__device__ __forceinline__ void sweep_levels(TS* t, int n, int nlev, const int* __restrict__ lptr,
                                             const TC* __restrict__ perm,
                                             const TC* __restrict__ col,
                                             const TF* __restrict__ val,
                                             const TF* __restrict__ diag, int w) {
    if (w > SWEEP_WP) {
        for (int l = 0; l < nlev; ++l) {
            const int p0 = lptr[l], p1 = lptr[l + 1];
            for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
                const int r = perm[p];
                TS acc = t[r];
                for (int k = 0; k < w; ++k)
                    acc = msub(acc, Load<TS>::f(val[(size_t)k * n + p]), t[col[(size_t)k * n + p]]);
                if (BACK) acc = div_diag(acc, Load<TS>::f(diag[p]));
                t[r] = acc;
            }
            __syncthreads();
        }
        return;
    }
    // registers for the first pass of the next level
    bool have = false;
    int r = 0;
    TS v[SWEEP_WP];
    int c[SWEEP_WP];
    TS d = (TS)1;
    auto fetch = [&](int p) {
        r = perm[p];
#pragma unroll
        for (int k = 0; k < SWEEP_WP; ++k) {
            if (k < w) {
                v[k] = Load<TS>::f(val[(size_t)k * n + p]);
                c[k] = col[(size_t)k * n + p];
            }
        }
        if (BACK) d = Load<TS>::f(diag[p]);
    };
    if (nlev > 0) {
        const int p = lptr[0] + threadIdx.x;
        have = p < lptr[1];
        if (have) fetch(p);
    }
    for (int l = 0; l < nlev; ++l) {
        const int p0 = lptr[l], p1 = lptr[l + 1];
        const bool cur = have;
        const int rc = r;
        TS vc[SWEEP_WP];
        int cc[SWEEP_WP];
#pragma unroll
        for (int k = 0; k < SWEEP_WP; ++k) {
            vc[k] = v[k];
            cc[k] = c[k];
        }
        const TS dc = d;
        have = false;
        if (l + 1 < nlev) {
            const int q = p1 + threadIdx.x;
            have = q < lptr[l + 2];
            if (have) fetch(q);
        }
        if (cur) {
            TS acc = t[rc];
#pragma unroll
            for (int k = 0; k < SWEEP_WP; ++k)
                if (k < w) acc = msub(acc, vc[k], t[cc[k]]);
            if (BACK) acc = div_diag(acc, dc);
            t[rc] = acc;
        }
        // rows of this level beyond the first pass
        for (int q = p0 + threadIdx.x + blockDim.x; q < p1; q += blockDim.x) {
            const int rr = perm[q];
            TS acc = t[rr];
            for (int k = 0; k < w; ++k)
                acc = msub(acc, Load<TS>::f(val[(size_t)k * n + q]), t[col[(size_t)k * n + q]]);
            if (BACK) acc = div_diag(acc, Load<TS>::f(diag[q]));
            t[rr] = acc;
        }
        __syncthreads();
    }
}

// mode 0: RAS (owned rows written), 1: ASM (all rows added atomically).
template <class TI, class TO, class TS, class TF, class TC>
__global__ void __launch_bounds__(SWEEP_T, 2)
k_sweep(const SubInfo* __restrict__ info, const int* __restrict__ order,
        const int* __restrict__ dofs, const TC* __restrict__ perm_f,
        const int* __restrict__ lev_f, const TC* __restrict__ lcol, const TF* __restrict__ lval,
        const TC* __restrict__ perm_b, const int* __restrict__ lev_b,
        const TC* __restrict__ ucol, const TF* __restrict__ uval,
        const TF* __restrict__ udiag, const int* __restrict__ ownloc,
        const int* __restrict__ owned_glob, const TI* __restrict__ x, TO* __restrict__ y,
        int mode, int coarse, const double* __restrict__ a0inv, const double* __restrict__ r0,
        int nc, TS* gscratch, int use_smem, const int* __restrict__ active,
        const int* __restrict__ sub_on) {
    if (active && *active == 0) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double s_zc;
    const int s = order[blockIdx.x];
    if (sub_on && !sub_on[s]) return;  // subdomain not needed by this apply
    const SubInfo inf = info[s];
    const int n = inf.n;
    TS* t = use_smem ? reinterpret_cast<TS*>(smraw) : gscratch + inf.row_off + s;
    const int* dof = dofs + inf.row_off;
    // restriction R_s x (gather with overlap)
    gather_rows<TS>(t, x, dof, n, blockDim.x);
    if (threadIdx.x == 0) t[n] = (TS)0;
    if (coarse) {
        // z0_s = (A0^{-1} r0)_s, scaled by the part's coarse basis value
        if (threadIdx.x < 32) {
            const double z = coarse_dot_warp0(a0inv + (size_t)s * nc, r0, nc);
            if (threadIdx.x == 0) s_zc = inf.cscale * z;
        }
        __syncthreads();
    }
    __syncthreads();
    // forward sweep (unit lower triangle), then backward sweep (upper
    // triangle and diagonal), level by level
    sweep_levels<TS, TF, TC, false>(t, n, inf.nlev_f, lev_f + inf.lev_off_f, perm_f + inf.row_off,
                                    lcol + inf.fl_off, lval + inf.fl_off, nullptr, inf.wl);
    sweep_levels<TS, TF, TC, true>(t, n, inf.nlev_b, lev_b + inf.lev_off_b, perm_b + inf.row_off,
                                   ucol + inf.fu_off, uval + inf.fu_off, udiag + inf.row_off,
                                   inf.wu);
    const double zc = coarse ? s_zc : 0.0;
    if (mode == 0) {
        // restricted prolongation: owned rows only (src/precond/ras.h:64-68)
        const int* ol = ownloc + inf.own_off;
        const int* og = owned_glob + inf.own_off;
        scatter_owned<TS, TO>(t, y, ol, og, inf.n_own, coarse, zc, blockDim.x);
    } else {
        // additive prolongation of every row (src/precond/asm.h:138-142)
        for (int li = threadIdx.x; li < n; li += blockDim.x)
            atomicAdd(&y[dof[li]], Store<TO>::f(t[li]));
        if (coarse) {
            const int* og = owned_glob + inf.own_off;
            for (int q = threadIdx.x; q < inf.n_own; q += blockDim.x)
                atomicAdd(&y[og[q]], Store<TO>::f(zc));
        }
    }
}

// ---------------------------------------------------------------- sync-free sweeps
// The same forward/backward sweeps without a barrier per level.  Thread t
// takes the rows at level-order positions t, t + blockDim, ... and, before
// using row c, waits until c's ready flag (one byte in shared memory) shows
// the current sweep; it then publishes its own row (value, block fence,
// flag).  Every dependency sits at an earlier position and each thread walks
// its positions in increasing order, so the waits always end; they are
// bounded anyway (on expiry the thread records an error word and carries on).
// The next row's factor entries are loaded before the current row's waits,
// so their global-memory latency overlaps the dependency chain.
constexpr long long SF_SPIN_LIMIT = 1ll << 24;

template <class TS, bool EXACT>
__device__ __forceinline__ TS sf_sub(TS acc, TS a, TS b) {
    if (EXACT) return msub(acc, a, b);
    return acc - a * b;  // contracts to a fused multiply-add
}

template <class TS, class TF, class TC, bool BACK, bool EXACT>
__device__ __forceinline__ void sweep_sf(TS* t, volatile unsigned char* fl, int n,
                                         const TC* __restrict__ perm, const TC* __restrict__ col,
                                         const TF* __restrict__ val, const TF* __restrict__ diag,
                                         int w, unsigned char epoch, int* err) {
    auto wait_row = [&](int c) {
        long long it = 0;
        while (fl[c] < epoch) {
            if (++it > SF_SPIN_LIMIT) {
                atomicExch(err, 2);
                break;
            }
        }
        __threadfence_block();
    };
    if (w > SWEEP_WP) {
        for (int p = threadIdx.x; p < n; p += blockDim.x) {
            const int r = perm[p];
            TS acc = t[r];
            for (int k = 0; k < w; ++k) {
                const int c = col[(size_t)k * n + p];
                const TS v = Load<TS>::f(val[(size_t)k * n + p]);
                wait_row(c);
                acc = sf_sub<TS, EXACT>(acc, v, t[c]);
            }
            if (BACK) acc = div_diag(acc, Load<TS>::f(diag[p]));
            t[r] = acc;
            __threadfence_block();
            fl[r] = epoch;
        }
        return;
    }
    int r = 0, c[SWEEP_WP];
    TS v[SWEEP_WP], d = (TS)1;
    auto fetch = [&](int p) {
        r = perm[p];
#pragma unroll
        for (int k = 0; k < SWEEP_WP; ++k)
            if (k < w) {
                c[k] = col[(size_t)k * n + p];
                v[k] = Load<TS>::f(val[(size_t)k * n + p]);
            }
        if (BACK) d = Load<TS>::f(diag[p]);
    };
    int p = threadIdx.x;
    if (p < n) fetch(p);
    for (; p < n; p += blockDim.x) {
        const int rc = r;
        int cc[SWEEP_WP];
        TS vc[SWEEP_WP];
#pragma unroll
        for (int k = 0; k < SWEEP_WP; ++k) {
            cc[k] = c[k];
            vc[k] = v[k];
        }
        const TS dc = d;
        if (p + (int)blockDim.x < n) fetch(p + blockDim.x);
        TS acc = t[rc];
#pragma unroll
        for (int k = 0; k < SWEEP_WP; ++k) {
            if (k < w) {
                wait_row(cc[k]);
                acc = sf_sub<TS, EXACT>(acc, vc[k], t[cc[k]]);
            }
        }
        if (BACK) acc = div_diag(acc, dc);
        t[rc] = acc;
        __threadfence_block();
        fl[rc] = epoch;
    }
}

template <class TI, class TO, class TS, class TF, class TC, bool EXACT>
__global__ void __launch_bounds__(SWEEP_T, 2)
k_sweep_sf(const SubInfo* __restrict__ info, const int* __restrict__ order,
           const int* __restrict__ dofs, const TC* __restrict__ perm_f,
           const TC* __restrict__ lcol, const TF* __restrict__ lval,
           const TC* __restrict__ perm_b, const TC* __restrict__ ucol,
           const TF* __restrict__ uval, const TF* __restrict__ udiag,
           const int* __restrict__ ownloc, const int* __restrict__ owned_glob,
           const TI* __restrict__ x, TO* __restrict__ y, int mode, int coarse,
           const double* __restrict__ a0inv, const double* __restrict__ r0, int nc, int* err,
           const int* __restrict__ active, const int* __restrict__ sub_on) {
    if (active && *active == 0) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double s_zc;
    const int s = order[blockIdx.x];
    if (sub_on && !sub_on[s]) return;  // subdomain not needed by this apply
    const SubInfo inf = info[s];
    const int n = inf.n;
    TS* t = reinterpret_cast<TS*>(smraw);
    volatile unsigned char* fl =
        smraw + (((size_t)(n + 1) * sizeof(TS) + 15) & ~(size_t)15);
    const int* dof = dofs + inf.row_off;
    gather_rows<TS>(t, x, dof, n, blockDim.x);
    for (int li = threadIdx.x; li < n; li += blockDim.x) fl[li] = 0;
    if (threadIdx.x == 0) {
        t[n] = (TS)0;  // padded entries read this zero
        fl[n] = 2;
    }
    if (coarse) {
        if (threadIdx.x < 32) {
            const double z = coarse_dot_warp0(a0inv + (size_t)s * nc, r0, nc);
            if (threadIdx.x == 0) s_zc = inf.cscale * z;
        }
        __syncthreads();
    }
    __syncthreads();
    sweep_sf<TS, TF, TC, false, EXACT>(t, fl, n, perm_f + inf.row_off, lcol + inf.fl_off,
                                       lval + inf.fl_off, nullptr, inf.wl, 1, err);
    __syncthreads();  // every forward read is done before rows change again
    sweep_sf<TS, TF, TC, true, EXACT>(t, fl, n, perm_b + inf.row_off, ucol + inf.fu_off,
                                      uval + inf.fu_off, udiag + inf.row_off, inf.wu, 2, err);
    __syncthreads();
    const double zc = coarse ? s_zc : 0.0;
    if (mode == 0) {
        const int* ol = ownloc + inf.own_off;
        const int* og = owned_glob + inf.own_off;
        scatter_owned<TS, TO>(t, y, ol, og, inf.n_own, coarse, zc, blockDim.x);
    } else {
        for (int li = threadIdx.x; li < n; li += blockDim.x)
            atomicAdd(&y[dof[li]], Store<TO>::f(t[li]));
        if (coarse) {
            const int* og = owned_glob + inf.own_off;
            for (int q = threadIdx.x; q < inf.n_own; q += blockDim.x)
                atomicAdd(&y[og[q]], Store<TO>::f(zc));
        }
    }
}

// ---------------------------------------------------------------- coarse space
// A0[i][j] in the reference's summation order (see oracle notes): for every
// owned row k of part i ascending, the part-j sum of row k in entry order
// (from 0.0), then c_i times it accumulated into A0[i][j] (from 0.0), all
// rounded op by op.  Only the accumulation over the rows is serial; one block
// per part i forms the rows' terms of j = i in parallel (own, global scratch)
// and lists the rows that touch other parts.  Then one thread folds the own
// terms while the other warps stage the listed rows, A0_CH at a time, and
// give each other part j a thread that folds its terms.  (One thread per part
// walking every row and entry: 8.2 ms for 64 parts of 4096 rows, a load's
// latency per entry; folding all entries of the listed rows 0.94; now 0.50,
// half of it the listed rows' staging.)
constexpr int A0_T = 256;
constexpr int A0_CH = 32;  // listed rows staged at a time
constexpr int A0_W = 32;   // their entries; longer rows are read from global memory
__device__ __forceinline__ void a0_sync() {  // the warps that fold the other parts
    asm volatile("bar.sync 1, %0;" ::"n"(A0_T - 32) : "memory");
}
__global__ void __launch_bounds__(A0_T)
k_a0_build(int nc, const int* __restrict__ owned_ptr, const int* __restrict__ owned,
           const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
           const int* __restrict__ part, const double* __restrict__ cscale, double* own,
           int* rows, double* a0) {
    extern __shared__ __align__(16) unsigned char smraw[];
    int* flag = reinterpret_cast<int*>(smraw);  // nc
    int* list = flag + nc;                      // nc
    __shared__ int s_nl, s_cnt[A0_T / 32];
    __shared__ int s_n[A0_CH], s_e[A0_CH], s_c[A0_CH], s_p[A0_CH][A0_W], s_q[A0_CH][A0_W];
    __shared__ double s_v[A0_CH][A0_W], s_t[A0_CH][A0_W];
    const int i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q0 = owned_ptr[i], q1 = owned_ptr[i + 1];
    const double c_i = cscale[i];
    for (int t = tid; t < nc; t += A0_T) flag[t] = 0;
    __syncthreads();
    int nb = 0;  // listed rows
    for (int b = q0; b < q1; b += A0_T) {
        const int q = b + tid;
        bool other = false;
        if (q < q1) {
            const int k = owned[q];
            const int e1 = rp[k + 1];
            double acc = 0.0;
            for (int e = rp[k]; e < e1; e += 8) {  // eight entries' loads in flight
                int p[8];
                double a[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) p[u] = e + u < e1 ? ci[e + u] : -1;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    a[u] = p[u] >= 0 ? v[e + u] : 0.0;
                    p[u] = p[u] >= 0 ? part[p[u]] : -1;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (p[u] < 0) continue;
                    if (p[u] == i) {
                        acc = __dadd_rn(acc, __dmul_rn(a[u], c_i));
                    } else {
                        flag[p[u]] = 1;
                        other = true;
                    }
                }
            }
            own[q] = __dmul_rn(c_i, acc);
        }
        // the rows with entries in other parts, in order
        const unsigned m = __ballot_sync(0xffffffffu, other);
        if (lane == 0) s_cnt[warp] = __popc(m);
        __syncthreads();
        int at = nb;
        for (int w = 0; w < A0_T / 32; ++w) {
            if (w < warp) at += s_cnt[w];
            nb += s_cnt[w];
        }
        if (other) rows[q0 + at + __popc(m & ((1u << lane) - 1u))] = q;
        __syncthreads();
    }
    if (warp == 0) {  // the other touched parts, ascending
        int base = 0;
        for (int t0 = 0; t0 < nc; t0 += 32) {
            const bool on = t0 + lane < nc && t0 + lane != i && flag[t0 + lane];
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) list[base + __popc(m & ((1u << lane) - 1u))] = t0 + lane;
            base += __popc(m);
        }
        if (lane == 0) s_nl = base;
    }
    for (int t = tid; t < nc; t += A0_T) a0[(size_t)i * nc + t] = 0.0;
    __syncthreads();
    if (warp == 0) {
        if (lane != 0) return;
        double row = 0.0;  // every row has its diagonal, so every row adds its term
        double t[16], tn[16];  // the next sixteen terms load while these are added
#pragma unroll
        for (int u = 0; u < 16; ++u) t[u] = q0 + u < q1 ? own[q0 + u] : 0.0;
        for (int q = q0; q < q1; q += 16) {
#pragma unroll
            for (int u = 0; u < 16; ++u) tn[u] = q + 16 + u < q1 ? own[q + 16 + u] : 0.0;
#pragma unroll
            for (int u = 0; u < 16; ++u)
                if (q + u < q1) row = __dadd_rn(row, t[u]);
#pragma unroll
            for (int u = 0; u < 16; ++u) t[u] = tn[u];
        }
        a0[(size_t)i * nc + i] = row;
        return;
    }
    const int nl = s_nl, ft = tid - 32;
    constexpr int FT = A0_T - 32;
    // a part per thread; more than FT parts take further rounds over the rows
    for (int x0 = 0; x0 < nl; x0 += FT) {
        const int jj = x0 + ft < nl ? list[x0 + ft] : -1;
        const double c_j = jj >= 0 ? cscale[jj] : 0.0;
        double row = 0.0;
        for (int b = 0; b < nb; b += A0_CH) {
            const int nr = min(A0_CH, nb - b);
            for (int t = ft; t < nr * 8; t += FT) {  // eight threads a row
                const int r = t >> 3, u = t & 7;
                const int k = owned[rows[q0 + b + r]];
                const int e0 = rp[k], n = rp[k + 1] - e0;
                if (u == 0) {
                    s_n[r] = n;
                    s_e[r] = e0;
                }
                if (n <= A0_W)
                    for (int e = u; e < n; e += 8) {
                        s_p[r][e] = part[ci[e0 + e]];
                        s_v[r][e] = v[e0 + e];
                    }
            }
            a0_sync();
            // the rows' terms: at the first entry of each other part, c_i
            // times the sum of the row's entries in it; a row's terms are put
            // one after another, in its order (most rows have one: a fold over
            // all seven entries of a row was most of this kernel's time)
            for (int t = ft; t < A0_CH * 8; t += FT) {
                const int r = t >> 3, u = t & 7, n = r < nr ? s_n[r] : 0;
                const unsigned group = 0xffu << (lane & 24);
                if (n > A0_W) continue;
                int base = 0;
                for (int e = u; e - u < n; e += 8) {
                    const int p = e < n ? s_p[r][e] : i;
                    bool first = p != i;
                    for (int d = 0; d < e && first; ++d) first = s_p[r][d] != p;
                    double acc = 0.0;
                    if (first) {
                        const double c = cscale[p];
                        for (int d = e; d < n; ++d)
                            if (s_p[r][d] == p) acc = __dadd_rn(acc, __dmul_rn(s_v[r][d], c));
                    }
                    const unsigned m = __ballot_sync(group, first) & group;
                    if (first) {
                        const int at = base + __popc(m & ((1u << lane) - 1u));
                        s_t[r][at] = __dmul_rn(c_i, acc);
                        s_q[r][at] = p;
                    }
                    base += __popc(m);
                }
                if (u == 0) s_c[r] = base;
            }
            a0_sync();
            if (jj >= 0) {
                for (int r0 = 0; r0 < nr; r0 += 4) {
                    int n[4], c[4], q[4];
                    double t[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {  // four rows' first terms in flight
                        n[u] = r0 + u < nr ? s_n[r0 + u] : 0;
                        c[u] = r0 + u < nr ? s_c[r0 + u] : 0;
                        q[u] = s_q[r0 + u][0];
                        t[u] = s_t[r0 + u][0];
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int r = r0 + u;
                        if (n[u] <= A0_W) {
                            if (c[u] > 0 && q[u] == jj) row = __dadd_rn(row, t[u]);
                            for (int e = 1; e < c[u]; ++e)
                                if (s_q[r][e] == jj) row = __dadd_rn(row, s_t[r][e]);
                            continue;
                        }
                        double acc = 0.0;
                        bool any = false;
                        for (int e = s_e[r]; e < s_e[r] + n[u]; ++e) {
                            if (part[ci[e]] != jj) continue;
                            acc = __dadd_rn(acc, __dmul_rn(v[e], c_j));
                            any = true;
                        }
                        if (any) row = __dadd_rn(row, __dmul_rn(c_i, acc));
                    }
                }
            }
            a0_sync();
        }
        if (jj >= 0) a0[(size_t)i * nc + jj] = row;
    }
}

// Dense LU with partial pivoting (src/precond/coarse_solve.h:15-47: first
// strictly larger magnitude, full row swaps, rounded ops in order), LU_NB
// columns at a time.  Every entry is updated by the same columns in the same
// order with the same two roundings wherever it is computed, so the factors do
// not depend on the blocking, bit for bit.
//
// The n^3 / 3 multiplications and subtractions bound it, on FP64 pipes of two
// lanes a cycle and SM: in one CTA they alone are 2.9 ms at n = 256.  Only a
// panel's columns need the pivots one by one and stay in one CTA (a thread a
// row, the panel in shared memory, magnitudes compared as integers, which
// leave the FP64 pipe alone); the rest is spread over the GPU.  One CTA
// for all: 0.29 ms at n = 64, 4.28 at 256; now 0.23 and 1.13.
constexpr int LU_NB = 16;
constexpr int LU_T = 512;
constexpr int LU_LD = LU_NB + 1;  // row stride of a panel in shared memory
__global__ void __launch_bounds__(LU_T)
k_lu_panel(int n, int k0, int in_smem, double* A, int* piv, int* status) {
    extern __shared__ __align__(16) unsigned char lu_raw[];
    __shared__ unsigned long long s_val[LU_T / 32];
    __shared__ int s_idx[LU_T / 32];
    if (*status) return;
    const int rows = n - k0, nb = min(LU_NB, rows), T = blockDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* P = in_smem ? reinterpret_cast<double*>(lu_raw) : A + (size_t)k0 * n + k0;
    const size_t ld = in_smem ? LU_LD : n;
    if (in_smem) {
        for (int t = tid; t < rows * LU_NB; t += T) {
            const int r = t / LU_NB, c = t % LU_NB;
            if (c < nb) P[r * ld + c] = A[(size_t)(k0 + r) * n + k0 + c];
        }
        __syncthreads();
    }
    for (int k = 0; k < nb; ++k) {
        unsigned long long bv = 0;  // 1 + the bits of |a|, ordered as |a|; 0 for NaN
        int bi = n;
        auto better = [&](unsigned long long a, int i) {
            if (a > bv || (a == bv && i < bi)) {
                bv = a;
                bi = i;
            }
        };
        for (int r = k + tid; r < rows; r += T) {
            const unsigned long long a =
                (unsigned long long)__double_as_longlong(P[r * ld + k]) & 0x7fffffffffffffffull;
            if (a <= 0x7ff0000000000000ull) better(a + 1, r);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            better(__shfl_xor_sync(0xffffffffu, bv, o), __shfl_xor_sync(0xffffffffu, bi, o));
        if (lane == 0) {
            s_val[warp] = bv;
            s_idx[warp] = bi;
        }
        __syncthreads();
        for (int w = 0; w < T / 32; ++w) better(s_val[w], s_idx[w]);
        if (bv < 1 + (unsigned long long)__double_as_longlong(1e-30)) {  // in every thread alike
            if (tid == 0) *status = 1;
            return;
        }
        if (tid == 0) piv[k0 + k] = k0 + bi;
        if (bi != k && tid < nb) {
            const double t = P[k * ld + tid];
            P[k * ld + tid] = P[bi * ld + tid];
            P[bi * ld + tid] = t;
        }
        __syncthreads();
        const double d = P[k * ld + k];
        for (int r = k + 1 + tid; r < rows; r += T) {
            const double l = P[r * ld + k] / d;
            P[r * ld + k] = l;
            for (int c = k + 1; c < nb; c += 4) {  // four at a time: their latencies overlap
                double a[4], u[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    a[e] = c + e < nb ? P[r * ld + c + e] : 0.0;
                    u[e] = c + e < nb ? P[k * ld + c + e] : 0.0;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) a[e] = __dsub_rn(a[e], __dmul_rn(l, u[e]));
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c + e < nb) P[r * ld + c + e] = a[e];
            }
        }
        __syncthreads();
    }
    if (in_smem)
        for (int t = tid; t < rows * LU_NB; t += T) {
            const int r = t / LU_NB, c = t % LU_NB;
            if (c < nb) A[(size_t)(k0 + r) * n + k0 + c] = P[r * ld + c];
        }
}

// The panel's row swaps in the other columns, a thread a column, and on its
// right the panel rows of U.  A thread reads and writes its own column only.
constexpr int LU_CT = 32;
__global__ void __launch_bounds__(LU_CT)
k_lu_rows(int n, int k0, double* A, const int* __restrict__ piv, const int* __restrict__ status) {
    __shared__ double l[LU_NB][LU_NB];
    __shared__ double u[LU_NB][LU_CT];
    if (*status) return;
    const int nb = min(LU_NB, n - k0), tid = threadIdx.x;
    const int q = blockIdx.x * LU_CT + tid, j = q < k0 ? q : q + nb;  // columns outside the panel
    for (int t = tid; t < LU_NB * LU_NB; t += LU_CT) {
        const int r = t / LU_NB, c = t % LU_NB;
        l[r][c] = r < nb && c < nb ? A[(size_t)(k0 + r) * n + k0 + c] : 0.0;
    }
    __syncthreads();
    if (j >= n) return;
#pragma unroll
    for (int k = 0; k < LU_NB; ++k) u[k][tid] = k < nb ? A[(size_t)(k0 + k) * n + j] : 0.0;
    for (int k = 0; k < nb; ++k) {
        const int r = piv[k0 + k];
        double* p = r < k0 + nb ? &u[r - k0][tid] : &A[(size_t)r * n + j];
        const double t = *p;
        *p = u[k][tid];
        u[k][tid] = t;
    }
    double x[LU_NB];
#pragma unroll
    for (int k = 0; k < LU_NB; ++k) x[k] = u[k][tid];
    if (j >= k0 + nb) {
#pragma unroll
        for (int k = 0; k < LU_NB; ++k)
#pragma unroll
            for (int i = k + 1; i < LU_NB; ++i) x[i] = __dsub_rn(x[i], __dmul_rn(l[i][k], x[k]));
    }
#pragma unroll
    for (int k = 0; k < LU_NB; ++k)
        if (k < nb) A[(size_t)(k0 + k) * n + j] = x[k];
}

// The rows and columns after the panel: 16 x 16 tiles, an entry a thread.
__global__ void __launch_bounds__(256)
k_lu_update(int n, int k0, double* A, const int* __restrict__ status) {
    __shared__ double l[LU_NB][LU_NB + 1];
    __shared__ double u[LU_NB][LU_NB];
    if (*status) return;
    const int tx = threadIdx.x % LU_NB, ty = threadIdx.x / LU_NB;
    const int r = k0 + LU_NB + blockIdx.y * LU_NB + ty, c = k0 + LU_NB + blockIdx.x * LU_NB + tx;
    const bool in = r < n && c < n;
    l[ty][tx] = r < n ? A[(size_t)r * n + k0 + tx] : 0.0;
    u[ty][tx] = c < n ? A[(size_t)(k0 + ty) * n + c] : 0.0;
    double a = in ? A[(size_t)r * n + c] : 0.0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < LU_NB; ++k) a = __dsub_rn(a, __dmul_rn(l[ty][k], u[k][tx]));
    if (in) A[(size_t)r * n + c] = a;
}

// Column t of A0^{-1} from the LU factors (one CTA per column): pivots and
// forward elimination as src/precond/coarse_solve.h:50-67, backward
// substitution by columns.
__global__ void __launch_bounds__(256) k_inv(int n, const double* __restrict__ L,
                                             const int* __restrict__ piv, double* inv) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* x = reinterpret_cast<double*>(smraw);
    const int t = blockIdx.x;
    for (int i = threadIdx.x; i < n; i += blockDim.x) x[i] = (i == t) ? 1.0 : 0.0;
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        if (threadIdx.x == 0 && piv[k] != k) {
            const double tmp = x[k];
            x[k] = x[piv[k]];
            x[piv[k]] = tmp;
        }
        __syncthreads();
        const double xk = x[k];
        for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x)
            x[i] = __dsub_rn(x[i], __dmul_rn(L[(size_t)i * n + k], xk));
        __syncthreads();
    }
    for (int k = n - 1; k >= 0; --k) {
        if (threadIdx.x == 0) x[k] = x[k] / L[(size_t)k * n + k];
        __syncthreads();
        const double xk = x[k];
        for (int i = threadIdx.x; i < k; i += blockDim.x)
            x[i] = __dsub_rn(x[i], __dmul_rn(L[(size_t)i * n + k], xk));
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) inv[(size_t)i * n + t] = x[i];
}

// r0[s] = c_s * sum of x over the owned rows of s
template <class TI>
__global__ void __launch_bounds__(1024)
k_restrict(const int* __restrict__ owned_ptr, const int* __restrict__ owned,
           const double* __restrict__ cscale, const TI* __restrict__ x, double* r0,
           const int* __restrict__ active) {
    if (active && *active == 0) return;
    __shared__ double red[RC_MAXCH];
    const int s = blockIdx.x;
    const int q0 = owned_ptr[s], q1 = owned_ptr[s + 1];
    const double z = restrict_chunks<TI>(owned + q0, x, q1 - q0, red);
    if (threadIdx.x == 0) r0[s] = cscale[s] * z;
}

template <class T>
T* dev_ptr(DBuf<T>& b) {
    return b.p;
}

template <class TS, class TF, class TC, class TI, class TO>
void sweep_launch(sg_precond* pc, const TF* lval, const TF* uval, const TF* udiag, const TI* x,
                  TO* y, int mode, bool coarse, const int* active, TS* gscratch) {
    sg_ctx* ctx = pc->ctx;
    // every buffer the kernel dereferences must exist (host-side guard)
    if (!pc->info.p || !pc->order.p || !pc->dofs.p || !pc->perm_f.p || !pc->perm_b.p ||
        !pc->lev_ptr_f.p || !pc->lev_ptr_b.p || !pc->lcol.p || !pc->ucol.p || !lval || !uval ||
        !udiag || !pc->ownloc_d.p || !pc->owned_d.p || (!pc->use_smem && !gscratch) ||
        (coarse && (!pc->a0inv.p || !pc->r0.p)))
        fail(SG_ERR_INTERNAL, "preconditioner device buffers missing for this apply");
    size_t smem = 0;
    if (pc->use_smem) {
        smem = ((size_t)(pc->max_n + 1) * sizeof(TS) + 15) & ~(size_t)15;
        allow_smem(ctx, k_sweep<TI, TO, TS, TF, TC>);
    }
    k_sweep<TI, TO, TS, TF, TC><<<pc->nparts, SWEEP_T, smem, ctx->stream>>>(
        pc->info.p, pc->order.p, pc->dofs.p, reinterpret_cast<const TC*>(pc->perm_f.p),
        pc->lev_ptr_f.p, reinterpret_cast<const TC*>(pc->lcol.p), lval,
        reinterpret_cast<const TC*>(pc->perm_b.p), pc->lev_ptr_b.p,
        reinterpret_cast<const TC*>(pc->ucol.p), uval, udiag, pc->ownloc_d.p, pc->owned_d.p,
        x, y, mode, coarse ? 1 : 0, pc->a0inv.p, pc->r0.p, pc->nc, gscratch,
        pc->use_smem ? 1 : 0, active, pc->sub_on);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

size_t sf_smem(const sg_precond* pc) {
    const size_t ts = pc->opts.sweep_dtype == SG_FP64 ? 8 : 4;
    return (((size_t)(pc->max_n + 1) * ts + 15) & ~(size_t)15) + (size_t)pc->max_n + 16;
}

template <class TS, class TF, class TC, bool EXACT, class TI, class TO>
void sf_launch(sg_precond* pc, const TF* lval, const TF* uval, const TF* udiag, const TI* x,
               TO* y, int mode, bool coarse, const int* active) {
    sg_ctx* ctx = pc->ctx;
    if (!pc->info.p || !pc->order.p || !pc->dofs.p || !pc->perm_f.p || !pc->perm_b.p ||
        !pc->lcol.p || !pc->ucol.p || !lval || !uval || !udiag || !pc->ownloc_d.p ||
        !pc->owned_d.p || !pc->err_d.p || (coarse && (!pc->a0inv.p || !pc->r0.p)))
        fail(SG_ERR_INTERNAL, "preconditioner device buffers missing for this apply");
    const size_t smem = sf_smem(pc);
    allow_smem(ctx, k_sweep_sf<TI, TO, TS, TF, TC, EXACT>);
    k_sweep_sf<TI, TO, TS, TF, TC, EXACT><<<pc->nparts, SWEEP_T, smem, ctx->stream>>>(
        pc->info.p, pc->order.p, pc->dofs.p, reinterpret_cast<const TC*>(pc->perm_f.p),
        reinterpret_cast<const TC*>(pc->lcol.p), lval, reinterpret_cast<const TC*>(pc->perm_b.p),
        reinterpret_cast<const TC*>(pc->ucol.p), uval, udiag, pc->ownloc_d.p, pc->owned_d.p, x, y,
        mode, coarse ? 1 : 0, pc->a0inv.p, pc->r0.p, pc->nc, pc->err_d.p, active, pc->sub_on);
    SG_CUDA(cudaGetLastError());
    count_launch(ctx);
}

template <class TC, class TI, class TO>
bool sf_dispatch(sg_precond* pc, const TI* x, TO* y, int mode, bool coarse, bool exact,
                 const int* active) {
    if (!pc->use_sf) return false;
    if (pc->opts.sweep_dtype == SG_FP64) {
        if (exact)
            sf_launch<double, double, TC, true>(pc, pc->lval64.p, pc->uval64.p, pc->udiag64.p, x, y,
                                                mode, coarse, active);
        else
            sf_launch<double, double, TC, false>(pc, pc->lval64.p, pc->uval64.p, pc->udiag64.p, x,
                                                 y, mode, coarse, active);
    } else if (pc->opts.factor_dtype == SG_BF16) {
        sf_launch<float, uint16_t, TC, false>(pc, pc->lval16.p, pc->uval16.p, pc->udiag16.p, x, y,
                                              mode, coarse, active);
    } else {
        sf_launch<float, float, TC, false>(pc, pc->lval32.p, pc->uval32.p, pc->udiag32.p, x, y,
                                           mode, coarse, active);
    }
    return true;
}

template <class TC, class TI, class TO>
void sweep_dispatch(sg_precond* pc, const TI* x, TO* y, int mode, bool coarse,
                    const int* active) {
    if (pc->opts.sweep_dtype == SG_FP64) {
        sweep_launch<double, double, TC>(pc, pc->lval64.p, pc->uval64.p, pc->udiag64.p, x, y, mode,
                                         coarse, active, pc->gscratch64.p);
    } else if (pc->opts.factor_dtype == SG_BF16) {
        sweep_launch<float, uint16_t, TC>(pc, pc->lval16.p, pc->uval16.p, pc->udiag16.p, x, y,
                                          mode, coarse, active, pc->gscratch32.p);
    } else {
        sweep_launch<float, float, TC>(pc, pc->lval32.p, pc->uval32.p, pc->udiag32.p, x, y, mode,
                                       coarse, active, pc->gscratch32.p);
    }
}

template <class TF, class TC>
void pack_launch(sg_precond* pc, TF* lval, TF* uval, TF* udiag) {
    k_pack<TF, TC><<<pc->nparts, SWEEP_T, 0, pc->ctx->stream>>>(
        pc->info.p, pc->lrp_d.p, pc->lci_d.p, pc->ldiag_d.p, pc->lu_d.p,
        reinterpret_cast<const TC*>(pc->perm_f.p), reinterpret_cast<const TC*>(pc->perm_b.p),
        reinterpret_cast<TC*>(pc->lcol.p), lval, reinterpret_cast<TC*>(pc->ucol.p), uval, udiag);
    SG_CUDA(cudaGetLastError());
}

// LU of the n x n matrix A in place, a panel at a time
void dense_lu(sg_ctx* ctx, int n, double* A, int* piv, int* status) {
    cudaStream_t st = ctx->stream;
    int max_smem = 0;
    SG_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
    // static scratch and the block's own kilobyte beside the panel; a panel of
    // more rows works in global memory
    const size_t room = (size_t)max_smem - 2048;
    allow_smem(ctx, k_lu_panel);
    for (int k0 = 0; k0 < n; k0 += LU_NB) {
        const int nb = std::min(LU_NB, n - k0), rest = n - k0 - nb;
        const size_t smem = (size_t)(n - k0) * LU_LD * sizeof(double);
        const bool fits = smem <= room;
        k_lu_panel<<<1, std::min(LU_T, (n - k0 + 31) & ~31), fits ? smem : 0, st>>>(n, k0, fits ? 1 : 0, A, piv, status);
        SG_CUDA(cudaGetLastError());
        if (n > nb) {
            k_lu_rows<<<(n - nb + LU_CT - 1) / LU_CT, LU_CT, 0, st>>>(n, k0, A, piv, status);
            SG_CUDA(cudaGetLastError());
        }
        if (rest > 0) {
            const unsigned t = (unsigned)(rest + LU_NB - 1) / LU_NB;
            k_lu_update<<<dim3(t, t), 256, 0, st>>>(n, k0, A, status);
            SG_CUDA(cudaGetLastError());
        }
    }
}

// the integer set-up's arrays -> device
void upload_structure(sg_precond* pc) {
    cudaStream_t st = pc->ctx->stream;
    pc->info.upload(pc->h_info, st);
    pc->order.upload(pc->h_order, st);
    pc->dofs.upload(pc->sub, st);
    pc->lev_ptr_f.upload(pc->h_lev_ptr_f, st);
    pc->lev_ptr_b.upload(pc->h_lev_ptr_b, st);
    pc->lrp_d.upload(pc->lrp, st);
    pc->lci_d.upload(pc->lci, st);
    pc->ldiag_d.upload(pc->ldiag, st);
    pc->lmap_d.upload(pc->lmap, st);
    pc->ownloc_d.upload(pc->ownloc, st);
    pc->owned_ptr_d.upload(pc->owned_ptr, st);
    pc->owned_d.upload(pc->owned, st);
    if (pc->wide_cols) {
        pc->perm_f.upload(reinterpret_cast<const uint16_t*>(pc->h_perm_f32.data()),
                          pc->h_perm_f32.size() * 2, st);
        pc->perm_b.upload(reinterpret_cast<const uint16_t*>(pc->h_perm_b32.data()),
                          pc->h_perm_b32.size() * 2, st);
    } else {
        pc->perm_f.upload(pc->h_perm_f16, st);
        pc->perm_b.upload(pc->h_perm_b16, st);
    }
}

template <class TC>
void factor_and_pack(sg_precond* pc, bool kept) {
    sg_ctx* ctx = pc->ctx;
    const bool whole = pc->nparts <= ctx->num_sms;
    auto* factor = whole ? k_factor<TC, FAC_T> : k_factor<TC, FAC_T / 2>;
    factor<<<pc->nparts, whole ? FAC_T : FAC_T / 2, 0, ctx->stream>>>(
        pc->info.p, pc->lrp_d.p, pc->lci_d.p, pc->ldiag_d.p,
        reinterpret_cast<const TC*>(pc->perm_f.p), pc->lev_ptr_f.p, pc->lu_d.p);
    SG_CUDA(cudaGetLastError());
    // sweep variants: TMA-fed level records (default), a barrier per level
    // with the factors read from global memory (reserved[0] = 1), sync-free
    // with per-row ready flags (reserved[0] = 4)
    const int variant = pc->opts.reserved[0];  // 0 TMA records, 1 level, 4 sync-free
    if (variant != 0) pc->use_rec = false;
    rec_setup_device(pc, kept);
    if (pc->use_rec) return;
    {
        int max_smem = 0;
        SG_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                       ctx->device));
        pc->use_sf = (variant & 4) && pc->use_smem && sf_smem(pc) + 1024 <= (size_t)max_smem;
    }
    if (!pc->err_d.p) {
        pc->err_d.alloc(1);
        if (!pc->err_h.p) pc->err_h.alloc(1);
        pc->err_d.zero(ctx->stream);
    }
    if (pc->wide_cols) {
        pc->lcol.alloc((size_t)pc->fl_total * 2);
        pc->ucol.alloc((size_t)pc->fu_total * 2);
    } else {
        pc->lcol.alloc((size_t)pc->fl_total);
        pc->ucol.alloc((size_t)pc->fu_total);
    }
    const size_t fl = (size_t)pc->fl_total, fu = (size_t)pc->fu_total, nr = (size_t)pc->total_rows;
    if (pc->opts.sweep_dtype == SG_FP64) {
        pc->lval64.alloc(fl); pc->uval64.alloc(fu); pc->udiag64.alloc(nr);
        pack_launch<double, TC>(pc, pc->lval64.p, pc->uval64.p, pc->udiag64.p);
    } else if (pc->opts.factor_dtype == SG_BF16) {
        pc->lval16.alloc(fl); pc->uval16.alloc(fu); pc->udiag16.alloc(nr);
        pack_launch<uint16_t, TC>(pc, pc->lval16.p, pc->uval16.p, pc->udiag16.p);
    } else {
        pc->lval32.alloc(fl); pc->uval32.alloc(fu); pc->udiag32.alloc(nr);
        pack_launch<float, TC>(pc, pc->lval32.p, pc->uval32.p, pc->udiag32.p);
    }
}

}  // namespace

// ---------------------------------------------------------------- set-up
void precond_setup_device(sg_precond* pc, const sg_csr* A) {
    sg_ctx* ctx = pc->ctx;
    cudaStream_t st = ctx->stream;
    const int n = A->nrows;
    if (pc->kind == SG_PC_NONE) return;
    if (pc->kind == SG_PC_JACOBI) {
        pc->inv_diag.alloc(n);
        pc->inv_diag32.alloc(n);
        k_jacobi_setup<<<ctx->num_sms * 4, 256, 0, st>>>(n, A->rp.p, A->ci.p, A->val.p,
                                                          pc->inv_diag.p, pc->inv_diag32.p);
        SG_CUDA(cudaGetLastError());
        return;
    }
    // ---- batched ILU(0): host structures -> device.  After a set-up of the
    // same structure they are there already, and every buffer has its size.
    // (Records laid out for values that needed the division are planned again.)
    const bool kept = pc->on_device && !pc->rec_divides;
    pc->on_device = false;
    auto reserve = [&](auto& b, size_t count) {
        if (!kept) b.alloc(count);
    };
    if (!kept) upload_structure(pc);
    const long long nz = (long long)pc->lci.size();
    reserve(pc->lu_d, (size_t)nz);
    k_gather_vals<<<ctx->num_sms * 4, 256, 0, st>>>(nz, pc->lmap_d.p, A->val.p, pc->lu_d.p);
    SG_CUDA(cudaGetLastError());
    if (pc->wide_cols) factor_and_pack<int>(pc, kept);
    else factor_and_pack<uint16_t>(pc, kept);
    if (!pc->use_smem && !pc->use_rec) {
        const size_t cnt = (size_t)pc->total_rows + (size_t)pc->nparts;
        if (pc->opts.sweep_dtype == SG_FP64) pc->gscratch64.alloc(cnt);
        else pc->gscratch32.alloc(cnt);
    }
    // ---- two-level coarse space
    if (pc->kind == SG_PC_TWOLEVEL_ASM || pc->kind == SG_PC_TWOLEVEL_RAS) {
        const int nc = pc->nparts;
        pc->nc = nc;
        if (!kept) {
            pc->part_d.upload(pc->part, st);
            pc->cscale_d.upload(pc->h_cscale, st);
        }
        reserve(pc->a0, (size_t)nc * nc);
        reserve(pc->lu0, (size_t)nc * nc);
        reserve(pc->a0inv, (size_t)nc * nc);
        reserve(pc->piv0, nc);
        reserve(pc->r0, nc);
        reserve(pc->status_d, 1);
        pc->status_d.zero(st);
        const size_t smem = (size_t)nc * (4 + 4);
        allow_smem(ctx, k_a0_build);
        reserve(pc->a0_own, (size_t)n);
        reserve(pc->a0_rows, (size_t)n);
        k_a0_build<<<nc, A0_T, smem, st>>>(nc, pc->owned_ptr_d.p, pc->owned_d.p, A->rp.p, A->ci.p,
                                           A->val.p, pc->part_d.p, pc->cscale_d.p, pc->a0_own.p,
                                           pc->a0_rows.p, pc->a0.p);
        SG_CUDA(cudaGetLastError());
        SG_CUDA(cudaMemcpyAsync(pc->lu0.p, pc->a0.p, sizeof(double) * nc * nc,
                                cudaMemcpyDeviceToDevice, st));
        dense_lu(ctx, nc, pc->lu0.p, pc->piv0.p, pc->status_d.p);
        int bad = 0;
        SG_CUDA(cudaMemcpyAsync(&bad, pc->status_d.p, sizeof(int), cudaMemcpyDeviceToHost, st));
        SG_CUDA(cudaStreamSynchronize(st));
        if (bad) fail(SG_ERR_SINGULAR, "Coarse matrix is singular");
        const size_t smem2 = (size_t)nc * 8;
        allow_smem(ctx, k_inv);
        k_inv<<<nc, 256, smem2, st>>>(nc, pc->lu0.p, pc->piv0.p, pc->a0inv.p);
        SG_CUDA(cudaGetLastError());
    }
    SG_CUDA(cudaStreamSynchronize(st));
    pc->on_device = true;
}

// ---------------------------------------------------------------- apply
template <class TI, class TO>
void precond_apply_device(sg_precond* pc, const TI* x, TO* y, const int* active, bool exact) {
    sg_ctx* ctx = pc->ctx;
    const int n = pc->n;
    const int grid = ctx->num_sms * 4;
    switch (pc->kind) {
    case SG_PC_NONE:
        launch_copy<TI, TO>(ctx, x, y, n, active);
        return;
    case SG_PC_HOST:
        host_precond_apply<TI, TO>(pc, x, y, active, nullptr);
        return;
    case SG_PC_JACOBI:
        if (pc->opts.sweep_dtype == SG_FP64)
            k_jacobi<TI, TO, double><<<grid, 256, 0, ctx->stream>>>(n, pc->inv_diag.p, x, y, active);
        else
            k_jacobi<TI, TO, float><<<grid, 256, 0, ctx->stream>>>(n, pc->inv_diag32.p, x, y, active);
        SG_CUDA(cudaGetLastError());
        count_launch(ctx);
        return;
    default:
        break;
    }
    const bool asm_mode = (pc->kind == SG_PC_ASM || pc->kind == SG_PC_TWOLEVEL_ASM);
    const bool coarse = (pc->kind == SG_PC_TWOLEVEL_ASM || pc->kind == SG_PC_TWOLEVEL_RAS);
    if (coarse) {
        if (!pc->owned_ptr_d.p || !pc->owned_d.p || !pc->cscale_d.p || !pc->r0.p)
            fail(SG_ERR_INTERNAL, "coarse-space device buffers missing");
        if (!sweep_fuses_restrict(pc)) {
            k_restrict<TI><<<pc->nc, 1024, 0, ctx->stream>>>(pc->owned_ptr_d.p, pc->owned_d.p,
                                                            pc->cscale_d.p, x, pc->r0.p, active);
            SG_CUDA(cudaGetLastError());
            count_launch(ctx);
        }
    }
    if (asm_mode) SG_CUDA(cudaMemsetAsync(y, 0, sizeof(TO) * (size_t)n, ctx->stream));
    if (sweep_tma<TI, TO>(pc, x, y, asm_mode ? 1 : 0, coarse, exact, active)) return;
    if (pc->wide_cols) {
        if (sf_dispatch<int, TI, TO>(pc, x, y, asm_mode ? 1 : 0, coarse, exact, active)) return;
    } else {
        if (sf_dispatch<uint16_t, TI, TO>(pc, x, y, asm_mode ? 1 : 0, coarse, exact, active))
            return;
    }
    if (pc->wide_cols) sweep_dispatch<int, TI, TO>(pc, x, y, asm_mode ? 1 : 0, coarse, active);
    else sweep_dispatch<uint16_t, TI, TO>(pc, x, y, asm_mode ? 1 : 0, coarse, active);
}

void precond_read_factors(sg_precond* pc, int s, double* lu_out) {
    const SubInfo& inf = pc->h_info[s];
    const int nnz = pc->lrp[inf.csr_row_off + inf.n];
    SG_CUDA(cudaMemcpyAsync(lu_out, pc->lu_d.p + inf.csr_nz_off, sizeof(double) * nnz,
                            cudaMemcpyDeviceToHost, pc->ctx->stream));
    SG_CUDA(cudaStreamSynchronize(pc->ctx->stream));
}

void precond_read_coarse(sg_precond* pc, double* a0_out) {
    SG_CUDA(cudaMemcpyAsync(a0_out, pc->a0.p, sizeof(double) * (size_t)pc->nc * pc->nc,
                            cudaMemcpyDeviceToHost, pc->ctx->stream));
    SG_CUDA(cudaStreamSynchronize(pc->ctx->stream));
}

template void precond_apply_device<double, double>(sg_precond*, const double*, double*,
                                                  const int*, bool);
template void precond_apply_device<double, float>(sg_precond*, const double*, float*,
                                                 const int*, bool);
template void precond_apply_device<float, float>(sg_precond*, const float*, float*, const int*,
                                                bool);

}  // namespace sg
