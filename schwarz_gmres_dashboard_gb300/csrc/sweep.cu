// sweep.cu -- the batched ILU(0) subdomain solve fed by TMA bulk copies.
//
// One CTA owns one subdomain (RAS/ASM, src/precond/ras.h:45-70,
// src/precond/asm.h:34-60).  The overlapped right-hand side is gathered into
// shared memory (the restriction that replaces the reference's MPI halo
// exchange), then the forward and backward sweeps of src/precond/ilu0.h:57-79
// run level by level: rows of one level are independent and a __syncthreads
// separates levels.
//
// A level's factor data is one contiguous, 16-byte-aligned record.  Rows with
// 2, 3 or 4 nonzeros per triangle (the 5-, 7- and 9-point stencils) are row
// structs [row slot, w column slots u16 | w values (| reciprocal diagonal)];
// other widths are stored by component,
//   [row slot u16 x C][column slot u16 x C x w][value x C x w](diagonal x C)
// (C = rows rounded up to 8).  A slot is the row's place in the shared-memory
// vector, tslot, whose per-subdomain padding keeps the rows of a level in
// distinct banks.  A subdomain's records form one stream (forward levels,
// then backward) that flows through a shared-memory byte ring in groups of
// whole levels: the block's last thread copies a group with one
// cp.async.bulk tracked by an mbarrier, as far ahead as the ring allows (at
// 128^3 all CTAs together stream ~120 MB of records per apply, so the copies
// need tens of KB in flight each).  Where each group lands in the ring and
// after which level it may be issued is a static schedule computed at
// set-up, which also checks that no level can wait for a copy not yet
// issued.  A level costs shared-memory latency plus one barrier; the width
// of the rows is a template parameter of each sweep direction's loop.  Every
// mbarrier wait is bounded (about one second of clock cycles); on expiry
// the CTA records an error word, waits (bounded again) for the copies it
// issued, and returns without touching the output.
#include <algorithm>
#include <type_traits>

#include "dev_common.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace sg {

namespace {

constexpr int SW_T = 512;
template <class TS, bool EXACT>
__device__ __forceinline__ TS sub_mul(TS acc, TS a, TS b);
template <>
__device__ __forceinline__ double sub_mul<double, true>(double acc, double a, double b) {
    return __dsub_rn(acc, __dmul_rn(a, b));
}
template <>
__device__ __forceinline__ double sub_mul<double, false>(double acc, double a, double b) {
    return fma(-a, b, acc);
}
template <>
__device__ __forceinline__ float sub_mul<float, true>(float acc, float a, float b) {
    return fmaf(-a, b, acc);
}
template <>
__device__ __forceinline__ float sub_mul<float, false>(float acc, float a, float b) {
    return fmaf(-a, b, acc);
}

template <class TF>
__device__ __forceinline__ TF to_factor(double v);
template <>
__device__ __forceinline__ double to_factor<double>(double v) { return v; }
template <>
__device__ __forceinline__ float to_factor<float>(double v) { return (float)v; }
template <>
__device__ __forceinline__ uint16_t to_factor<uint16_t>(double v) {
    return __bfloat16_as_ushort(__float2bfloat16_rn((float)v));
}

// ---- shared-memory accesses by 32-bit shared-window address.  The level
// loop's row updates are chains of dependent shared-memory loads; explicit
// 32-bit addressing keeps the address arithmetic between them short.
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
    return v;
}
template <class T>
__device__ __forceinline__ T lds(uint32_t a);
template <>
__device__ __forceinline__ float lds<float>(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
template <>
__device__ __forceinline__ double lds<double>(uint32_t a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
template <>
__device__ __forceinline__ uint16_t lds<uint16_t>(uint32_t a) {
    return (uint16_t)lds_u16(a);
}
__device__ __forceinline__ void sts(uint32_t a, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void sts(uint32_t a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// Records stored by component, any width w: a row computes acc = t[r]; acc -=
// v_k t[c_k] for k = 0..w-1 in order; backward: acc /= d.  The loads of four
// nonzeros at a time.
template <class TS, class TF, bool EXACT>
__device__ __forceinline__ void level_rows_any(TS* t, const unsigned char* R, int C, int c,
                                               int w, bool back, int nthreads) {
    const uint16_t* rr = reinterpret_cast<const uint16_t*>(R);
    const uint16_t* cc = rr + C;
    const TF* vv = reinterpret_cast<const TF*>(cc + (size_t)C * w);
    for (int q = threadIdx.x; q < c; q += nthreads) {
        const int r = rr[q];
        TS acc = t[r];
        for (int k0 = 0; k0 < w; k0 += 4) {
            int ci[4];
            TF vi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int o = (k0 + u < w ? k0 + u : k0) * C + q;
                ci[u] = cc[o];
                vi[u] = vv[o];
            }
            TS xi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) xi[u] = t[ci[u]];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k0 + u < w) acc = sub_mul<TS, EXACT>(acc, Load<TS>::f(vi[u]), xi[u]);
        }
        if (back) acc = div_diag(acc, Load<TS>::f(vv[w * C + q]));
        t[r] = acc;
    }
}

// Factored local CSR (FP64, reference layout) -> level records of type TF.
template <class TF>
__device__ __forceinline__ void put_recip(unsigned char* p, double d);
template <>
__device__ __forceinline__ void put_recip<double>(unsigned char* p, double d) {
    const double y = 1.0 / d;
    reinterpret_cast<double*>(p)[0] = y;
    reinterpret_cast<double*>(p)[1] = fma(-y, d, 1.0) * y;  // what rounding y left
    reinterpret_cast<double*>(p)[2] = d;
}
// |d| in [2^-300, 2^301): its quotients may be formed from the reciprocal
__device__ __forceinline__ bool recip_safe(double d) {
    return (unsigned)(((__double2hiint(d) >> 20) & 0x7ff) - 723) <= 600u;
}
template <>
__device__ __forceinline__ void put_recip<float>(unsigned char* p, double d) {
    *reinterpret_cast<float*>(p) = 1.0f / to_factor<float>(d);
}
template <>
__device__ __forceinline__ void put_recip<uint16_t>(unsigned char* p, double d) {
    *reinterpret_cast<float*>(p) = 1.0f / bf16_to_f(to_factor<uint16_t>(d));
}

// One level's record: the c rows of perm, then padding (component records up
// to C rows; row structs: the row that computes 0 in the unused slot).
template <class TF, bool BACK>
__device__ __forceinline__ void pack_level(const SubInfo& inf, const int* rp, const int* ci,
                                           const int* dg, const double* v, const uint16_t* perm,
                                           int c, int C, int w, bool rows, unsigned char* R,
                                           int* far) {
    constexpr int SF = (int)sizeof(TF);
    const uint16_t zero = (uint16_t)tslot(inf.n, inf.tshift);
    const int rb = rec_row_bytes(w, BACK, SF), vo = rec_val_off(w, SF);
    uint16_t* rr = reinterpret_cast<uint16_t*>(R);
    uint16_t* cc = rr + C;
    TF* vv = reinterpret_cast<TF*>(cc + (size_t)C * w);
    for (int q = threadIdx.x; q < (rows ? c + 1 : C); q += blockDim.x) {
        const int r = q < c ? perm[q] : 0;
        unsigned char* P = R + (size_t)q * rb;
        auto col = [&](int k) -> uint16_t& {
            return rows ? reinterpret_cast<uint16_t*>(P)[1 + k] : cc[(size_t)k * C + q];
        };
        auto val = [&](int k) -> TF& {
            return rows ? reinterpret_cast<TF*>(P + vo)[k] : vv[(size_t)k * C + q];
        };
        (rows ? reinterpret_cast<uint16_t*>(P)[0] : rr[q]) =
            q < c ? (uint16_t)tslot(r, inf.tshift) : (rows ? zero : (uint16_t)0);
        int k = 0;
        if (q < c) {
            for (int e = BACK ? dg[r] + 1 : rp[r]; e < rp[r + 1] && k < w; ++e) {
                const int cl = ci[e];
                if (!BACK && cl >= r) break;
                col(k) = (uint16_t)tslot(cl, inf.tshift);
                val(k) = to_factor<TF>(v[e]);
                ++k;
            }
        }
        for (; k < w; ++k) {
            col(k) = zero;
            val(k) = to_factor<TF>(0.0);
        }
        if (BACK) {
            const double d = q < c ? v[dg[r]] : 1.0;
            if (SF == 8 && rows && !recip_safe(d)) *far = 1;
            if (rows) put_recip<TF>(P + rec_recip_off(w, SF), d);
            else (vv + (size_t)C * w)[q] = to_factor<TF>(d);
        }
    }
}

// Block (s, y) packs every gridDim.y-th level of subdomain s: a row is a few
// dependent loads, so one block a subdomain waits most of its time (64
// subdomains of 64^3: 0.35 ms, with 16 blocks each 0.057).
template <class TF>
__global__ void __launch_bounds__(256)
k_pack_rec(const SubInfo* __restrict__ info, const int* __restrict__ lrp,
           const int* __restrict__ lci, const int* __restrict__ ldiag,
           const double* __restrict__ lu, const uint16_t* __restrict__ perm_f,
           const uint16_t* __restrict__ perm_b, const int* __restrict__ lev_f,
           const int* __restrict__ lev_b, const long long* __restrict__ off_f,
           const long long* __restrict__ off_b, const int* __restrict__ rows_f,
           const int* __restrict__ rows_b, int row_structs, unsigned char* rec, int* far) {
    const SubInfo inf = info[blockIdx.x];
    const int* rp = lrp + inf.csr_row_off;
    const int* ci = lci + inf.csr_nz_off;
    const double* v = lu + inf.csr_nz_off;
    const int* dg = ldiag + inf.row_off;
    const bool sf = row_structs && rec_is_rows(inf.wl), sb = row_structs && rec_is_rows(inf.wu);
    for (int l = blockIdx.y; l < inf.nlev_f; l += gridDim.y) {
        const int i = inf.lev_off_f + l, p0 = lev_f[i];
        pack_level<TF, false>(inf, rp, ci, dg, v, perm_f + inf.row_off + p0, lev_f[i + 1] - p0,
                              rows_f[i], inf.wl, sf, rec + off_f[i], far);
    }
    for (int l = blockIdx.y; l < inf.nlev_b; l += gridDim.y) {
        const int i = inf.lev_off_b + l, p0 = lev_b[i];
        pack_level<TF, true>(inf, rp, ci, dg, v, perm_b + inf.row_off + p0, lev_b[i + 1] - p0,
                             rows_b[i], inf.wu, sb, rec + off_b[i], far);
    }
}

// ---- R right-hand sides at once (FP32 sweeps): the shared vector holds R
// interleaved floats per slot, so every level record is read once for all of
// them; the row arithmetic per right-hand side is the single-vector code's.
template <int R>
struct FVec;
template <>
struct FVec<4> {
    __device__ __forceinline__ static void ld(uint32_t a, float (&v)[4]) {
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                     : "r"(a)
                     : "memory");
    }
    __device__ __forceinline__ static void st(uint32_t a, const float (&v)[4]) {
        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(v[0]), "f"(v[1]),
                     "f"(v[2]), "f"(v[3])
                     : "memory");
    }
};

// the component-wise records of any width w for R right-hand sides
template <bool BACK, class TF, int R>
__device__ __forceinline__ void level_rows_mr(uint32_t tb, uint32_t Rr, int C, int c, int w,
                                              int nthreads) {
    constexpr uint32_t SF = sizeof(TF), ST = 4u * R;
    const uint32_t cstride = 2u * (uint32_t)C;
    const uint32_t vbase = Rr + cstride * (uint32_t)(1 + w);
    const uint32_t vstride = SF * (uint32_t)C;
    for (int q = threadIdx.x; q < c; q += nthreads) {
        const uint32_t rq = Rr + 2u * (uint32_t)q;
        const uint32_t vq = vbase + SF * (uint32_t)q;
        const uint32_t r = lds_u16(rq);
        float acc[R];
        FVec<R>::ld(tb + ST * r, acc);
        for (int k = 0; k < w; ++k) {
            const uint32_t ci = lds_u16(rq + cstride * (uint32_t)(k + 1));
            const float v = Load<float>::f(lds<TF>(vq + vstride * (uint32_t)k));
            float xv[R];
            FVec<R>::ld(tb + ST * ci, xv);
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i] = fmaf(-v, xv[i], acc[i]);
        }
        if (BACK) {
            const float rd = 1.0f / Load<float>::f(lds<TF>(vq + vstride * (uint32_t)w));
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i] = acc[i] * rd;
        }
        FVec<R>::st(tb + ST * r, acc);
    }
}

// ---- row structs.  One struct of RB bytes holds everything a row reads
// besides the vector; its words are loaded together (16, 8 or 4 bytes at a
// time, whichever RB allows; every RB is conflict-free across a warp).
template <int W, bool BACK, class TF>
struct RowRec {
    static constexpr int SF = (int)sizeof(TF);
    static constexpr int RB = rec_row_bytes(W, BACK, SF);
    static constexpr int VO = rec_val_off(W, SF);
    static constexpr int DO = rec_recip_off(W, SF);
    static constexpr int NW = (BACK ? DO + (SF == 8 ? 24 : 4) : VO + W * SF + 3) / 4;  // words read
    uint32_t w[(NW + 3) / 4 * 4];

    __device__ __forceinline__ void load(uint32_t a) {
        if constexpr (RB % 16 == 0) {
#pragma unroll
            for (int i = 0; i < NW; i += 4)
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                             : "=r"(w[i]), "=r"(w[i + 1]), "=r"(w[i + 2]), "=r"(w[i + 3])
                             : "r"(a + 4u * i)
                             : "memory");
        } else if constexpr (RB % 8 == 0) {
#pragma unroll
            for (int i = 0; i < NW; i += 2)
                asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];"
                             : "=r"(w[i]), "=r"(w[i + 1])
                             : "r"(a + 4u * i)
                             : "memory");
        } else {
#pragma unroll
            for (int i = 0; i < NW; ++i)
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[i]) : "r"(a + 4u * i) : "memory");
        }
    }
    // slot k: the row (0) or column k - 1
    __device__ __forceinline__ uint32_t slot(int k) const {
        return (k & 1) ? w[k / 2] >> 16 : w[k / 2] & 0xffffu;
    }
    template <class TS>
    __device__ __forceinline__ TS value(int k) const {
        if constexpr (SF == 2) {
            const int h = VO / 2 + k;
            return (TS)__uint_as_float((h & 1) ? w[h / 2] & 0xffff0000u : w[h / 2] << 16);
        } else if constexpr (SF == 4) {
            return (TS)__uint_as_float(w[VO / 4 + k]);
        } else {
            return (TS)__hiloint2double((int)w[VO / 4 + 2 * k + 1], (int)w[VO / 4 + 2 * k]);
        }
    }
    // FP64 sweeps: i = 0 the reciprocal, 1 what rounding it left, 2 the diagonal
    template <class TS>
    __device__ __forceinline__ TS recip(int i) const {
        if constexpr (SF == 8)
            return (TS)__hiloint2double((int)w[DO / 4 + 2 * i + 1], (int)w[DO / 4 + 2 * i]);
        else
            return (TS)__uint_as_float(w[DO / 4]);
    }
};

// a / d rounded to nearest from y = 1 / d rounded to nearest: two corrected
// quotients (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", 1990).  a y is within two units in the last
// place, the first correction makes it faithful, and the last residual, exact
// in one fused multiply-add, rounds the quotient correctly -- five dependent
// operations where the division takes the time of seven and twice the FP64
// slots.  Outside the exponents where no residual can lose bits (and for
// infinities and NaN) the division itself; a zero keeps the sign of a y, but
// not where y overflowed (|d| < 2^-1024: 0 * inf is NaN, 0 / d is 0).
__device__ __noinline__ double div_plain(double a, double d) { return a / d; }
__device__ __forceinline__ double div_recip(double a, double d, double y) {
    const int ha = __double2hiint(a);
    const int ea = (ha >> 20) & 0x7ff, ed = (__double2hiint(d) >> 20) & 0x7ff;
    // also the lanes past a level's end
    const bool zero = ((ha << 1) | __double2loint(a)) == 0 &&
                      (__double2hiint(y) & 0x7ff00000) != 0x7ff00000;
    const double q0 = a * y;
    double q = fma(fma(-q0, d, a), y, q0);
    q = fma(fma(-q, d, a), y, q);
    if (zero) q = q0;
    const bool safe = (unsigned)(ea - 423) <= 1200u && (unsigned)(ed - 723) <= 600u;
    if (!safe && !zero) q = div_plain(a, d);  // a call: inlined, it would run for every row
    return q;
}

// ---- the gather and the restricted scatter of the TMA-fed sweep.  Rows are
// spread over the threads (consecutive rows on consecutive lanes, so index
// loads, element copies and stores stay coalesced) and each thread keeps
// SW_ILP index loads in flight: a cold gather or scatter of ~9,000 rows
// costs two or three memory round trips.  With R right-hand sides, element
// i of row li sits at x[i * ldx + dof[li]] and in slot component i.
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}
template <class T>
__device__ __forceinline__ void cp_async_elt(uint32_t dst, const T* src) {
    if constexpr (sizeof(T) == 8) cp_async8(dst, src);
    else cp_async4(dst, src);
}

constexpr int SW_ILP = 16;

// input of the sweep's own type: every element copied global -> shared by
// cp.async (no register holds a value, so all of a thread's copies stay in
// flight); the caller waits with cp_async_wait_all
template <class T, int R>
__device__ __forceinline__ void gather_async(uint32_t t_s, const T* __restrict__ x,
                                             long long ldx, const int* __restrict__ dof, int n,
                                             int bs, int p) {
    constexpr int U = sizeof(T) == 8 ? SW_ILP / 2 : SW_ILP;
    for (int li = threadIdx.x; li < n; li += U * bs) {
        int d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) d[u] = li + u * bs < n ? __ldg(dof + li + u * bs) : -1;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (d[u] >= 0) {
                const uint32_t slot = t_s + (uint32_t)(sizeof(T) * R * tslot(li + u * bs, p));
#pragma unroll
                for (int i = 0; i < R; ++i)
                    cp_async_elt<T>(slot + (uint32_t)(sizeof(T) * i), x + i * ldx + d[u]);
            }
    }
}

// other input types convert through registers
template <class TS, class TI, int R>
__device__ __forceinline__ void gather_convert(TS* t, const TI* __restrict__ x, long long ldx,
                                               const int* __restrict__ dof, int n, int bs, int p) {
    // values in flight per thread (U x R inputs held in registers)
    constexpr int U = R > 1 ? 2 : (sizeof(TI) == 8 ? 4 : 8);
    for (int li = threadIdx.x; li < n; li += U * bs) {
        int d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) d[u] = li + u * bs < n ? __ldg(dof + li + u * bs) : -1;
        TI v[U][R];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < R; ++i) v[u][i] = d[u] >= 0 ? x[i * ldx + d[u]] : (TI)0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (d[u] >= 0)
#pragma unroll
                for (int i = 0; i < R; ++i)
                    t[(size_t)R * tslot(li + u * bs, p) + i] = Load<TS>::f(v[u][i]);
    }
}

// y[i * ldy + og[q]] = t[tslot(ol[q])][i] (+ the coarse term), q < n_own
template <class TS, class TO, int R>
__device__ __forceinline__ void scatter_ilp(const TS* t, TO* __restrict__ y, long long ldy,
                                            const int* __restrict__ ol, const int* __restrict__ og,
                                            int n_own, int coarse, double zc, int bs, int p) {
    const CoarseAdd<TO> add(zc);
    constexpr int U = sizeof(TO) == 8 ? SW_ILP / 2 : SW_ILP;
    for (int q = threadIdx.x; q < n_own; q += U * bs) {
        int l[U], g[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = q + u * bs < n_own;
            l[u] = in ? __ldg(ol + q + u * bs) : -1;
            g[u] = in ? __ldg(og + q + u * bs) : 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (l[u] >= 0) {
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const TS v = t[(size_t)R * tslot(l[u], p) + i];
                    y[i * ldy + g[u]] = coarse ? add(v) : Store<TO>::f(v);
                }
            }
    }
}

// Static schedule of one subdomain's record stream through the ring: the
// stream (forward records, then backward, contiguous from `base` in the
// packed array) is cut into groups of whole levels of one direction, each
// copied by one cp.async.bulk into a fixed ring position and tracked by
// mbarrier (group % RING_NBAR).  Per group (int4): x = stream offset, y =
// bytes / 16 | ring position / 16 << 16, z = its first entry, w = the groups
// that may have been issued once it is done.  Per entry (int2), one pass over
// at most as many rows as the level threads take (component records: one entry
// a level): x = rows left of the level | 0x10000 when a barrier follows, y = the
// record's byte offset in the ring.  An entry of no rows ends a group.
struct RingSub {
    long long base;
    int ent_off, grp_off, nent, ngrp, ngrp_f, ninit;  // groups [0, ngrp_f) are forward
};
constexpr int RING_LOG_NBAR = 5;
constexpr int RING_NBAR = 1 << RING_LOG_NBAR;

struct RecArgs {
    const SubInfo* info;
    const int* order;
    const int* dofs;
    const RingSub* ring;
    const int2* ent;
    const int4* grp;
    const unsigned char* rec;
    const int* ownloc;
    const int* owned;
    const double* a0inv;
    const double* r0;
    int nparts;
    int nc;
    int a0pre;       // 1: the coarse row a0inv[s] is prefetched into shared memory
    int row_structs; // 1: levels of width 2 to 4 are row structs
    int ring_bytes;  // bytes of the record ring
    int t_len;       // slots of the subdomain vector region (largest tslot(n) + 1)
    int max_ent, max_grp;  // largest counts of schedule entries and groups
    int level_threads;     // threads of the level loop
    long long ldx, ldy;  // distance between right-hand sides (R > 1)
    int* err;
    // optional per-subdomain switches, one array of nparts per right-hand
    // side (0: skipped; a subdomain runs when any of its R switches is on)
    const int* sub_on;
    // persistent launch: CTAs take subdomains (in `order`) from work[0];
    // work[1] counts the CTAs that are done, and the last one resets both
    int persist;
    unsigned* work;
    // coarse restriction fused into the sweep (cooperative launch, all blocks
    // resident): each restriction is written to r0[s] and counted in sync[0];
    // sync[1] counts the subdomains done with r0 (the last one resets both).
    // Blocks from nparts on compute restrictions only.
    int fuse;
    double* r0w;
    unsigned* sync;
    // bounded waits: cycle budget of the record and restriction waits, and
    // the test mode that makes one of them run out without any fault
    // (1: record group 0 is never copied; 2: no restriction is counted)
    long long wait_budget;
    int wait_test;
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// The ring side of the level loop.  Set-up has checked that every group is
// issued (after the group its schedule names) before its first level waits
// for it, and that a group re-arms an mbarrier or overwrites ring bytes only
// after every thread has observed, and finished with, the group before it.
//
// A wait that gives up marks the thread (bad: it computes no more rows and
// waits for no further group) and the block (the shared word fail); a thread
// that finds the word set before a wait does the same without waiting.  All
// threads still pass every level's barrier, and the block gives up together
// after the last one.  No thread reads a group that it has not seen land.
struct RecRing {
    const unsigned char* src;
    const int4* grp;       // shared memory
    volatile int* fail;    // shared memory
    uint32_t bars_s, ring_s;
    long long budget;
    int gbase;     // groups this CTA streamed for earlier subdomains: group j
                   // of this one uses mbarrier (gbase + j) % RING_NBAR with
                   // phase parity ((gbase + j) / RING_NBAR) & 1
    int issued;    // producer: groups issued
    int observed;  // groups this thread has seen complete
    bool producer, bad;
    int wait_test;

    __device__ __forceinline__ uint32_t bar(int j) const {
        return bars_s + 8u * (uint32_t)((gbase + j) & (RING_NBAR - 1));
    }
    __device__ __forceinline__ uint32_t parity(int j) const {
        return (uint32_t)((gbase + j) >> RING_LOG_NBAR) & 1u;
    }
    __device__ __forceinline__ void issue_to(int limit) {
        if (issued >= limit || *fail != 0) return;
        fence_proxy_async();  // the ring bytes it overwrites were read by the generic proxy
        do {
            const int4 gi = grp[issued];
            const uint32_t bytes = ((uint32_t)gi.y & 0xffffu) << 4;
            const uint32_t pos = ((uint32_t)gi.y >> 16) << 4;
            if (!(wait_test == 1 && issued == 0)) {
                mbar_expect_tx(bar(issued), bytes);
                bulk_g2s_stream(ring_s + pos, src + (uint32_t)gi.x, bytes, bar(issued));
            }
        } while (++issued < limit);
    }
    // whether group j has landed (one probe, no wait)
    __device__ __forceinline__ bool landed(int j) const { return mbar_try(bar(j), parity(j)); }
    // this thread's first access to group j: the first try costs one mbarrier
    // probe; the bounded loop (which reads the clock) runs only when the copy
    // has not landed yet
    __device__ __forceinline__ void open(int j) {
        if (bad) return;
        if (*fail == 0 && (landed(j) || mbar_wait(bar(j), parity(j), budget))) {
            observed = j + 1;
        } else {
            bad = true;
            *fail = 1;
        }
    }
    // the block leaves after a wait gave up: the producer waits (full budget
    // each) for the copies it issued that it has not seen land, so none
    // lands after the block has left; if one still does not arrive -- only
    // possible when a copy never lands at all -- the error word says 2
    __device__ void drain(int* err) const {
        if (!producer) return;
        int code = 1;
        for (int k = observed; k < issued; ++k) {
            if (wait_test == 1 && k == 0) continue;
            if (!mbar_wait(bar(k), parity(k), WAIT_CYCLES)) code = 2;
        }
        atomicMax(err, code);
    }
};

// barrier among the NC level threads
__device__ __forceinline__ void level_sync(int NC) {
    asm volatile("bar.sync 1, %0;" ::"r"(NC) : "memory");
}

// One sweep direction over component-wise records: groups [j0, j1), any
// width w.  Per group the wait for its copy, then per level the rows and one
// barrier, then the producer issues the groups the schedule allows.
template <bool BACK, class TS, class TF, bool EXACT, int R>
__device__ __forceinline__ void level_loop_any(const int2* ent, int j0, int j1, int w,
                                               RecRing& ring, TS* t, uint32_t t_s,
                                               unsigned char* ring_g, int NC) {
    for (int j = j0; j < j1; ++j) {
        ring.open(j);
        const int e1 = ring.grp[j + 1].z - 1;
        for (int e = ring.grp[j].z; e < e1; ++e) {
            const int2 md = ent[e];
            if (!ring.bad) {
                const int c = md.x & 0xffff, C = (c + 7) & ~7;
                if constexpr (R > 1)
                    level_rows_mr<BACK, TF, R>(t_s, ring.ring_s + (uint32_t)md.y, C, c, w, NC);
                else
                    level_rows_any<TS, TF, EXACT>(t, ring_g + md.y, C, c, w, BACK, NC);
            }
            level_sync(NC);
        }
        if (ring.producer) ring.issue_to(ring.grp[j].w);
    }
}

// One sweep direction over row structs of W nonzeros, groups [j0, j1).  The
// time of a level is a chain of latencies -- shared loads, multiply-adds, the
// barrier (a dependent FP64 multiply-add takes ~75 cycles here, a division
// ~560) -- so everything that does not depend on the previous level is taken
// out of it, and the loop over a group's levels is straight-line predicated
// code (a divergent branch or an inner loop costs 40 to 80 cycles a level):
//  * a thread loads the struct of its next row before the barrier, between
//    the loads of this level's vector elements and their first use;
//  * the diagonal comes as its reciprocal.  Exact FP64 sweeps round the quotient
//    correctly with it (div_recip); the solver's take the reciprocal in two
//    parts, a / d = fma(a, y, a y2) (N. Brisebarre, J.-M. Muller, S. K. Raina,
//    "Accelerating correctly rounded floating-point division when the divisor
//    is known in advance", 2004): within 2^-104 of the quotient before its one
//    rounding (2.4 10^9 random and hard quotients all equal the division; a y
//    alone is another number for 26% of them).  One operation deeper than a y:
//    solves of 100 x 100 in 4 parts 12.7 -> 13.6 ms, 64^3 in 64 18.1 -> 19.2;
//  * the lanes past a level's end take the row that computes 0 in the unused
//    slot, so no store is conditional within a warp;
//  * a level of more rows than the threads take is several entries of the
//    schedule;
//  * of R interleaved right-hand sides a thread takes one, R neighbouring lanes
//    a row (their struct loads are one broadcast): a level of the small
//    subdomains that are solved in batches has ~20 rows, and a thread with all
//    four spent ~350 cycles a level issuing their multiply-adds.
// Cycles per level in isolation, component records with the row's loads after
// the barrier -> this loop: 51 x 51 FP32 223 -> 104, 15^3 FP32 288 -> 165;
// 51 x 51 FP64 354 forward, 995 backward -> 214, 270; 14^3 FP64 481, 1159 ->
// 414, 519 (backward with a y; with its second part ~80 more, by the solves
// above).  Warps without rows still take the predicated FP64 instructions'
// slots of the narrow FP64 pipe, so FP64 sweeps either run their levels on few
// warps (270 cycles with 2 warps, 507 with 8) or, with FP64_SKIP threads or
// more, branch around the level in warps that have no rows (SKIP: 350 cycles
// with 8 warps, and a level of many rows takes fewer passes).
constexpr int FP64_SKIP = 256;
template <int W, bool BACK, class TS, class TF, bool EXACT, int R, bool SKIP>
__device__ __forceinline__ void level_loop(const int2* ent, int j0, int j1, RecRing& ring,
                                           uint32_t t_s, int NC) {
    using Row = RowRec<W, BACK, TF>;
    constexpr uint32_t ST = (uint32_t)(sizeof(TS) * R);
    const int q = threadIdx.x / R;  // this thread's row of a pass
    t_s += (uint32_t)sizeof(TS) * (threadIdx.x % R);
    for (int j = j0; j < j1; ++j) {
        ring.open(j);
        // first row of this warp
        const int wid = ring.bad ? 1 << 30 : ((int)threadIdx.x & ~31) / R;
        int e = ring.grp[j].z;
        const int e1 = ring.grp[j + 1].z - 1;
        int2 md = ent[e], mn = ent[e + 1];
        int c = md.x & 0xffff, sync = md.x >> 16;
        uint32_t a = ring.ring_s + (uint32_t)(md.y + Row::RB * min(q, c));
        bool on = wid < c;
        Row row;
        if (on) row.load(a);
        for (; e < e1; ++e) {
            if (SKIP && !on && !(wid < (mn.x & 0xffff))) {  // nothing here, nothing to load
                const int f = sync;
                md = mn;
                sync = md.x >> 16;
                mn = ent[e + 2];
                if (f) level_sync(NC);
                continue;
            }
            const bool cur = on;
            const int f = sync;
            uint32_t ar = 0;
            TS xk[W], acc, vk[W], rd = (TS)1, dg = (TS)1;
            if (cur) {
                ar = t_s + ST * row.slot(0);
#pragma unroll
                for (int k = 0; k < W; ++k) xk[k] = lds<TS>(t_s + ST * row.slot(k + 1));
                acc = lds<TS>(ar);
#pragma unroll
                for (int k = 0; k < W; ++k) vk[k] = row.template value<TS>(k);
                if (BACK) rd = row.template recip<TS>(0);
                if (BACK && sizeof(TS) == 8) dg = row.template recip<TS>(EXACT ? 2 : 1);
            }
            md = mn;
            c = md.x & 0xffff;
            sync = md.x >> 16;
            a = ring.ring_s + (uint32_t)(md.y + Row::RB * min(q, c));
            on = wid < c;
            mn = ent[e + 2];
            if (on) row.load(a);
            if (cur) {
#pragma unroll
                for (int k = 0; k < W; ++k) acc = sub_mul<TS, EXACT>(acc, vk[k], xk[k]);
                if (BACK) {
                    if constexpr (EXACT && sizeof(TS) == 8) acc = div_recip(acc, dg, rd);
                    else if constexpr (sizeof(TS) == 8) acc = fma(acc, rd, acc * dg);
                    else acc = acc * rd;
                }
                sts(ar, acc);
            }
            if (f) level_sync(NC);
        }
        if (ring.producer) ring.issue_to(ring.grp[j].w);
    }
}

template <bool BACK, class TS, class TF, bool EXACT, int R>
__device__ __forceinline__ void level_loop_w(const int2* ent, int j0, int j1, int w, bool rows,
                                             RecRing& ring, TS* t, uint32_t t_s,
                                             unsigned char* ring_g, int NC) {
    if constexpr (sizeof(TS) == 8) {
        if (rows && rec_is_rows(w) && NC >= FP64_SKIP) {
            if (w == 2) level_loop<2, BACK, TS, TF, EXACT, R, true>(ent, j0, j1, ring, t_s, NC);
            else if (w == 3) level_loop<3, BACK, TS, TF, EXACT, R, true>(ent, j0, j1, ring, t_s, NC);
            else level_loop<4, BACK, TS, TF, EXACT, R, true>(ent, j0, j1, ring, t_s, NC);
            return;
        }
    }
    switch (rows ? w : 0) {
    case 2: return level_loop<2, BACK, TS, TF, EXACT, R, false>(ent, j0, j1, ring, t_s, NC);
    case 3: return level_loop<3, BACK, TS, TF, EXACT, R, false>(ent, j0, j1, ring, t_s, NC);
    case 4: return level_loop<4, BACK, TS, TF, EXACT, R, false>(ent, j0, j1, ring, t_s, NC);
    default:
        return level_loop_any<BACK, TS, TF, EXACT, R>(ent, j0, j1, w, ring, t, t_s, ring_g, NC);
    }
}

// The shared memory of one CTA of the sweep.
struct SweepSmem {
    unsigned char* raw;   // RING_NBAR mbarriers, then the ring
    unsigned char* ring;  // ring_bytes
    void* t;              // t_len slots of R elements
    int4* grp;            // max_grp + 1
    int2* ent;            // max_ent
    double* a0row;        // nc (a0pre)
};

// The coarse restriction of subdomain s (the order of k_restrict), published
// for the blocks that add the coarse term.
template <class TI>
__device__ __forceinline__ void publish_restriction(const RecArgs& a, int s, const SubInfo& inf,
                                                    const TI* __restrict__ x, double* red) {
    const double z = restrict_chunks<TI>(a.owned + inf.own_off, x, inf.n_own, red);
    if (threadIdx.x == 0) {
        a.r0w[s] = inf.cscale * z;
        __threadfence();
        if (a.wait_test != 2) atomicAdd(&a.sync[0], 1u);
    }
}

// One subdomain: stage its schedule, start its record stream, gather its
// right-hand side(s) (and, in the fused two-level mode, the coarse
// restrictions this block owes), run both sweeps, add the coarse term and
// write the owned rows.  Returns false when the block must leave (a bounded
// wait gave up; the error word is set).
template <class TI, class TO, class TS, class TF, bool EXACT, int R>
__device__ __forceinline__ bool sweep_one(const RecArgs& a, int s, const TI* __restrict__ x,
                                          TO* __restrict__ y, int mode, int coarse,
                                          const SweepSmem& sm, int& gbase, bool first) {
    __shared__ double s_zc;
    __shared__ double s_red[RC_MAXCH];
    __shared__ int s_ok;
    __shared__ int s_fail;
    const int NC = (int)blockDim.x;
    TS* t = reinterpret_cast<TS*>(sm.t);
    const SubInfo inf = a.info[s];
    const RingSub rs = a.ring[s];
    const int n = inf.n;
    // the schedule, staged once (the level loop touches global memory only
    // through the ring)
    for (int e = threadIdx.x; e < rs.nent; e += NC) sm.ent[e] = a.ent[rs.ent_off + e];
    for (int j = threadIdx.x; j <= rs.ngrp; j += NC) sm.grp[j] = a.grp[rs.grp_off + j];

    RecRing ring;
    ring.src = a.rec + rs.base;
    ring.grp = sm.grp;
    ring.bars_s = smem_u32(sm.raw);
    ring.ring_s = smem_u32(sm.ring);
    ring.budget = a.wait_budget;
    ring.fail = &s_fail;
    ring.gbase = gbase;
    ring.issued = 0;
    ring.observed = 0;
    ring.bad = false;
    ring.wait_test = a.wait_test;
    // the producer is the last of the level threads: levels rarely have rows
    // for it, so its copies overlap the other threads' work.  The mbarriers are
    // initialised with the CTA's first subdomain; later ones continue their
    // phases (every group of the previous subdomain was issued and observed).
    const int LT = a.level_threads;
    ring.producer = (int)threadIdx.x == LT - 1;
    if (ring.producer) {
        if (first)
            for (int i = 0; i < RING_NBAR; ++i) mbar_init(ring.bars_s + 8u * (uint32_t)i, 1);
        fence_mbar_init();
        s_fail = 0;
    }
    gbase += rs.ngrp;
    __syncthreads();
    if (ring.producer) ring.issue_to(rs.ninit);
    // gather while the first records are in flight; with a coarse term the
    // subdomain's row of the coarse inverse comes into shared memory with it
    const int* dof = a.dofs + inf.row_off;
    const int tp = inf.tshift;
    if (coarse && a.a0pre && threadIdx.x < 32) {
        const double* row = a.a0inv + (size_t)s * a.nc;
        for (int q = threadIdx.x; q < a.nc; q += 32) cp_async8(smem_u32(sm.a0row + q), row + q);
    }
    if constexpr (std::is_same<TI, TS>::value) {
        gather_async<TS, R>(smem_u32(t), x, a.ldx, dof, n, NC, tp);
    } else {
        gather_convert<TS, TI, R>(t, x, a.ldx, dof, n, NC, tp);
    }
    cp_async_wait_all();
    if (threadIdx.x < R) t[(size_t)R * tslot(n, tp) + threadIdx.x] = (TS)0;
    if (coarse && a.fuse && (int)gridDim.x == a.nparts && (int)blockIdx.x >= a.nparts / 2) {
        // no blocks to spare for the restrictions.  Blocks run largest
        // subdomain first, so the second half -- the smaller subdomains, with
        // slack -- computes its own and its mirror block's before the level
        // loop, and the critical first half computes none.
        const int mirror = a.nparts - 1 - (int)blockIdx.x;
        for (int pass = 0; pass < (mirror == (int)blockIdx.x ? 1 : 2); ++pass) {
            const int sr = pass == 0 ? s : a.order[mirror];
            publish_restriction<TI>(a, sr, pass == 0 ? inf : a.info[sr], x, s_red);
        }
    }
    __syncthreads();

    // the level loop -- the latency chain of the sweep -- one direction at a
    // time, specialised on the row width
    const uint32_t t_s = smem_u32(t);
    if ((int)threadIdx.x < LT) {
        level_loop_w<false, TS, TF, EXACT, R>(sm.ent, 0, rs.ngrp_f, inf.wl, a.row_structs != 0,
                                              ring, t, t_s, sm.ring, LT);
        level_loop_w<true, TS, TF, EXACT, R>(sm.ent, rs.ngrp_f, rs.ngrp, inf.wu,
                                             a.row_structs != 0, ring, t, t_s, sm.ring, LT);
    }
    __syncthreads();
    if (s_fail) {  // a wait gave up
        ring.drain(a.err);
        return false;
    }

    if (coarse) {
        if (a.fuse) {
            // every block published its restriction before its level loop;
            // all blocks are resident (cooperative launch), so this bounded
            // wait ends as soon as the slowest block got there
            if (threadIdx.x == 0) {
                const long long t0 = clock64();
                int ok = 1;
                while (ld_acquire(&a.sync[0]) < (unsigned)a.nparts) {
                    if (clock64() - t0 > a.wait_budget) {
                        ok = 0;
                        break;
                    }
                    __nanosleep(64);
                }
                s_ok = ok;
            }
            __syncthreads();
            if (!s_ok) {
                if (threadIdx.x == 0) atomicMax(a.err, 1);
                return false;
            }
        }
        if (threadIdx.x < 32) {
            const double* row = a.a0pre ? sm.a0row : a.a0inv + (size_t)s * a.nc;
            const double z = a.fuse ? coarse_dot_warp0<true>(row, a.r0, a.nc)
                                    : coarse_dot_warp0<false>(row, a.r0, a.nc);
            if (threadIdx.x == 0) {
                s_zc = inf.cscale * z;
                // the last block done with r0 resets the counters
                if (a.fuse && atomicAdd(&a.sync[1], 1u) == (unsigned)a.nparts - 1) {
                    a.sync[0] = 0u;
                    a.sync[1] = 0u;
                }
            }
        }
        __syncthreads();
    }
    const double zc = coarse ? s_zc : 0.0;
    if (mode == 0) {
        scatter_ilp<TS, TO, R>(t, y, a.ldy, a.ownloc + inf.own_off, a.owned + inf.own_off,
                               inf.n_own, coarse, zc, NC, tp);
    } else {
        for (int li = threadIdx.x; li < n; li += NC)
#pragma unroll
            for (int i = 0; i < R; ++i)
                atomicAdd(&y[i * a.ldy + dof[li]], Store<TO>::f(t[(size_t)R * tslot(li, tp) + i]));
        if (coarse) {
            const int* og = a.owned + inf.own_off;
            for (int q = threadIdx.x; q < inf.n_own; q += NC)
                atomicAdd(&y[og[q]], Store<TO>::f(zc));
        }
    }
    return true;
}

// The same as a call of its own, for CTAs that loop over subdomains: inlined
// there, values hoisted out of that loop spill inside the level loops.
template <class TI, class TO, class TS, class TF, bool EXACT, int R>
__device__ __noinline__ bool sweep_one_call(const RecArgs& a, int s, const TI* __restrict__ x,
                                            TO* __restrict__ y, int mode, int coarse,
                                            const SweepSmem& sm, int& gbase, bool first) {
    return sweep_one<TI, TO, TS, TF, EXACT, R>(a, s, x, y, mode, coarse, sm, gbase, first);
}

// mode 0: RAS (owned rows written), 1: ASM (all rows added atomically).  One
// subdomain per CTA, or (PERSIST) CTAs looping over subdomains taken largest
// first from a work counter.
template <class TI, class TO, class TS, class TF, bool EXACT, int R, bool PERSIST>
__global__ void __launch_bounds__(SW_T, 2)
k_sweep_tma(const __grid_constant__ RecArgs a, const TI* __restrict__ x, TO* __restrict__ y, int mode, int coarse,
            const int* __restrict__ active) {
    if (active && *active == 0) return;
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr uint32_t HDR = RING_NBAR * 8;
    SweepSmem sm;
    sm.raw = smraw;
    sm.ring = smraw + HDR;
    sm.t = sm.ring + a.ring_bytes;
    sm.grp = reinterpret_cast<int4*>(reinterpret_cast<unsigned char*>(sm.t) +
                                     (((size_t)a.t_len * R * sizeof(TS) + 15) & ~(size_t)15));
    sm.ent = reinterpret_cast<int2*>(sm.grp + a.max_grp + 1);
    sm.a0row = reinterpret_cast<double*>(sm.ent + a.max_ent);
    auto on = [&](int s) {
        if (!a.sub_on) return true;
        bool v = false;
#pragma unroll
        for (int i = 0; i < R; ++i) v = v || a.sub_on[(size_t)i * a.nparts + s] != 0;
        return v;
    };
    int gbase = 0;  // record groups this CTA has streamed (mbarrier phases)
    if constexpr (!PERSIST) {
        if (a.fuse && (int)blockIdx.x >= a.nparts) {
            double* red = reinterpret_cast<double*>(sm.ring);  // the ring and vector are unused
            for (int q = (int)blockIdx.x - a.nparts; q < a.nparts; q += (int)gridDim.x - a.nparts) {
                const int sr = a.order[q];
                publish_restriction<TI>(a, sr, a.info[sr], x, red);
                __syncthreads();
            }
            return;
        }
        const int s = a.order[blockIdx.x];
        if (!on(s)) return;  // subdomain not needed by this apply
        sweep_one<TI, TO, TS, TF, EXACT, R>(a, s, x, y, mode, coarse, sm, gbase, true);
    } else {
        __shared__ int s_next;
        bool first = true;
        for (;;) {
            __syncthreads();  // every thread has read the previous index
            if (threadIdx.x == 0) s_next = (int)atomicAdd(&a.work[0], 1u);
            __syncthreads();
            const int idx = s_next;
            if (idx >= a.nparts) break;
            const int s = a.order[idx];
            if (!on(s)) continue;
            if (!sweep_one_call<TI, TO, TS, TF, EXACT, R>(a, s, x, y, mode, coarse, sm, gbase,
                                                          first))
                return;
            first = false;
        }
        if (threadIdx.x == 0 && atomicAdd(&a.work[1], 1u) == gridDim.x - 1) {
            a.work[0] = 0u;  // every CTA has taken its last index: the counters restart
            a.work[1] = 0u;
        }
    }
}

bool sweep_a0_prefetch(const sg_precond* pc);

RecArgs rec_args(sg_precond* pc, const RingPlan& plan, bool fuse) {
    RecArgs a;
    a.fuse = fuse ? 1 : 0;
    a.r0w = pc->r0.p;
    a.sync = pc->coarse_sync.p;
    a.info = pc->info.p;
    a.order = pc->order.p;
    a.dofs = pc->dofs.p;
    a.ring = reinterpret_cast<const RingSub*>(plan.sub_d.p);
    a.ent = reinterpret_cast<const int2*>(plan.ent_d.p);
    a.grp = reinterpret_cast<const int4*>(plan.grp_d.p);
    a.rec = pc->rec_d.p;
    a.ownloc = pc->ownloc_d.p;
    a.owned = pc->owned_d.p;
    a.a0inv = pc->a0inv.p;
    a.r0 = pc->r0.p;
    a.nparts = pc->nparts;
    a.nc = pc->nc;
    a.a0pre = sweep_a0_prefetch(pc) ? 1 : 0;
    a.row_structs = pc->rec_rows ? 1 : 0;
    a.ring_bytes = (int)plan.ring_bytes;
    a.t_len = pc->t_len;
    a.max_ent = plan.max_ent;
    a.max_grp = plan.max_grp;
    a.level_threads = plan.level_threads;
    a.ldx = 0;
    a.ldy = 0;
    a.err = pc->err_d.p;
    a.sub_on = pc->sub_on;
    a.persist = (plan.grid > 0 && !fuse) ? 1 : 0;
    a.work = plan.work.p;
    a.wait_test = pc->wait_test;
    a.wait_budget = pc->wait_test ? WAIT_TEST_CYCLES : WAIT_CYCLES;
    return a;
}

// two-level preconditioners with at most 1024 subdomains keep the
// subdomain's row of the coarse inverse in shared memory
bool sweep_a0_prefetch(const sg_precond* pc) {
    return (pc->kind == SG_PC_TWOLEVEL_ASM || pc->kind == SG_PC_TWOLEVEL_RAS) &&
           pc->nparts <= 1024;
}

// dynamic shared memory of the sweep: the mbarriers, the record ring, the
// subdomain vector (R elements per slot), the schedule's groups and entries,
// the coarse row
size_t sweep_smem_for(const sg_precond* pc, const RingPlan& plan, long long ring_bytes) {
    const size_t ts = pc->opts.sweep_dtype == SG_FP64 ? 8 : 4;
    const size_t tbytes = ((size_t)pc->t_len * ts * plan.R + 15) & ~(size_t)15;
    const size_t a0 = sweep_a0_prefetch(pc) ? (size_t)pc->nparts * 8 : 0;
    return RING_NBAR * 8 + (size_t)ring_bytes + tbytes + ((size_t)plan.max_grp + 1) * 16 +
           (size_t)plan.max_ent * 8 + a0;
}
size_t sweep_smem(const sg_precond* pc, const RingPlan& plan) {
    return sweep_smem_for(pc, plan, plan.ring_bytes);
}

// Blocks of the fused sweep that compute restrictions only: one a subdomain,
// or as many as still fit when that leaves each at most four.  32 subdomains
// of a 201 x 187 grid: sweep 35.7 -> 31.4 us; 108 of 96^3 (44 blocks): apply
// 167 -> 164; with 48 blocks for 256 subdomains of 128^3 66.4 -> 66.6, so not
// there (the second half of the sweeping blocks has the time).
int restrict_blocks(int nparts, int cap) {
    const int room = std::min(nparts, cap - nparts);
    return room > 0 && 4LL * room >= nparts ? room : 0;
}

template <class TI, class TO, class TS, class TF, bool EXACT, int R>
void launch_tma(sg_precond* pc, const RingPlan& plan, const TI* x, TO* y, int mode, bool coarse,
                const int* active, bool fuse = false, long long ldx = 0, long long ldy = 0) {
    const size_t smem = sweep_smem(pc, plan);
    const int nt = plan.threads > 0 ? plan.threads : SW_T;
    RecArgs a = rec_args(pc, plan, fuse);
    // persistent CTAs only for FP32 sweeps (the FP64 ones keep their
    // registers for the level loop)
    if (sizeof(TS) == 8) a.persist = 0;
    auto kern = k_sweep_tma<TI, TO, TS, TF, EXACT, R, false>;
    if constexpr (sizeof(TS) == 4) {
        if (a.persist) kern = k_sweep_tma<TI, TO, TS, TF, EXACT, R, true>;
    }
    allow_smem(pc->ctx, kern);
    a.ldx = ldx;
    a.ldy = ldy;
    const int coarse_i = coarse ? 1 : 0;
    if (fuse) {
        // the blocks wait for one another's restriction: co-residency is
        // guaranteed by the cooperative launch (checked at set-up).  Where the
        // GPU holds more blocks than subdomains, the others take the
        // restrictions off the sweeping ones.
        auto& cap = plan.resident[reinterpret_cast<const void*>(kern)];
        if (cap == 0) {
            int per_sm = 0;
            SG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nt, smem));
            cap = per_sm * pc->ctx->num_sms;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(pc->nparts + restrict_blocks(pc->nparts, cap));
        cfg.blockDim = dim3(nt);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = pc->ctx->stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        SG_CUDA(cudaLaunchKernelEx(&cfg, kern, a, x, y, mode, coarse_i, active));
    } else {
        const int grid = a.persist ? plan.grid : pc->nparts;
        kern<<<grid, nt, smem, pc->ctx->stream>>>(a, x, y, mode, coarse_i, active);
    }
    SG_CUDA(cudaGetLastError());
    count_launch(pc->ctx);
}

}  // namespace

// Builds the static ring schedule of every subdomain (see RingSub) into
// `plan` for level loops of nlt threads, groups of at most gmax bytes (a
// larger level is a group of its own) and the ring that `budget` bytes of
// dynamic shared memory leave.  Groups are placed one after another and start
// over at the ring's beginning when they would cross its end.  Group j may be
// issued after the last level of every earlier group whose ring bytes it
// overwrites and of group j - RING_NBAR (its mbarrier's previous user); the
// schedule is feasible when that is always before group j's first level.
// Returns false when it is not.
static bool ring_schedule(const sg_precond* pc, RingPlan& plan, long long budget, long long gmax,
                          int nlt) {
    const int sf = rec_value_bytes(pc);
    const int pass = std::max(1, nlt / plan.R);  // rows the level threads take at once
    std::vector<RingSub> subs((size_t)pc->nparts);
    std::vector<int> ent, grp;  // int2 / int4 entries as ints
    struct Group {
        int first, last;  // levels
        long long start, bytes, pos;
    };
    std::vector<Group> groups;  // of all subdomains
    int max_ent = 0, max_grp = 0;
    for (int s = 0; s < pc->nparts; ++s) {
        const SubInfo& inf = pc->h_info[s];
        const int nf = inf.nlev_f, T = inf.nlev_f + inf.nlev_b;
        RingSub& r = subs[s];
        r.base = nf > 0 ? pc->h_rec_off_f[inf.lev_off_f]
                        : (T > 0 ? pc->h_rec_off_b[inf.lev_off_b] : 0);
        const size_t g0 = groups.size();
        r.ngrp_f = 0;
        int nent = 0;
        for (int g = 0; g < T; ++g) {
            const bool back = g >= nf;
            const int i = back ? inf.lev_off_b + (g - nf) : inf.lev_off_f + g;
            const std::vector<int>& lp = back ? pc->h_lev_ptr_b : pc->h_lev_ptr_f;
            const int c = lp[i + 1] - lp[i], w = back ? inf.wu : inf.wl;
            const long long rel = (back ? pc->h_rec_off_b[i] : pc->h_rec_off_f[i]) - r.base;
            const long long B = rec_level_bytes(pc, w, back, c);
            if (groups.size() == g0 || g == nf || groups.back().bytes + B > gmax) {
                groups.push_back({g, g, rel, B, 0});
                ++nent;  // the entry that ends it
                if (!back) ++r.ngrp_f;
            } else {
                groups.back().last = g;
                groups.back().bytes = rel + B - groups.back().start;
            }
            nent += pc->rec_rows && rec_is_rows(w) ? (c + pass - 1) / pass : 1;
        }
        r.ngrp = (int)(groups.size() - g0);
        r.nent = nent + 1;  // the loop reads one entry past the last
        max_ent = std::max(max_ent, r.nent);
        max_grp = std::max(max_grp, r.ngrp);
    }
    plan.max_ent = max_ent;
    plan.max_grp = max_grp;
    plan.level_threads = nlt;
    const long long ring = (budget - (long long)sweep_smem_for(pc, plan, 0)) & ~15ll;
    if (ring < pc->rec_stage_bytes) return false;
    std::vector<int> ia;
    size_t gbase = 0;
    for (int s = 0; s < pc->nparts; ++s) {
        const SubInfo& inf = pc->h_info[s];
        const int nf = inf.nlev_f;
        RingSub& r = subs[s];
        const int G = r.ngrp;
        Group* gr = groups.data() + gbase;
        gbase += (size_t)G;
        long long pos = 0;
        for (int j = 0; j < G; ++j) {
            if (gr[j].bytes > ring || gr[j].bytes >= (1ll << 20)) return false;
            if (pos + gr[j].bytes > ring) pos = 0;
            gr[j].pos = pos;
            pos += gr[j].bytes;
        }
        // ia[j]: the group after which group j may be issued (-1: at once)
        ia.assign(G, -1);
        int run = -1;
        for (int j = 0; j < G; ++j) {
            int v = -1;
            for (int i = std::max(0, j - RING_NBAR); i < j; ++i)
                if (gr[i].pos < gr[j].pos + gr[j].bytes && gr[j].pos < gr[i].pos + gr[i].bytes)
                    v = i;
            if (j >= RING_NBAR) v = std::max(v, j - RING_NBAR);
            run = std::max(run, v);
            ia[j] = run;
        }
        r.ninit = 0;
        while (r.ninit < G && ia[r.ninit] < 0) ++r.ninit;
        r.ent_off = (int)(ent.size() / 2);
        r.grp_off = (int)(grp.size() / 4);
        int ji = 0, ne = 0;
        for (int j = 0; j < G; ++j) {
            while (ji < G && ia[ji] <= j) ++ji;
            grp.push_back((int)gr[j].start);
            grp.push_back((int)((gr[j].bytes >> 4) | ((gr[j].pos >> 4) << 16)));
            grp.push_back(ne);
            grp.push_back(ji);
            for (int g = gr[j].first; g <= gr[j].last; ++g) {
                const bool back = g >= nf;
                const int i = back ? inf.lev_off_b + (g - nf) : inf.lev_off_f + g;
                const std::vector<int>& lp = back ? pc->h_lev_ptr_b : pc->h_lev_ptr_f;
                const int c = lp[i + 1] - lp[i], w = back ? inf.wu : inf.wl;
                const long long rel = (back ? pc->h_rec_off_b[i] : pc->h_rec_off_f[i]) - r.base;
                const int at = (int)(gr[j].pos + rel - gr[j].start);
                const bool rows = pc->rec_rows && rec_is_rows(w);
                const int step = rows ? pass : c, rb = rec_row_bytes(w, back, sf);
                for (int q = 0; q < c; q += step, ++ne) {
                    ent.push_back((c - q) | (q + step >= c ? 0x10000 : 0));
                    ent.push_back(at + (rows ? q * rb : 0));
                }
            }
            ent.push_back(0);
            ent.push_back(0);
            ++ne;
        }
        ent.push_back(0);
        ent.push_back(0);
        for (int v : {0, 0, ne, G}) grp.push_back(v);
    }
    plan.sub.assign(reinterpret_cast<const unsigned char*>(subs.data()),
                    reinterpret_cast<const unsigned char*>(subs.data() + subs.size()));
    plan.ent.swap(ent);
    plan.grp.swap(grp);
    plan.ring_bytes = ring;
    plan.gmax = gmax;
    return true;
}

static void ring_upload(sg_precond* pc, RingPlan& plan) {
    cudaStream_t st = pc->ctx->stream;
    plan.sub_d.upload(plan.sub, st);
    plan.ent_d.upload(plan.ent, st);
    plan.grp_d.upload(plan.grp, st);
}

// Resident CTAs per SM of the sweep kernel for the plan's shared memory and
// block size.
template <class K>
static int sweep_occupancy(sg_precond* pc, const RingPlan& plan, K kern) {
    const size_t smem = sweep_smem(pc, plan);
    const int nt = plan.threads > 0 ? plan.threads : SW_T;
    int per_sm = 0;
    allow_smem(pc->ctx, kern);
    SG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nt, smem));
    return per_sm;
}

// Block sizes to time, and how many of the threads run the level loop.  FP64
// levels run on few warps (see level_loop) while the whole block gathers and
// scatters; opts.reserved[1] forces one size for both.  One- and two-warp CTAs
// are not timed: on the 2D subdomains of the batched workload (~20 rows per
// level) they measured slower than 128 threads (the gather, scatter and
// record stream lose more than the cheaper barrier gains).
struct BlockShape {
    int threads, level_threads;
};
static std::vector<BlockShape> block_shapes(const sg_precond* pc) {
    const int forced = pc->opts.reserved[1];
    if (forced > 0) return {{forced, forced}};
    if (pc->opts.sweep_dtype == SG_FP64) return {{384, 384}, {256, 256}, {256, 128}, {256, 64}};
    return {{512, 512}, {384, 384}, {256, 256}, {128, 128}};
}

// The dynamic shared memory a plan's CTAs may use (what the CTAs that must
// share an SM leave each other) and the record-group sizes whose schedule is
// feasible in it.
struct RingFit {
    long long budget = 0;
    std::vector<long long> gmax;
};
static RingFit ring_size(sg_precond* pc, RingPlan& plan) {
    sg_ctx* ctx = pc->ctx;
    int max_smem = 0, sm_smem = 0;
    SG_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                   ctx->device));
    SG_CUDA(cudaDeviceGetAttribute(&sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor,
                                   ctx->device));
    const int static_smem = 1024;  // reduction scratch and the like
    // CTAs per SM needed to keep every subdomain resident at once (more
    // subdomains than that run persistent or in waves)
    int want = (pc->nparts + ctx->num_sms - 1) / ctx->num_sms;
    if (want > 4) want = 4;
    const int nlt = block_shapes(pc).front().level_threads;  // the fewest entries
    RingFit fit;
    for (int per_sm = want < 1 ? 1 : want; per_sm >= 1 && fit.gmax.empty(); --per_sm) {
        fit.budget = std::min<long long>((long long)sm_smem / per_sm - static_smem - 1024,
                                         (long long)max_smem - static_smem);
        // group size: opts.reserved[3] when set, else timed among two sizes
        // (never below the largest record): 8 and 16 KB, or 16 and 32 KB where
        // the ring holds four of them -- each group costs the level loop ~160
        // cycles, and the first one delays the first level
        plan.max_ent = plan.max_grp = 0;
        const long long room = fit.budget - (long long)sweep_smem_for(pc, plan, 0);
        std::vector<long long> gcand = {8192, 16384};
        if (room >= 131072) gcand = {16384, 32768};
        if (pc->opts.reserved[3] > 0) gcand = {pc->opts.reserved[3]};
        for (long long target : gcand) {
            for (long long gmax : {target, target / 2, target / 4}) {
                if (gmax < pc->rec_stage_bytes) gmax = pc->rec_stage_bytes;
                if (ring_schedule(pc, plan, fit.budget, gmax, nlt)) {
                    if (std::find(fit.gmax.begin(), fit.gmax.end(), gmax) == fit.gmax.end())
                        fit.gmax.push_back(gmax);
                    break;
                }
            }
        }
    }
    return fit;
}

void tune_plan(sg_precond* pc, RingPlan& plan, const RingFit& fit);

// Packs the level records.  Returns false where they are row structs of an
// FP64 sweep and a diagonal is so small, large or non-finite that its quotients
// have to be divided.
static bool pack_records(sg_precond* pc) {
    cudaStream_t st = pc->ctx->stream;
    const bool check = pc->opts.sweep_dtype == SG_FP64 && pc->rec_rows;
    if (!pc->far_d.p) {
        pc->far_d.alloc(1);
        pc->far_h.alloc(1);
    }
    if (check) pc->far_d.zero(st);
    const uint16_t* pf = pc->perm_f.p;
    const uint16_t* pb = pc->perm_b.p;
    const int per = std::min(16, std::max(1, 8 * pc->ctx->num_sms / pc->nparts));
#define SG_PACK(TF)                                                                        \
    k_pack_rec<TF><<<dim3(pc->nparts, per), 256, 0, st>>>(                                 \
        pc->info.p, pc->lrp_d.p, pc->lci_d.p, pc->ldiag_d.p, pc->lu_d.p, pf, pb,            \
        pc->lev_ptr_f.p, pc->lev_ptr_b.p, pc->rec_off_f_d.p, pc->rec_off_b_d.p,             \
        pc->rec_rows_f_d.p, pc->rec_rows_b_d.p, pc->rec_rows ? 1 : 0, pc->rec_d.p, pc->far_d.p)
    if (pc->opts.sweep_dtype == SG_FP64) SG_PACK(double);
    else if (pc->opts.factor_dtype == SG_BF16) SG_PACK(uint16_t);
    else SG_PACK(float);
#undef SG_PACK
    SG_CUDA(cudaGetLastError());
    if (!check) return true;
    SG_CUDA(cudaMemcpyAsync(pc->far_h.p, pc->far_d.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    SG_CUDA(cudaStreamSynchronize(st));
    return *pc->far_h.p == 0;
}

// Packs the level records in the configured factor type, plans the
// one-vector ring and times its block size, record-group size and launch
// shape.  All but the records depends on the structure alone: a set-up with
// new values of the same structure (kept) packs them again and leaves the
// rest (the plan's 56 timed sweeps took 3 of the 6.2 ms of a re-set-up at
// 64^3).
void rec_setup_device(sg_precond* pc, bool kept) {
    if (!pc->use_rec) return;
    sg_ctx* ctx = pc->ctx;
    cudaStream_t st = ctx->stream;
    RingPlan& plan = pc->ring1;
    if (kept) {
        pc->err_d.zero(st);
        if (pc->coarse_sync.p) pc->coarse_sync.zero(st);
        if (pack_records(pc)) return;
    }
    plan.R = 1;
    plan.ready = false;
    pc->ring4.ready = false;  // a new set-up plans the four-vector ring again when asked
    // records of row structs, unless their rings do not fit beside the vector
    // of a subdomain near the shared-memory limit (component records are
    // smaller) or a diagonal needs the division (their rows divide)
    RingFit fit;
    pc->rec_divides = false;
    for (bool rows = true;; rows = false) {
        rec_layout(pc, rows);
        fit = ring_size(pc, plan);
        if (fit.gmax.empty() && rows) continue;
        if (fit.gmax.empty() || (pc->opts.reserved[0] & 1)) {
            pc->use_rec = false;
            return;
        }
        if (pc->rec_stage_bytes % 16 != 0 || pc->rec_total % 16 != 0)
            fail(SG_ERR_INTERNAL, "level records are not 16-byte multiples");
        pc->rec_depth = 1;
        pc->rec_off_f_d.upload(pc->h_rec_off_f, st);
        pc->rec_off_b_d.upload(pc->h_rec_off_b, st);
        pc->rec_rows_f_d.upload(pc->h_rec_rows_f, st);
        pc->rec_rows_b_d.upload(pc->h_rec_rows_b, st);
        pc->rec_d.alloc((size_t)pc->rec_total);
        pc->err_d.alloc(1);
        if (!pc->err_h.p) pc->err_h.alloc(1);
        pc->err_d.zero(st);
        if (pack_records(pc)) break;
        pc->rec_divides = true;
    }
    // block size (forced by opts.reserved[1], else timed), record-group size
    // and launch shape.  Levels of a 3D subdomain hold ~100+ rows, those of a
    // small 2D one ~20: a 512-thread block then idles at every level
    // barrier, while narrower blocks let more subdomains run at once.
    tune_plan(pc, plan, fit);
    pc->sweep_threads = plan.threads;
    // two-level: the coarse restriction runs inside the sweep when every
    // subdomain's CTA can be resident at once (a cooperative launch)
    pc->fuse_restrict = false;
    if (pc->kind == SG_PC_TWOLEVEL_ASM || pc->kind == SG_PC_TWOLEVEL_RAS) {
        int coop = 0, per_sm = 0;
        SG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
        if (pc->opts.sweep_dtype == SG_FP64)
            per_sm = sweep_occupancy(pc, plan, k_sweep_tma<double, double, double, double, false, 1, false>);
        else if (pc->opts.factor_dtype == SG_BF16)
            per_sm = sweep_occupancy(pc, plan, k_sweep_tma<float, float, float, uint16_t, false, 1, false>);
        else
            per_sm = sweep_occupancy(pc, plan, k_sweep_tma<float, float, float, float, false, 1, false>);
        if (coop && (long long)per_sm * ctx->num_sms >= pc->nparts && pc->opts.reserved[2] == 0) {
            pc->coarse_sync.alloc(2);
            pc->coarse_sync.zero(st);
            pc->fuse_restrict = true;
        }
    }
}

bool sweep_fuses_restrict(const sg_precond* pc) {
    return pc->use_rec && pc->rec_depth > 0 && pc->fuse_restrict && !pc->sub_on;
}

// Times the sweep (RAS mode, no coarse term, zero input; R interleaved
// vectors) for every record-group size of the fit, every block shape and, when there are more
// subdomains than resident CTAs, one CTA per subdomain against a persistent
// grid; keeps the fastest.
void tune_plan(sg_precond* pc, RingPlan& plan, const RingFit& fit) {
    sg_ctx* ctx = pc->ctx;
    cudaStream_t st = ctx->stream;
    const int R = plan.R;
    const size_t n = (size_t)std::max(pc->n, 1) * R;
    const bool f64 = pc->opts.sweep_dtype == SG_FP64;
    const bool bf16 = pc->opts.factor_dtype == SG_BF16;
    DBuf<double> x64, y64;
    DBuf<float> x32, y32;
    if (f64) {
        x64.alloc(n);
        y64.alloc(n);
        x64.zero(st);
    } else {
        x32.alloc(n);
        y32.alloc(n);
        x32.zero(st);
    }
    if (!plan.work.p) {
        plan.work.alloc(2);
        plan.work.zero(st);
    }
    const long long ld = pc->n;
    auto run = [&] {
        if (f64) launch_tma<double, double, double, double, false, 1>(pc, plan, x64.p, y64.p, 0, false, nullptr);
        else if (R == 4 && bf16) launch_tma<float, float, float, uint16_t, false, 4>(pc, plan, x32.p, y32.p, 0, false, nullptr, false, ld, ld);
        else if (R == 4) launch_tma<float, float, float, float, false, 4>(pc, plan, x32.p, y32.p, 0, false, nullptr, false, ld, ld);
        else if (bf16) launch_tma<float, float, float, uint16_t, false, 1>(pc, plan, x32.p, y32.p, 0, false, nullptr);
        else launch_tma<float, float, float, float, false, 1>(pc, plan, x32.p, y32.p, 0, false, nullptr);
    };
    auto occupancy = [&]() -> int {
        if (f64) return sweep_occupancy(pc, plan, k_sweep_tma<double, double, double, double, false, 1, false>);
        if (R == 4 && bf16) return sweep_occupancy(pc, plan, k_sweep_tma<float, float, float, uint16_t, false, 4, false>);
        if (R == 4) return sweep_occupancy(pc, plan, k_sweep_tma<float, float, float, float, false, 4, false>);
        if (bf16) return sweep_occupancy(pc, plan, k_sweep_tma<float, float, float, uint16_t, false, 1, false>);
        return sweep_occupancy(pc, plan, k_sweep_tma<float, float, float, float, false, 1, false>);
    };
    plan.resident.clear();
    cudaEvent_t e0, e1;
    SG_CUDA(cudaEventCreate(&e0));
    SG_CUDA(cudaEventCreate(&e1));
    float best = -1.f;
    BlockShape best_sh{SW_T, SW_T};
    int best_grid = 0;
    long long best_g = fit.gmax.front();
    for (long long gmax : fit.gmax) {
        // every shape with the first group size, the fastest of them with the
        // others (all pairs: 16 subdomains of a graph of 40,000 rows, 0.5 ms a
        // sweep, 42 ms a set-up; 33 so)
        const std::vector<BlockShape> shapes =
            best < 0.f ? block_shapes(pc) : std::vector<BlockShape>{best_sh};
        for (const BlockShape& sh : shapes) {
            if (!ring_schedule(pc, plan, fit.budget, gmax, sh.level_threads)) continue;
            ring_upload(pc, plan);
            plan.threads = sh.threads;
            plan.grid = 0;
            const int per_sm = occupancy();
            if (per_sm < 1) continue;
            const long long cap = (long long)per_sm * ctx->num_sms;
            // launch shape: opts.reserved[4] 1 forces one CTA per subdomain,
            // 2 a persistent grid of the resident CTAs, k > 2 a persistent
            // grid of k CTAs (at most the resident ones); 0 times one CTA per
            // subdomain against the persistent grid when there are more
            // subdomains than resident CTAs
            std::vector<int> grids = {0};
            const int shape = pc->opts.reserved[4];
            if (shape == 2) grids = {(int)std::min<long long>(cap, pc->nparts)};
            else if (shape > 2) grids = {(int)std::min<long long>(std::min<long long>(cap, shape), pc->nparts)};
            else if (shape == 0 && cap < pc->nparts) grids.push_back((int)cap);
            if (f64) grids = {0};  // FP64 sweeps run one CTA per subdomain
            for (int grid : grids) {
                plan.grid = grid;
                run();
                run();
                cudaEventRecord(e0, st);
                for (int r = 0; r < 5; ++r) run();
                cudaEventRecord(e1, st);
                cudaError_t e = cudaEventSynchronize(e1);
                float ms = 0.f;
                if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
                if (e != cudaSuccess) {
                    cudaEventDestroy(e0);
                    cudaEventDestroy(e1);
                    SG_CUDA(e);
                }
                if (best < 0.f || ms < best) {
                    best = ms;
                    best_sh = sh;
                    best_g = gmax;
                    best_grid = grid;
                }
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (best < 0.f) fail(SG_ERR_INTERNAL, "no sweep configuration fits the GPU");
    plan.threads = best_sh.threads;
    plan.grid = best_grid;
    if (!ring_schedule(pc, plan, fit.budget, best_g, best_sh.level_threads)) fail(SG_ERR_INTERNAL, "ring schedule lost");
    ring_upload(pc, plan);
    plan.ready = true;
}

template <class TI, class TO>
bool sweep_tma(sg_precond* pc, const TI* x, TO* y, int mode, bool coarse, bool exact,
               const int* active) {
    if (!pc->use_rec || pc->rec_depth == 0) return false;
    const RingPlan& plan = pc->ring1;
    const bool fuse = coarse && sweep_fuses_restrict(pc);
    if (pc->opts.sweep_dtype == SG_FP64) {
        if (exact) launch_tma<TI, TO, double, double, true, 1>(pc, plan, x, y, mode, coarse, active, fuse);
        else launch_tma<TI, TO, double, double, false, 1>(pc, plan, x, y, mode, coarse, active, fuse);
    } else if (pc->opts.factor_dtype == SG_BF16) {
        launch_tma<TI, TO, float, uint16_t, false, 1>(pc, plan, x, y, mode, coarse, active, fuse);
    } else {
        launch_tma<TI, TO, float, float, false, 1>(pc, plan, x, y, mode, coarse, active, fuse);
    }
    return true;
}

// Plans (and times) the four-vector ring of a RAS preconditioner with FP32
// sweeps, once per set-up; call it outside stream capture.  False when the
// preconditioner has no such sweep.
bool sweep_plan4(sg_precond* pc) {
    if (!pc->use_rec || pc->rec_depth == 0 || pc->opts.sweep_dtype == SG_FP64) return false;
    if (pc->kind != SG_PC_RAS) return false;
    RingPlan& plan = pc->ring4;
    if (plan.ready) return true;
    plan.R = 4;
    const RingFit fit = ring_size(pc, plan);
    if (fit.gmax.empty()) return false;
    const int* keep = pc->sub_on;
    pc->sub_on = nullptr;
    tune_plan(pc, plan, fit);
    pc->sub_on = keep;
    return true;
}

// Four right-hand sides at once (RAS without a coarse term, FP32 sweeps): x
// and y hold them ld apart; sub_on (NULL or 4 x nparts switches) gates the
// subdomains.  Returns false, launching nothing, when the four-vector ring
// has not been planned (sweep_plan4).
template <class TI, class TO>
bool sweep_tma4(sg_precond* pc, const TI* x, TO* y, long long ld, const int* sub_on) {
    if (!pc->use_rec || pc->rec_depth == 0 || pc->opts.sweep_dtype == SG_FP64) return false;
    if (pc->kind != SG_PC_RAS || !pc->ring4.ready) return false;
    const RingPlan& plan = pc->ring4;
    const int* keep = pc->sub_on;
    pc->sub_on = sub_on;
    struct Restore {
        sg_precond* pc;
        const int* v;
        ~Restore() { pc->sub_on = v; }
    } restore{pc, keep};
    if (pc->opts.factor_dtype == SG_BF16)
        launch_tma<TI, TO, float, uint16_t, false, 4>(pc, plan, x, y, 0, false, nullptr, false, ld, ld);
    else
        launch_tma<TI, TO, float, float, false, 4>(pc, plan, x, y, 0, false, nullptr, false, ld, ld);
    return true;
}

void sweep_error_fetch(sg_precond* pc) {
    if (pc->err_d.p)
        SG_CUDA(cudaMemcpyAsync(pc->err_h.p, pc->err_d.p, sizeof(int), cudaMemcpyDeviceToHost,
                                pc->ctx->stream));
}

int sweep_error(sg_precond* pc) {
    if (!pc->err_d.p) return 0;
    sweep_error_fetch(pc);
    SG_CUDA(cudaStreamSynchronize(pc->ctx->stream));
    return sweep_error_fetched(pc);
}

int sweep_error_fetched(sg_precond* pc) {
    if (!pc->err_d.p) return 0;
    const int e = *pc->err_h.p;
    // reported once: clear the error word, the fused restriction's counters
    // and the persistent launches' work counters, which a sweep that gave up
    // may have left mid-count, so the next apply starts clean
    if (e) {
        pc->err_d.zero(pc->ctx->stream);
        if (pc->coarse_sync.p) pc->coarse_sync.zero(pc->ctx->stream);
        if (pc->ring1.work.p) pc->ring1.work.zero(pc->ctx->stream);
        if (pc->ring4.work.p) pc->ring4.work.zero(pc->ctx->stream);
        SG_CUDA(cudaStreamSynchronize(pc->ctx->stream));
    }
    return e;
}

bool sweep_wait_test_supported(const sg_precond* pc, int mode) {
    if (mode == 0) return true;
    if (!pc->use_rec || pc->rec_depth == 0) return false;
    if (mode == 1) return true;
    return mode == 2 && sweep_fuses_restrict(pc);
}

template bool sweep_tma<double, double>(sg_precond*, const double*, double*, int, bool, bool,
                                        const int*);
template bool sweep_tma<double, float>(sg_precond*, const double*, float*, int, bool, bool,
                                       const int*);
template bool sweep_tma<float, float>(sg_precond*, const float*, float*, int, bool, bool,
                                      const int*);
template bool sweep_tma4<double, float>(sg_precond*, const double*, float*, long long, const int*);
template bool sweep_tma4<float, float>(sg_precond*, const float*, float*, long long, const int*);

}  // namespace sg

namespace sg {

// Host check of the TMA-fed sweep's data -- what a debug build's bounds
// asserts in the kernel would test, done on the host so that no check can
// fault a GPU: the level records are read back and
//  * every row slot of a level is a real row of the subdomain and every
//    column slot a real row or the zero slot (all inside the shared vector);
//  * every column a row reads was computed by an earlier level of the same
//    sweep (forward: the lower triangle; backward: the upper), i.e. the level
//    schedule respects the factor's dependences;
//  * every level's record lies inside its group's ring bytes and inside the
//    ring, each group is issued before the level that waits for it, and no
//    group overwrites ring bytes or re-arms an mbarrier of a group that a
//    later level still reads; each group's stream bytes match its records'
//    packed offsets.
// plant = 1 (testing) first corrupts one column slot of the host copy.
// Returns the number of violations found (0: all hold).
static long long plan_check(sg_precond* pc, const RingPlan& plan, int plant);

long long sweep_check(sg_precond* pc, int plant) {
    if (!pc->use_rec || pc->rec_depth == 0) return 0;
    long long bad = plan_check(pc, pc->ring1, plant);
    if (pc->ring4.ready) bad += plan_check(pc, pc->ring4, 0);
    return bad;
}

static long long plan_check(sg_precond* pc, const RingPlan& plan, int plant) {
    cudaStream_t st = pc->ctx->stream;
    std::vector<unsigned char> rec((size_t)pc->rec_total);
    SG_CUDA(cudaMemcpyAsync(rec.data(), pc->rec_d.p, rec.size(), cudaMemcpyDeviceToHost, st));
    SG_CUDA(cudaStreamSynchronize(st));
    const int sf = rec_value_bytes(pc);
    const RingSub* subs = reinterpret_cast<const RingSub*>(plan.sub.data());
    const int* ent = plan.ent.data();
    const int* grp = plan.grp.data();
    long long bad = 0;
    bool planted = false;
    std::vector<char> done;
    for (int s = 0; s < pc->nparts; ++s) {
        const SubInfo& inf = pc->h_info[s];
        const RingSub& r = subs[s];
        const int nf = inf.nlev_f, T = inf.nlev_f + inf.nlev_b, n = inf.n, p = inf.tshift;
        const int zero_slot = tslot(n, p);
        // slot -> is it a real row
        std::vector<char> real((size_t)zero_slot + 1, 0);
        for (int li = 0; li < n; ++li) real[tslot(li, p)] = 1;
        // ---- records: bounds and dependences
        for (int dir = 0; dir < 2; ++dir) {
            done.assign((size_t)zero_slot + 1, 0);
            const int w = dir == 0 ? inf.wl : inf.wu;
            const int nl = dir == 0 ? inf.nlev_f : inf.nlev_b;
            for (int l = 0; l < nl; ++l) {
                const int i = (dir == 0 ? inf.lev_off_f : inf.lev_off_b) + l;
                const int c = dir == 0 ? pc->h_lev_ptr_f[i + 1] - pc->h_lev_ptr_f[i]
                                       : pc->h_lev_ptr_b[i + 1] - pc->h_lev_ptr_b[i];
                const int C = dir == 0 ? pc->h_rec_rows_f[i] : pc->h_rec_rows_b[i];
                const int nq = pc->rec_rows && rec_is_rows(w) ? c + 1 : c;
                const long long off = dir == 0 ? pc->h_rec_off_f[i] : pc->h_rec_off_b[i];
                const long long bytes = rec_level_bytes(pc, w, dir != 0, c);
                if (C % 8 || c > C || off < 0 || off + bytes > pc->rec_total) {
                    ++bad;
                    continue;
                }
                // slot k of row q: the row itself (0) or its column k - 1
                const bool rows_rec = pc->rec_rows && rec_is_rows(w);
                const int rb = rec_row_bytes(w, dir != 0, sf);
                auto slot = [&](int q, int k) -> uint16_t& {
                    unsigned char* R = rec.data() + off;
                    return rows_rec ? reinterpret_cast<uint16_t*>(R + (size_t)q * rb)[k]
                                    : reinterpret_cast<uint16_t*>(R)[(size_t)k * C + q];
                };
                if (plant && !planted && l > 0 && c > 0 && w > 0) {
                    slot(0, 1) = slot(0, 0);  // a row reading itself: not yet computed
                    planted = true;
                }
                for (int q = 0; q < nq; ++q) {
                    const int rs = slot(q, 0);
                    if (q == c) {  // the row past the end: the unused slot only
                        for (int k = 0; k <= w; ++k)
                            if (slot(q, k) != zero_slot) ++bad;
                        continue;
                    }
                    if (rs >= zero_slot || !real[rs]) {
                        ++bad;
                        continue;
                    }
                    for (int k = 0; k < w; ++k) {
                        const int cs = slot(q, k + 1);
                        if (cs > zero_slot) ++bad;
                        else if (cs != zero_slot && (!real[cs] || !done[cs])) ++bad;
                    }
                }
                for (int q = 0; q < c; ++q)
                    if (slot(q, 0) < zero_slot) done[slot(q, 0)] = 1;
            }
        }
        // ---- ring schedule: simulate the producer and the level loop
        const int G = r.ngrp;
        int issued = r.ninit, e = 0, g = 0;  // groups issued, entry, level
        if (issued > G || r.ngrp_f > G) ++bad;
        for (int j = 0; j < G; ++j) {
            const int* gj = grp + 4 * ((size_t)r.grp_off + j);
            const long long gstart = (unsigned)gj[0];
            const long long gbytes = (long long)(((unsigned)gj[1] & 0xffffu) << 4);
            const long long gpos = (long long)(((unsigned)gj[1] >> 16) << 4);
            if (j >= issued) ++bad;  // waits for a copy not yet issued
            if (gj[2] != e || gpos + gbytes > plan.ring_bytes) ++bad;
            const int e1 = gj[4 + 2] - 1;  // the entry that ends it
            if (e1 >= r.nent || e1 < e) {
                ++bad;
                break;
            }
            while (e < e1 && g < T) {
                const bool back = g >= nf;
                if (back != (j >= r.ngrp_f)) ++bad;
                const int i = back ? inf.lev_off_b + (g - nf) : inf.lev_off_f + g;
                const int w = back ? inf.wu : inf.wl;
                const int c = back ? pc->h_lev_ptr_b[i + 1] - pc->h_lev_ptr_b[i]
                                   : pc->h_lev_ptr_f[i + 1] - pc->h_lev_ptr_f[i];
                const long long B = rec_level_bytes(pc, w, back, c);
                const long long rel = (back ? pc->h_rec_off_b[i] : pc->h_rec_off_f[i]) - r.base;
                const bool rows = pc->rec_rows && rec_is_rows(w);
                const int step = rows ? std::max(1, plan.level_threads / plan.R) : c;
                const int rb = rec_row_bytes(w, back, sf);
                // the ring copy holds the whole record, in this group's bytes
                const long long at = gpos + rel - gstart;
                if (rel < gstart || rel + B > gstart + gbytes) ++bad;
                for (int q = 0; q < c && e < e1; q += step, ++e) {
                    const int* m = ent + 2 * ((size_t)r.ent_off + e);
                    if ((m[0] & 0xffff) != c - q || (m[0] >> 16) != (q + step >= c ? 1 : 0) ||
                        m[1] != at + (rows ? (long long)q * rb : 0))
                        ++bad;
                }
                ++g;
            }
            if (e != e1 || ent[2 * ((size_t)r.ent_off + e1)] != 0) ++bad;
            e = e1 + 1;
            // issued after group j: what the new groups overwrite must be done
            for (int k = issued; k < gj[3] && k < G; ++k) {
                const int* gk = grp + 4 * ((size_t)r.grp_off + k);
                const long long kb = (long long)(((unsigned)gk[1] & 0xffffu) << 4);
                const long long kp = (long long)(((unsigned)gk[1] >> 16) << 4);
                for (int q = j + 1; q < k; ++q) {
                    const int* gq = grp + 4 * ((size_t)r.grp_off + q);
                    const long long qb = (long long)(((unsigned)gq[1] & 0xffffu) << 4);
                    const long long qp = (long long)(((unsigned)gq[1] >> 16) << 4);
                    if (kp < qp + qb && qp < kp + kb) ++bad;
                }
                if (k >= RING_NBAR && k - RING_NBAR > j) ++bad;
            }
            if (gj[3] > issued) issued = gj[3];
        }
        if (g != T || (issued != G && T > 0)) ++bad;  // every level, every group
        // groups issued at once never overlap each other
        for (int k = 0; k < r.ninit && k < G; ++k)
            for (int q = 0; q < k; ++q) {
                const int *gk = grp + 4 * ((size_t)r.grp_off + k), *gq = grp + 4 * ((size_t)r.grp_off + q);
                const long long kb = (long long)(((unsigned)gk[1] & 0xffffu) << 4), kp = (long long)(((unsigned)gk[1] >> 16) << 4);
                const long long qb = (long long)(((unsigned)gq[1] & 0xffffu) << 4), qp = (long long)(((unsigned)gq[1] >> 16) << 4);
                if (kp < qp + qb && qp < kp + kb) ++bad;
            }
    }
    if (plant && !planted) ++bad;  // nothing to corrupt: report it as found
    return bad;
}

}  // namespace sg
