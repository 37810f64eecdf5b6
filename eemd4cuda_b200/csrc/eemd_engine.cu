// eemd_engine.cu -- sm_100a EEMD engine: kernels and the C ABI (include/eemd_b200.h).
//
// Reference algorithm (misureaudio/EEMD4CUDA):
//   emd_ref.py:31-48    interior tridiagonal system of the natural cubic spline
//   emd_ref.py:50-65    no-pivot Thomas solve
//   emd_ref.py:67-75    spline evaluation (searchsorted interval, cubic in a, b)
//   emd_ref.py:77-103   envelope through strict maxima / minima, mirror ends
//   emd_ref.py:108-156  emd_1d: IMF loop, sift loop, SD stop rule
//   emd_gpu.py:120-285  numba kernel: same loop, one block per trial
//   emd_gpu_v5_dsbt.py:51-74, 77-115  seam-window Thomas and tile extrema scan
//   emd_par.py:198-254  ensemble noise and per-mode masked mean
//
// Numerics.  exact=1 reproduces the reference's float64 operation order
// (separately rounded products, IEEE divisions, serial-Thomas recurrences;
// the file is compiled with --fmad=false so the compiler never contracts
// a*b+c).  exact=0 uses explicit fma(), a Newton-refined reciprocal per row,
// a seam-window elimination of five rows per lane whose forward (c, d) meet
// the neighbouring lanes' in shared memory, and the monomial form of each
// spline interval.
#include "../../include/eemd_b200.h"
#include "eemd_internal.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <memory>
#include <mutex>
#include <new>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

namespace cg = cooperative_groups;

namespace eemd {

// ---------------------------------------------------------------------------
// small device helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ void raise_error(Header* h, int code, int info) {
    if (atomicCAS(&h->error, 0, code) == 0) h->error_info = info;
}

template <typename T>
__device__ __forceinline__ double ldv(const void* p, int64_t i) {
    return (double)(static_cast<const T*>(p)[i]);
}

// value rounded to the storage type, held in double
template <typename T>
__device__ __forceinline__ double rnd(double v) { return (double)(T)v; }

// fused multiply-add in the storage type
__device__ __forceinline__ float fmat(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmat(double a, double b, double c) { return __fma_rn(a, b, c); }

// 1/x: the hardware's gross approximation (the upper 32 bits of a double, relative
// error below 2^-19.9 over 2^30 mantissas) refined by one Newton step on
// f(y) = 1/y - x, y <- y + y(1 - xy), which squares it: below 2^-39.8.
__device__ __forceinline__ double fast_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, e, y);
}

// Asynchronous global->shared copies (sm_80+ cp.async): a thread issues its
// copies, commits them as a group and later waits for the group.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
// 256-bit global accesses (sm_100): a lane's run of samples, 32-byte aligned.
// The loads leave L1 to the interval records (samples are read once per step).
__device__ __forceinline__ void ld256(const float* p, float (&v)[8]) {
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ void ld256(const double* p, double (&v)[4]) {
    asm volatile("ld.global.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];\n"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                 : "l"(p));
}
__device__ __forceinline__ void st256(float* p, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};\n" ::"f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st256(double* p, const double (&v)[4]) {
    asm volatile("st.global.v4.f64 [%4], {%0, %1, %2, %3};\n" ::"d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]), "l"(p)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// emd_ref.py:67-75 (and emd_gpu.py:96-100), reference operation order
__device__ __forceinline__ double spline_exact(double t, double tl, double tr, double yl, double yr,
                                               double Ml, double Mr) {
    double h = tr - tl;
    double a = (tr - t) / h;
    double b = (t - tl) / h;
    double a3 = a * a * a;
    double b3 = b * b * b;
    return (a * yl + b * yr) + (((a3 - a) * Ml + (b3 - b) * Mr) * (h * h)) / 6.0;
}

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) and Box-Muller normals
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
    const uint32_t W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(M0, c.x), lo0 = M0 * c.x;
        uint32_t hi1 = __umulhi(M1, c.z), lo1 = M1 * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += W0;
        k.y += W1;
    }
    return c;
}

// standard normal numbers for samples t (even) and t + 1 of (signal, trial): the
// two outputs of one Box-Muller transform
__device__ __forceinline__ double2 philox_pair(uint64_t seed, int signal, int trial, int64_t t) {
    uint4 ctr = make_uint4((uint32_t)(t >> 1), (uint32_t)trial, (uint32_t)signal, 0x45454D44u);
    uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    uint4 r = philox4x32_10(ctr, key);
    uint64_t a = (((uint64_t)r.x << 32) | r.y) >> 11;
    uint64_t b = (((uint64_t)r.z << 32) | r.w) >> 11;
    double u1 = ((double)a + 1.0) * 0x1.0p-53;  // (0, 1]
    double u2 = (double)b * 0x1.0p-53;          // [0, 1)
    double rad = sqrt(-2.0 * log(u1));
    double s, c;
    sincospi(2.0 * u2, &s, &c);
    return make_double2(rad * c, rad * s);
}

// (called, not inlined, in the float32 kernel: at 128 registers the transform's
// inlined float64 functions cost the sifting steps 2 %; at 168 the call does)
__device__ __noinline__ double2 philox_pair_call(uint64_t seed, int signal, int trial, int64_t t) {
    return philox_pair(seed, signal, trial, t);
}

template <typename T>
__device__ __forceinline__ double2 philox_normals(uint64_t seed, int signal, int trial, int64_t t) {
    if constexpr (sizeof(T) == 4) return philox_pair_call(seed, signal, trial, t);
    else return philox_pair(seed, signal, trial, t);
}

// standard normal number for sample t of (signal, trial)
template <typename T>
__device__ __forceinline__ double philox_normal(uint64_t seed, int signal, int trial, int64_t t) {
    const double2 z = philox_normals<T>(seed, signal, trial, t & ~(int64_t)1);
    return (t & 1) ? z.y : z.x;
}

// out[e][t] = the standard normal the Philox noise mode adds to trial
// trial_begin + e of signal `signal` at sample t (before the eps*std(x) scale)
__global__ void k_philox_fill(uint64_t seed, int signal, int trial_begin, int trials, int64_t n, double* out) {
    const int64_t total = (int64_t)trials * n;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = philox_normal<double>(seed, signal, trial_begin + (int)(i / n), i % n);
}

// ---------------------------------------------------------------------------
// block reductions (fixed order => deterministic)
// ---------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ double2 block_sum2(double2 v, double2* sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_down_sync(0xffffffffu, v.x, o);
        v.y += __shfl_down_sync(0xffffffffu, v.y, o);
    }
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = (lane < NT / 32) ? sh[lane] : make_double2(0.0, 0.0);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v.x += __shfl_down_sync(0xffffffffu, v.x, o);
            v.y += __shfl_down_sync(0xffffffffu, v.y, o);
        }
    }
    __syncthreads();
    return v;  // valid in thread 0
}

// ---------------------------------------------------------------------------
// k_sigma: per-signal eps*std(x) (population std, emd_par.py:117, 225)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(1024) k_sigma(const SignalDesc* sdesc, const void* xv, double eps,
                                                double* sigma_out) {
    __shared__ double2 sh[32];
    __shared__ double mean_s;
    const int s = blockIdx.x;
    const SignalDesc d = sdesc[s];
    const T* x = static_cast<const T*>(xv) + d.x_off;
    double acc = 0.0;
#pragma unroll 8
    for (int64_t i = threadIdx.x; i < d.n; i += 1024) acc += (double)x[i];
    double2 r = block_sum2<1024>(make_double2(acc, 0.0), sh);
    if (threadIdx.x == 0) mean_s = r.x / (double)d.n;
    __syncthreads();
    const double mean = mean_s;
    acc = 0.0;
#pragma unroll 8
    for (int64_t i = threadIdx.x; i < d.n; i += 1024) {
        const double dv = (double)x[i] - mean;
        acc += dv * dv;
    }
    r = block_sum2<1024>(make_double2(acc, 0.0), sh);
    if (threadIdx.x == 0) sigma_out[s] = eps * sqrt(r.x / (double)d.n);
}

// ---------------------------------------------------------------------------
// per-CTA task context (shared memory)
// ---------------------------------------------------------------------------
constexpr int MAXSEG = MAXC * MAXNW;  // knot segments per task: one per warp of up to MAXC CTAs

struct Xchg {              // one CTA's published step results (DSMEM-visible)
    double2 sd[MAXNW];     // SD partial sums (num, den) of each warp's range, where the stop test reads them
    int cnt[2][MAXNW];     // new knots (maxima, minima) found by each warp
    int err;               // this CTA raised an error during the step: the task stops
};

struct TaskSm {
    int task, n, s0, s1, rank, csize;
    int phase, imf, sift, kpar, src_resid, imf_from_resid;
    int nsift_total, nmode, mode_sifts_cur, flags, step, mode;
    int P[2];                  // current knot totals
    int pref[2][2][MAXSEG + 1];  // [list parity][env]: knots before each (CTA, warp) segment
    int mir[2], p2[2];         // mirror ends in use; knots in mirror space
    int rcur;                  // current residual: 0 = the task's residual array, 1 = slot scratch
    Xchg x[2];                 // step results, by step parity
};

// An error of the running task: recorded in the header (first error wins) and
// in the CTA's step results, which decide() ORs over the cluster so that every
// CTA stops the task at the same step (no further step reads what the failed
// step left behind).
__device__ __forceinline__ void task_error(const Ctx& C, TaskSm& S, int code) {
    raise_error(C.hdr, code, S.task);
    S.x[S.step & 1].err = 1;
}

#ifdef EEMD_CHECKED
// checked build: an interval record index outside [0, hi] is reported and
// clamped instead of read out of bounds
#define EEMD_CHECK_IV(k, hi)                                     \
    do {                                                         \
        if ((k) < 0 || (k) > (hi)) {                             \
            task_error(C, S, EEMD_E_KNOT_OVERFLOW);              \
            (k) = max(0, min((k), (hi)));                        \
        }                                                        \
    } while (0)
#else
#define EEMD_CHECK_IV(k, hi) \
    do {                     \
    } while (0)
#endif

// Sweep geometry for storage type T.  A warp tile is WT = 32*RUN samples: each
// lane owns a run of RUN consecutive samples, 32 bytes, which one 256-bit load
// brings into registers (and one 256-bit store writes back).
template <typename T>
struct Geo {
    static constexpr int RUN = sizeof(T) == 4 ? 8 : 4;  // consecutive samples per lane
    static constexpr int WT = 32 * RUN;                 // samples per warp tile
};

__host__ __device__ inline int stage_pad(int k) { return k + (k >> 4); }

__host__ __device__ inline size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }

// rows of one fast-solve pass: 32 lanes of FAST_B rows
constexpr int FAST_ROWS = 32 * FAST_B;
// largest seam halo of the fast solve, and the knots one fast pass stages:
// its rows, the left halo and the two knots past the last row
constexpr int FAST_SMAX = 64;
constexpr int WSCAP_FAST = FAST_ROWS + FAST_SMAX + 3;
static_assert(WSCAP_FAST <= 2 * FAST_ROWS, "the slopes of a pass fit the (c, d) area");

// Per-warp staging area of the solve.  What the CTAs' areas leave of the SM's
// on-chip memory is L1, which the sweep's record gathers live in.
//   exact: slopes (double), knot times (int) and values (double) of WSCAP
//     knots, one slot of padding every 16 (the lanes of a pass read knots one
//     window of 16 apart, which would share a bank);
//   fast: the rows (diagonal, right-hand side) and the knots (float32: pairs
//     of time and value; float64: times, then values) of WSCAP_FAST knots, and
//     the forward (c, d) of a pass's rows, whose space first holds the slopes.
//     Lanes read FAST_B elements apart: odd strides hit distinct banks.
__host__ __device__ inline size_t wsolve_bytes(size_t bt, bool exact) {
    if (exact) {
        const size_t sp = (size_t)stage_pad(WSCAP);
        return align16(sp * 8) + align16(sp * 4) + align16(sp * 8);
    }
    return (size_t)WSCAP_FAST * 16 + align16((size_t)WSCAP_FAST * 4) + align16((size_t)WSCAP_FAST * bt) + 16 +
           (size_t)FAST_ROWS * 16;
}

// dynamic shared memory of k_emd: the solve's per-warp areas (the sweep works in registers)
__host__ __device__ inline size_t smem_bytes(int bt, bool exact, int nw) {
    return nw * wsolve_bytes((size_t)bt, exact);
}

// ---------------------------------------------------------------------------
// segmented knot lists: real knot i lives in segment r = seg_of(i) at
// position i - pref[r] of that segment's list
// ---------------------------------------------------------------------------
struct Slot {
    int32_t* kt;   // knot lists (segmented): float32 storage pairs of (index, value),
    void* ky;      //   float64 storage indices here and values in ky
    void* M;       // interval records, mirror space (struct Rec)
    void* w1;      // scratch h buffer of the running task (storage type)
    void* w0;      // a second one, or null (the IMF slot serves)
    void* r1;      // second residual buffer of the running task (storage type)
    uint32_t* ri;  // run records [2 parity][runs] (run_record)
};

__device__ __forceinline__ int64_t knot_index(const Ctx& C, int par, int env, int seg, int i) {
    return ((int64_t)((par * 2 + env) * C.csize * C.nw + seg)) * C.segcap + i;
}

// segment holding real knot i: largest r in [lo, hi) with pref[r] <= i
__device__ __forceinline__ int seg_of(const int* pref, int lo, int hi, int i) {
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pref[mid] <= i) lo = mid; else hi = mid;
    }
    return lo;
}

// element offset of real knot i in the current knot lists
__device__ __forceinline__ int64_t real_off(const Ctx& C, const TaskSm& S, int env, int i) {
    const int* pr = S.pref[S.kpar][env];
    const int a = S.rank * C.nw, b = a + C.nw;  // most lookups fall in the CTA's own segments
    const int r = (i >= pr[a] && i < pr[b]) ? seg_of(pr, a, b, i) : seg_of(pr, 0, S.csize * C.nw, i);
    return knot_index(C, S.kpar, env, r, i - pr[r]);
}

// knot at element offset o of the lists: float32 storage keeps (index, value)
// pairs, so a knot is one 8-byte access; float64 storage two arrays
template <typename T>
__device__ __forceinline__ void get_knot(const Slot& sl, int64_t o, int& t, T& y) {
    if constexpr (sizeof(T) == 4) {
        const int2 k = __ldcg(reinterpret_cast<const int2*>(sl.kt) + o);
        t = k.x;
        y = __int_as_float(k.y);
    } else {
        t = __ldcg(sl.kt + o);
        y = __ldcg(static_cast<const T*>(sl.ky) + o);
    }
}
template <typename T>
__device__ __forceinline__ void put_knot(const Slot& sl, int64_t o, int t, T y) {
    if constexpr (sizeof(T) == 4) {
        reinterpret_cast<int2*>(sl.kt)[o] = make_int2(t, __float_as_int(y));
    } else {
        sl.kt[o] = t;
        static_cast<T*>(sl.ky)[o] = y;
    }
}

template <typename T>
__device__ __forceinline__ void real_knot(const Ctx& C, const Slot& sl, const TaskSm& S, int env, int i,
                                          int& t, double& y) {
    T v;
    get_knot<T>(sl, real_off(C, S, env, i), t, v);
    y = (double)v;
}

// Mirror space (emd_ref.py:92-96): with mir = 1 (three knots or more) the list
// is [2t0-t1, t0..t_{P-1}, 2t_{P-1}-t_{P-2}] with values [y1, y.., y_{P-2}].
// The two virtual knots of a staged range are formed from their neighbours
// once those have arrived (get, set: a staged knot).
template <typename Get, typename Set>
__device__ __forceinline__ void mirror_ends(const TaskSm& S, int env, int rlo, int kcount, int lane, Get get, Set set) {
    if (!S.mir[env] || lane != 0) return;
    if (rlo == 0) {
        const auto a = get(1), b = get(2);
        set(0, 2 * a.t - b.t, b.y);
    }
    if (rlo + kcount == S.P[env] + 2) {
        const auto a = get(kcount - 2), b = get(kcount - 3);
        set(kcount - 1, 2 * a.t - b.t, b.y);
    }
}
template <typename T>
struct KnotVal {
    int t;
    T y;
};

// Exact mode: stage the mirror-space knots rlo .. rlo+kcount-1 (lane-strided);
// each lane finds the segment of its first real knot by binary search and then
// walks forward, since its later knots follow in the same or later segments.
__device__ __forceinline__ void stage_exact(const Ctx& C, const Slot& sl, TaskSm& S, int env, int rlo, int kcount,
                                            int* skt, double* sky, int lane) {
    const int* pr = S.pref[S.kpar][env];
    const int nseg = S.csize * C.nw;
    const int mir = S.mir[env], P = S.P[env];
    int r = -1;
    for (int k = lane; k < kcount; k += 32) {
        int i2 = rlo + k;
        int* kt_s = &skt[stage_pad(k)];
        double* ky_s = &sky[stage_pad(k)];
        if (mir) {
            if (i2 == 0 || i2 == P + 1) continue;  // the virtual knots follow from their staged neighbours
            i2 -= 1;
        }
        if (r < 0) r = seg_of(pr, 0, nseg, i2);
        while (r + 1 < nseg && i2 >= pr[r + 1]) ++r;
#ifdef EEMD_CHECKED
        if (i2 < 0 || i2 >= P || i2 - pr[r] >= C.segcap) {
            task_error(C, S, EEMD_E_KNOT_OVERFLOW);
            continue;
        }
#endif
        const int64_t o = knot_index(C, S.kpar, env, r, i2 - pr[r]);
        cp_async4(kt_s, sl.kt + o);
        cp_async8(ky_s, static_cast<const double*>(sl.ky) + o);
    }
}

// Staged knots of the fast solve
template <typename T>
struct Knots {
    int* t;     // float32: pairs (time, value bits); float64: times
    double* v;  // float64: values
    __device__ __forceinline__ int time(int k) const { return sizeof(T) == 4 ? t[2 * k] : t[k]; }
    __device__ __forceinline__ T val(int k) const {
        if constexpr (sizeof(T) == 4) return __int_as_float(t[2 * k + 1]);
        else return v[k];
    }
    __device__ __forceinline__ void get(int k, int& tk, T& y) const {
        if constexpr (sizeof(T) == 4) {
            const int2 p = reinterpret_cast<const int2*>(t)[k];
            tk = p.x;
            y = __int_as_float(p.y);
        } else {
            tk = t[k];
            y = v[k];
        }
    }
    __device__ __forceinline__ void set(int k, int tk, T y) const {
        if constexpr (sizeof(T) == 4) {
            reinterpret_cast<int2*>(t)[k] = make_int2(tk, __float_as_int(y));
        } else {
            t[k] = tk;
            v[k] = y;
        }
    }
    __device__ __forceinline__ void copy(int k, const Slot& sl, int64_t o) const {  // asynchronously
        if constexpr (sizeof(T) == 4) {
            cp_async8(t + 2 * k, sl.kt + 2 * o);
        } else {
            cp_async4(t + k, sl.kt + o);
            cp_async8(v + k, static_cast<const double*>(sl.ky) + o);
        }
    }
};

// Fast mode: stage the mirror-space knots rlo .. rlo+kcount-1.  The real knots
// among them lie in consecutive (CTA, warp) segments: up to STAGE_PIECES
// segments are copied piece by piece (a pass of dense knots spans one or two),
// more by a lane-strided walk as in stage_exact (the sparse knots of the late
// IMFs, a few per segment).
constexpr int STAGE_PIECES = 4;
template <typename T>
__device__ __forceinline__ void stage_fast(const Ctx& C, const Slot& sl, TaskSm& S, int env, int rlo, int kcount,
                                           const Knots<T>& K, int lane) {
    const int* pr = S.pref[S.kpar][env];
    const int nseg = S.csize * C.nw;
    const int mir = S.mir[env], P = S.P[env];
    int a = max(rlo - mir, 0);                       // real knots [a, b)
    const int b = min(rlo + kcount - mir, P);
    const int shift = mir - rlo;                     // staging position of real knot i: i + shift
    // segments of the first and last knot: the last one that starts at or before it
    int ra = 0, rb = 0;
#pragma unroll
    for (int k = 0; k < (MAXSEG + 31) / 32; ++k) {
        const int sg = 32 * k + lane;
        const int v = sg < nseg ? pr[sg] : INT_MAX;
        ra += __popc(__ballot_sync(0xffffffffu, v <= a));
        rb += __popc(__ballot_sync(0xffffffffu, v <= b - 1));
    }
    ra -= 1;
    rb -= 1;
    if (rb - ra < STAGE_PIECES) {
        for (int r = ra; r <= rb; ++r) {
            const int e = min(b, pr[r + 1]);
            const int64_t o = knot_index(C, S.kpar, env, r, 0) - pr[r];
#ifdef EEMD_CHECKED
            if (a < pr[r] || e - pr[r] > C.segcap || a + shift < 0 || e + shift > WSCAP_FAST) {
                task_error(C, S, EEMD_E_KNOT_OVERFLOW);
                return;
            }
#endif
            for (int i = a + lane; i < e; i += 32) K.copy(i + shift, sl, o + i);
            a = e;
        }
    } else {
        int r = -1;
        for (int i = a + lane; i < b; i += 32) {
            if (r < 0) r = seg_of(pr, 0, nseg, i);
            while (r + 1 < nseg && i >= pr[r + 1]) ++r;
#ifdef EEMD_CHECKED
            if (i - pr[r] >= C.segcap || i + shift < 0 || i + shift >= WSCAP_FAST) {
                task_error(C, S, EEMD_E_KNOT_OVERFLOW);
                continue;
            }
#endif
            K.copy(i + shift, sl, knot_index(C, S.kpar, env, r, i - pr[r]));
        }
    }
}

// ---------------------------------------------------------------------------
// solve: decay-seamed block Thomas over the cluster
// ---------------------------------------------------------------------------
// Row i (mirror space, i = 0..n-1 for M2[i+1]) from staged knots k = i - base:
//   H0 = t_{i+1}-t_i, H1 = t_{i+2}-t_{i+1}, d = 2(H0+H1), l = H0 (i>=1),
//   u = H1 (i<=n-2), r = 6(slope_{i+1} - slope_i)          (emd_ref.py:31-48)
// The sweeps slide along the rows: each row loads one new knot and one slope.
struct Row {
    double dg, l, u, r;
};

__device__ __forceinline__ Row row_of(int ta, int tb, int tc, double sa, double sb, int i, int n) {
    const double H0 = (double)(tb - ta), H1 = (double)(tc - tb);
    Row w;
    w.dg = 2.0 * (H0 + H1);
    w.l = (i >= 1) ? H0 : 0.0;
    w.u = (i <= n - 2) ? H1 : 0.0;
    w.r = 6.0 * (sb - sa);
    return w;
}

#define SKT(k) skt[stage_pad(k)]
#define SSL(k) ssl[stage_pad(k)]

// Interval records of one envelope in mirror space: for interval k (knots k,
// k+1) the four coefficients c[4k..4k+3] (fast: y_k, c1, c2, c3 of the
// monomial; exact: y_k, M_k), one 16-byte (float32) or 32-byte (float64) vector
// that the sweep gathers with one load, and apart from them the knot's sample
// index t[k], read once per run of samples.
template <typename T>
struct Rec {
    T* c;
    int32_t* t;
    __device__ __forceinline__ Rec(void* M, int env, int kcap) {
        c = static_cast<T*>(M) + (int64_t)env * 4 * kcap;
        t = reinterpret_cast<int32_t*>(static_cast<T*>(M) + (int64_t)8 * kcap) + (int64_t)env * kcap;
    }
    __device__ __forceinline__ void put(int k, int tk, T y, T c1, T c2, T c3) const {
        t[k] = tk;
        if constexpr (sizeof(T) == 4) {
            reinterpret_cast<float4*>(c)[k] = make_float4(y, c1, c2, c3);
        } else {
            const T v[4] = {y, c1, c2, c3};
            st256(c + 4 * (int64_t)k, v);
        }
    }
};

// exact: forward elimination from w0 (outer coupling dropped), back
// substitution from w1; identical recurrences to serial Thomas (emd_ref.py:50-65).
// Writes (t_k, y_k, M_k) of the owned knots k = o0+1 .. o1+1 (+ both end knots).
template <typename T>
__device__ void window_exact(const Ctx& C, const int* skt, const T* sky, const double* ssl, int base,
                             int n, int w, const Rec<T>& R, int p2) {
    const int B = C.B, S = C.S;
    const int o0 = w * B;
    const int o1 = min(n, o0 + B) - 1;
    const int w0 = max(0, o0 - S);
    const int w1 = min(n - 1, o1 + S);
    const int64_t gthreads = (int64_t)gridDim.x * blockDim.x;
    double2* sc = C.scr + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double cp = 0.0, dp = 0.0;
    int ta = SKT(w0 - base), tb = SKT(w0 + 1 - base);
    double sa = SSL(w0 - base);
    for (int i = w0; i <= w1; ++i) {
        const int tc = SKT(i + 2 - base);
        const double sb = SSL(i + 1 - base);
        const Row rw = row_of(ta, tb, tc, sa, sb, i, n);
        const double c = (i == w1) ? 0.0 : rw.u / (rw.dg - rw.l * cp);
        const double dv = (rw.r - rw.l * dp) / (rw.dg - rw.l * cp);
        if (i >= o0) sc[(int64_t)(i - o0) * gthreads] = make_double2(c, dv);
        cp = c;
        dp = dv;
        ta = tb;
        tb = tc;
        sa = sb;
    }
    auto put = [&](int k, double Mk) {
        R.put(k, SKT(k - base), sky[stage_pad(k - base)], (T)Mk, (T)0, (T)0);
    };
    double xv = dp;
    if (w1 <= o1) put(w1 + 1, xv);
    for (int i = w1 - 1; i >= o0; --i) {
        const double2 cd = sc[(int64_t)(i - o0) * gthreads];
        xv = cd.y - cd.x * xv;
        if (i <= o1) put(i + 1, xv);
    }
    if (o0 == 0) put(0, 0.0);
    if (o1 == n - 1) put(p2 - 1, 0.0);
}

#undef SKT
#undef SSL

// fast: each lane owns FAST_B consecutive rows of a pass.  The forward
// elimination (coupling dropped S rows before the lane's first row, where the
// influence of the neglected rows has decayed like prod c_i) stores (c_i, d_i)
// of the owned rows in the warp's shared memory; after __syncwarp each
// committing lane back-substitutes from S rows past its last row (x there
// truncated to d, the neglected term decaying the same way) down to its first
// row and writes the monomial interval records of its rows.  The lanes of a
// pass's last H = ceil(S / FAST_B) windows only provide that right halo
// (unless the pass reaches the envelope's last row) and are solved for good
// by the next pass.  Per owned row: (S + FAST_B) / FAST_B eliminated rows and
// as many back-substitution steps (one fused multiply-add each).
//
// A row is formed once per pass, by the lane that owns its knot, and read by
// the (S + FAST_B) / FAST_B lanes that eliminate it: {d_i, r_i} in one 16-byte
// load, with d_i = 2 (H_i + H_{i+1}) and r_i = 6 (slope_{i+1} - slope_i).  The
// off-diagonals follow from d_i alone, H_{i+1} = d_i / 2 - H_i, exactly (they
// are differences of sample indices).  The first and last row need no special
// case: the terms their outer couplings multiply are zero.  The elimination is
// a chain of dependent float64 operations at 13 to 16 warps per SM; forming a
// row in every lane that eliminates it (three conversions and four operations
// more per row, and two loads) made k_emd 48 000 x 100 float32 3.96 ms, this
// form 3.53; 48 000 x 64 float64 1.19 and 1.10; 2^22 x 64 float64 349 and 330.
template <typename T>
__device__ __forceinline__ void window_fast_fwd(const Knots<T>& K, const double2* rows, int base, int n, int w,
                                                int S, double2* cd, int cdbase) {
    const int o0 = w * FAST_B;
    const int o1 = min(n, o0 + FAST_B) - 1;
    const int r0 = max(0, o0 - S);
    double cp = 0.0, dp = 0.0;
    double l = (double)(K.time(r0 + 1 - base) - K.time(r0 - base));  // H_i
    auto step = [&](int i) {
        const double2 rw = rows[i - base];
        const double u = fma(0.5, rw.x, -l);
        const double inv = fast_rcp(fma(-l, cp, rw.x));
        dp = fma(-l, dp, rw.y) * inv;
        cp = u * inv;
        l = u;
    };
#pragma unroll 4
    for (int i = r0; i < o0; ++i) step(i);
#pragma unroll
    for (int k = 0; k < FAST_B; ++k) {
        if (o0 + k <= o1) {
            step(o0 + k);
            cd[o0 + k - cdbase] = make_double2(cp, dp);
        }
    }
}

// Back substitution of window w (rows o0..o1; x_i = M at mirror knot i+1) and
// its interval records: interval i+1 for every owned row i (knots i+1, i+2),
// and interval 0 (M_0 = 0 at the natural end) for the first window.
template <typename T>
__device__ __forceinline__ void window_fast_back(const Knots<T>& K, int base, int n, int w, int S, const double2* cd,
                                                 int cdbase, const Rec<T>& R) {
    const int o0 = w * FAST_B;
    const int o1 = min(n, o0 + FAST_B) - 1;
    const int rh = min(n - 1, o1 + S);
    double xn = 0.0;  // x_{i+1}: zero past the natural end (M = 0) or at the truncation
#pragma unroll 4
    for (int i = rh; i > o1; --i) {
        const double2 c = cd[i - cdbase];
        xn = fma(-c.x, xn, c.y);
    }
    // monomial record of interval k (knots k, k+1; M_k = Ma, M_{k+1} = Mb):
    // y_k + s(c1 + s(c2 + s c3)), s = t - t_k, c1 = slope - h(2Ma + Mb)/6,
    // c2 = Ma/2, c3 = (Mb - Ma)/(6h)
    int t1;
    T y1;
    K.get(o1 + 2 - base, t1, y1);
    auto put = [&](int k, double Ma, double Mb) {
        int t0;
        T y0;
        K.get(k - base, t0, y0);
        const double h = (double)(t1 - t0), rh_ = fast_rcp(h);
        const double slope = ((double)y1 - (double)y0) * rh_;
        R.put(k, t0, y0, (T)fma(-h * (1.0 / 6.0), fma(2.0, Ma, Mb), slope), (T)(0.5 * Ma),
              (T)((Mb - Ma) * rh_ * (1.0 / 6.0)));
        t1 = t0;
        y1 = y0;
    };
#pragma unroll
    for (int k = FAST_B - 1; k >= 0; --k) {
        const int i = o0 + k;
        if (i <= o1) {
            const double2 c = cd[i - cdbase];
            const double xi = fma(-c.x, xn, c.y);
            put(i + 1, xi, xn);
            xn = xi;
        }
    }
    if (o0 == 0) put(0, 0.0, xn);
}

template <typename T, bool EXACT, int NW>
__device__ void solve_task(const Ctx& C, const Slot& sl, TaskSm& S, unsigned char* smem) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
#ifdef EEMD_TRACE
    unsigned long long scyc[3] = {0, 0, 0};
    long long smark = clock64();
#define SUB(k)                                          \
    do {                                                \
        const long long now_ = clock64();               \
        scyc[k] += (unsigned long long)(now_ - smark);  \
        smark = now_;                                   \
    } while (0)
#else
#define SUB(k) \
    do {       \
    } while (0)
#endif
    // one or two knots: a constant or the straight line through them (M = 0)
    for (int env = 0; env < 2; ++env) {
        const int p2 = S.p2[env];
        if (p2 - 2 > 0 || S.rank != 0 || tid >= p2) continue;
        const Rec<T> R(sl.M, env, C.kcap);
        int tk, t1;
        double yk, y1;
        real_knot<T>(C, sl, S, env, tid, tk, yk);  // (no mirror knots below three)
        T c1 = (T)0;
        if (!EXACT && tid + 1 < p2) {
            real_knot<T>(C, sl, S, env, tid + 1, t1, y1);
            c1 = (T)((y1 - yk) / (double)(t1 - tk));
        }
        R.put(tid, tk, (T)yk, c1, (T)0, (T)0);
    }
    // The windows of both envelopes form one list (envelope 0 first); CTA r
    // takes an even share of it and each warp a contiguous part of the CTA's
    // share, solved 32 windows (one per lane) at a time from the warp's own
    // knot staging area: no block-wide barriers.
    const int Bw = EXACT ? C.B : FAST_B;
    const int n0 = max(0, S.p2[0] - 2), n1 = max(0, S.p2[1] - 2);
    const int nw0 = (n0 + Bw - 1) / Bw, nw1 = (n1 + Bw - 1) / Bw;
    const int nwt = nw0 + nw1;
    const int ca = (int)((int64_t)S.rank * nwt / S.csize), cb = (int)((int64_t)(S.rank + 1) * nwt / S.csize);
    const int wa = ca + (int)((int64_t)wid * (cb - ca) / NW);
    const int wb = ca + (int)((int64_t)(wid + 1) * (cb - ca) / NW);
    unsigned char* ws = smem + (size_t)wid * wsolve_bytes(sizeof(T), EXACT);
    // exact: slopes, knot times, knot values
    double* ssl = reinterpret_cast<double*>(ws);
    int* skt = reinterpret_cast<int*>(ws + align16(stage_pad(WSCAP) * 8));
    double* sky = reinterpret_cast<double*>(ws + align16(stage_pad(WSCAP) * 8) + align16(stage_pad(WSCAP) * 4));
    // fast: rows, (c, d) or slopes, knots
    double2* rows = reinterpret_cast<double2*>(ws);
    double2* cd = rows + WSCAP_FAST;
    Knots<T> K;
    K.t = reinterpret_cast<int*>(cd + FAST_ROWS);
    K.v = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(K.t) + align16((size_t)WSCAP_FAST * 4));
    // exact: windows of B rows with halos on both sides, one per lane;
    // fast: lanes of FAST_B rows, the last H lanes of a pass as right halo
    const int H = (C.S + FAST_B - 1) / FAST_B;
    const int nlmax = min(32, (WSCAP_FAST - C.S - 3) / FAST_B);
    const int per = min(32, (WSCAP - 2 * C.S - 8) / Bw);  // exact windows per pass
    for (int g = wa; g < wb;) {
        const int env = (g < nw0) ? 0 : 1;
        const int w0 = env ? g - nw0 : g;  // first window of the pass (within its envelope)
        const int nwe = env ? nw1 : nw0;
        const int n = env ? n1 : n0;
        const int p2 = S.p2[env];
        int ncommit, nl, rlo, rhi;
        if (EXACT) {
            ncommit = nl = min(w0 + per, min(nwe, w0 + (wb - g))) - w0;
            rlo = max(0, w0 * Bw - C.S);
            rhi = min(n - 1, min(n, (w0 + nl) * Bw) - 1 + C.S);
        } else {
            const int rem = min(wb - g, nwe - w0);  // this warp's windows left in the envelope
            if (w0 + rem == nwe && rem <= nlmax) {
                ncommit = nl = rem;  // the pass reaches the envelope's last row
            } else {
                ncommit = min(rem, nlmax - H);
                nl = min(nlmax, min(ncommit + H, nwe - w0));
            }
            rlo = max(0, w0 * FAST_B - C.S);
            rhi = min(n - 1, (w0 + nl) * FAST_B - 1);
        }
        const int kcount = rhi + 3 - rlo;  // knots rlo .. rhi+2
        const Rec<T> R(sl.M, env, C.kcap);
        const int w = w0 + lane;
        if constexpr (EXACT) {
            stage_exact(C, sl, S, env, rlo, kcount, skt, sky, lane);
            cp_async_commit();
            cp_async_wait<0>();
            __syncwarp();
            mirror_ends(S, env, rlo, kcount, lane,
                        [&](int k) { return KnotVal<double>{skt[stage_pad(k)], sky[stage_pad(k)]}; },
                        [&](int k, int t, double y) {
                            skt[stage_pad(k)] = t;
                            sky[stage_pad(k)] = y;
                        });
            __syncwarp();
            SUB(0);
            // emd_ref.py:47: (y_{q+1}-y_q)/H_q, the same IEEE division
            for (int k = lane; k + 1 < kcount; k += 32)
                ssl[stage_pad(k)] = (sky[stage_pad(k + 1)] - sky[stage_pad(k)]) /
                                    (double)(skt[stage_pad(k + 1)] - skt[stage_pad(k)]);
            __syncwarp();
            SUB(1);
            if (lane < nl) window_exact<T>(C, skt, sky, ssl, rlo, n, w, R, p2);
        } else {
            stage_fast<T>(C, sl, S, env, rlo, kcount, K, lane);
            cp_async_commit();
            cp_async_wait<0>();
            __syncwarp();
            if (S.mir[env]) {
                mirror_ends(S, env, rlo, kcount, lane,
                            [&](int k) {
                                KnotVal<T> v;
                                K.get(k, v.t, v.y);
                                return v;
                            },
                            [&](int k, int t, T y) { K.set(k, t, y); });
                __syncwarp();
            }
            SUB(0);
            double* slope = reinterpret_cast<double*>(cd);
            for (int k = lane; k + 1 < kcount; k += 32) {
                int ta, tb;
                T ya, yb;
                K.get(k, ta, ya);
                K.get(k + 1, tb, yb);
                slope[k] = ((double)yb - (double)ya) * fast_rcp((double)(tb - ta));
            }
            __syncwarp();
            for (int k = lane; k + 2 < kcount; k += 32) {
                const double d = 2.0 * (double)(K.time(k + 2) - K.time(k));
                rows[k] = make_double2(d, 6.0 * (slope[k + 1] - slope[k]));
            }
            __syncwarp();
            SUB(1);
            if (lane < nl) window_fast_fwd<T>(K, rows, rlo, n, w, C.S, cd, w0 * FAST_B);
            __syncwarp();
            if (lane < ncommit) window_fast_back<T>(K, rlo, n, w, C.S, cd, w0 * FAST_B, R);
        }
        __syncwarp();
        SUB(2);
        g += ncommit;
    }
#ifdef EEMD_TRACE
    if (lane == 0) {
        for (int k = 0; k < 3; ++k) atomicAdd(&C.hdr->sweep_cycles[4 + k], scyc[k]);
    }
#endif
#undef SUB
}

// ---------------------------------------------------------------------------
// sweep: the fused per-segment pass
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ double trial_input(const Ctx& C, const TaskDesc& d, int64_t t) {
    const double xv = ldv<T>(C.x, d.x_off + t);
    switch (C.noise_mode) {
        case EEMD_NOISE_INJECTED: return rnd<T>(xv + ldv<T>(C.noise, d.noise_off + t));
        case EEMD_NOISE_SCALED:
            // the product, then the sum, each rounded (the reference forms beta * w, then x + that)
            return rnd<T>(__dadd_rn(xv, __dmul_rn(C.noise_scale, ldv<T>(C.noise, d.noise_off + t))));
        case EEMD_NOISE_PHILOX:
            return rnd<T>(xv + C.sigma[d.signal] * philox_normal<T>(C.seed, d.signal, d.trial, t));
        default: return xv;  // NONE, PREPERTURBED
    }
}

// One interval of an envelope (fast: monomial; exact: the two end knots).
template <typename T>
struct Iv {
    int k, t0, t1;
    T y0, c1, c2, c3, y1, m1;  // fast: y0 + s(c1 + s(c2 + s c3)); exact: y0, M0 = c1, y1, M1
};

// the four coefficients of interval record k
template <typename T>
__device__ __forceinline__ void load_coef(const T* c, int k, T& y0, T& c1, T& c2, T& c3) {
    if constexpr (sizeof(T) == 4) {
        const float4 a = reinterpret_cast<const float4*>(c)[k];
        y0 = a.x;
        c1 = a.y;
        c2 = a.z;
        c3 = a.w;
    } else {
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];\n"
                     : "=d"(y0), "=d"(c1), "=d"(c2), "=d"(c3)
                     : "l"(c + 4 * (int64_t)k));
    }
}

// loads interval record k (and k+1 in exact mode) of an envelope's records
template <typename T, bool EXACT>
__device__ __forceinline__ void load_iv(Iv<T>& v, const Rec<T>& R, int k) {
    v.k = k;
    v.t0 = R.t[k];
    load_coef<T>(R.c, k, v.y0, v.c1, v.c2, v.c3);
    if (EXACT) {
        T a, b;
        v.t1 = R.t[k + 1];
        load_coef<T>(R.c, k + 1, v.y1, v.m1, a, b);
    }
}

template <typename T, bool EXACT>
__device__ __forceinline__ T iv_eval(const Iv<T>& v, int t) {
    if (EXACT)
        return (T)spline_exact((double)t, (double)v.t0, (double)v.t1, (double)v.y0, (double)v.y1, (double)v.c1,
                               (double)v.m1);
    const T s = (T)(t - v.t0);
    return fmat(s, fmat(s, fmat(s, v.c3, v.c2), v.c1), v.y0);
}

// envelope value at t with `cless` real knots strictly before t: mirror-space
// interval = searchsorted - 1 clipped (emd_ref.py:70), that is (knots before t)
// + mir - 1 clipped to [0, p2 - 2] (where a sample lies outside the virtual
// mirror knots too, the clip gives the same interval); reloads the interval
// record only when the interval changes.  One knot: the constant y of record 0.
template <typename T, bool EXACT>
__device__ __forceinline__ T env_at(const TaskSm& S, Iv<T>& v, const Rec<T>& R, int env, int cless, int t) {
    const int p2 = S.p2[env];
    if (p2 < 2) return R.c[0];
    const int k = max(0, min(cless + S.mir[env] - 1, p2 - 2));
    if (k != v.k) load_iv<T, EXACT>(v, R, k);
    return iv_eval<T, EXACT>(v, t);
}

// a lane's run of RUN samples (nv of them inside the range): one 256-bit
// access when it is whole and p's array is 32-byte aligned, element accesses
// otherwise
template <typename T, int RUN>
__device__ __forceinline__ void load_run(const T* p, T (&v)[RUN], int nv, bool vec) {
    if (vec && nv == RUN) {
        ld256(p, v);
    } else {
#pragma unroll
        for (int i = 0; i < RUN; ++i) v[i] = (i < nv) ? p[i] : (T)0;
    }
}
template <typename T, int RUN>
__device__ __forceinline__ void store_run(T* p, const T (&v)[RUN], int nv, bool vec) {
    if (vec && nv == RUN) {
        st256(p, v);
    } else {
#pragma unroll
        for (int i = 0; i < RUN; ++i)
            if (i < nv) p[i] = v[i];
    }
}
// samples from one IMF row to the next: rows of the workspace start on 32 bytes
template <typename T>
__device__ __forceinline__ int64_t row_stride(int n, int pad) {
    constexpr int A = 32 / (int)sizeof(T);
    return pad ? (n + A - 1) / A * A : n;
}
__device__ __forceinline__ bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }

// value at tile position pos (lane pos/RUN, element pos%RUN), to every lane
template <typename T, int RUN>
__device__ __forceinline__ T tile_at(const T (&v)[RUN], int pos) {
    const int e = pos % RUN;
    T x = v[0];
#pragma unroll
    for (int i = 1; i < RUN; ++i)
        if (e == i) x = v[i];
    return __shfl_sync(0xffffffffu, x, pos / RUN);
}

// Run record of one lane's run, 32 bits: the knots of each kind the tile holds
// before the run (maxima in bits 0-7, minima in 8-15; a tile holds at most
// WT / 2 = 128 of a kind) and the run's knot masks (maxima 16-23, minima
// 24-31).  The reader of a range adds the tiles' totals up itself, so the
// record needs no list position.
__device__ __forceinline__ uint32_t run_record(int px, int pn, unsigned mx, unsigned mn) {
    return (uint32_t)px | ((uint32_t)pn << 8) | (mx << 16) | (mn << 24);
}

// whether the stop test reads the step's SD: from the second sift on, where a
// sum of squares over another can fall below tau at all
__device__ __forceinline__ bool reads_sd(const Ctx& C, const TaskSm& S) {
    return S.mode == TM_SIFT && S.sift >= 1 && C.tau > 0.0;
}

// Pointers and flags of one sweep step.
template <typename T>
struct StepIo {
    const T* hsrc;   // h read by the step (sifting, TRANS from a sift)
    const T* rcur;   // current residual
    T* rnxt;         // residual written by LAST / TRANS / INIT
    T* hdst;         // h written by SIFT
    T* imf_m;        // the IMF slot (written by LAST, and by TRANS when the IMF is elsewhere)
    bool trans_imf;  // TRANS copies the IMF into its slot
};

// new value f and next-knot value g of sample t from h / r (not the envelopes)
template <typename T, int MODE>
__device__ __forceinline__ void plain_value(const Ctx& C, const TaskSm& S, const TaskDesc& d, int t, T h, T r,
                                            T& f, T& g) {
    if (MODE == TM_TRANS) {
        f = r - (S.imf_from_resid ? r : h);
        g = f;
    } else {  // TM_INIT
        f = (T)trial_input<T>(C, d, t);
        g = f;
    }
}

// next-knot value of a sample outside the warp range (t = range start - 1 or
// range end), evaluated by one lane from global memory
template <typename T, bool EXACT, int MODE>
__device__ T outside_g(const Ctx& C, const TaskSm& S, const TaskDesc& d, const StepIo<T>& io, const Rec<T>& R0,
                       const Rec<T>& R1, int t, int cl0, int cl1) {
    constexpr bool SIFTING = (MODE == TM_SIFT || MODE == TM_LAST);
    const T h = (SIFTING || (MODE == TM_TRANS && !S.imf_from_resid)) ? __ldcg(io.hsrc + t) : (T)0;
    const T r = (MODE == TM_LAST || MODE == TM_TRANS) ? __ldcg(io.rcur + t) : (T)0;
    if (SIFTING) {
        Iv<T> v0, v1;
        v0.k = v1.k = -1;
        const T eu = env_at<T, EXACT>(S, v0, R0, 0, cl0, t);
        const T el = env_at<T, EXACT>(S, v1, R1, 1, cl1, t);
        const T fn = h - (T)0.5 * (eu + el);
        return (MODE == TM_LAST) ? r - fn : fn;
    }
    T f, g;
    plain_value<T, MODE>(C, S, d, t, h, r, f, g);
    return g;
}

// The sweep.  The CTA's segment [s0, s1) is cut into warp tiles of WT = 32*RUN
// samples and warp w owns a contiguous range of them; lane u of a tile owns
// the run of RUN samples at u*RUN.  Each warp works through its range without
// block-wide barriers and without shared memory, and keeps its own knot lists
// (one knot segment per warp, so no cross-warp prefix is needed).  Per tile:
//   - the lane's run of each stream it reads and its run record from the
//     previous step were loaded into registers during the previous tile (one
//     256-bit load per stream);
//   - the run record gives each lane the interval of its first sample and the
//     masks of the intervals that end inside the run, so the interval of every
//     sample is a running count; each sample gathers its interval's four
//     coefficients from L1 with one vector load per envelope.  All loads of a
//     run are independent of one another and there is no branch, so they and
//     the evaluations overlap; the sample's offset in its interval is 1 right
//     after a knot and grows by 1, both exact;
//   - new values and SD partials; strict extrema of the new values with lane
//     neighbours by shuffle; the tile's last sample is decided with the next
//     tile (its right neighbour), so only the two samples just outside the
//     warp's range are ever evaluated twice;
//   - a warp-shuffle scan places the knots in the warp's lists, and the
//     samples, knots and this step's run records are written.
// Every step reads one set of buffers and writes another (ping-pong), so the
// warps of a step never see each other's writes.
//
// The sweep is bound by instruction issue and by the latency of its dependent
// chains, not by traffic, hence registers instead of staging, gathers instead
// of branches and 4-byte run records (they were 16 bytes, a third of the
// step's traffic).  k_emd with samples staged in shared memory, records of 32
// or 48 bytes loaded in a divergent branch per sample and knots compacted in
// shared memory, against this form (B200): 48 000 samples x 100 trials
// float32 5.77 -> 3.95 ms, 48 000 x 64 float64 1.71 -> 1.19 ms, 2^22 x 64
// float64 505 -> 348 ms, one 8192-sample float64 EMD 0.331 -> 0.262 ms.
template <typename T, bool EXACT, int MODE, int NW>
__device__ void sweep(const Ctx& C, const Slot& sl, TaskSm& S) {
    using G = Geo<T>;
    constexpr int RUN = G::RUN, WT = G::WT;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr bool SIFTING = (MODE == TM_SIFT || MODE == TM_LAST);
    constexpr bool USES_R = (MODE == TM_LAST || MODE == TM_TRANS);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n = S.n, s0 = S.s0, s1 = S.s1, rank = S.rank;
    const bool needs_h = SIFTING || (MODE == TM_TRANS && !S.imf_from_resid);
    const int q = S.step & 1;
    const TaskDesc d = C.td[S.task];
    StepIo<T> io;
    {
        T* const r0 = static_cast<T*>(C.resid) + d.s_off;
        T* const r1 = static_cast<T*>(sl.r1);
        T* const w1 = static_cast<T*>(sl.w1);
        io.imf_m = static_cast<T*>(C.imfs) + d.imf_off + (int64_t)min(S.imf, C.max_imf - 1) * row_stride<T>(n, C.imf_pad);
        io.rcur = S.rcur ? r1 : r0;
        io.rnxt = S.rcur ? r0 : r1;
        // h buffers W0 = the IMF slot (where the caller's rows are not 32-byte aligned, a second
        // slot scratch), W1 = slot scratch: sift k writes W[(max_sifts-1-k) & 1], so the last
        // sift writes the IMF slot; sift k > 0 reads what sift k-1 wrote
        const int wd = (C.max_sifts - 1 - S.sift) & 1;
        T* const w0 = sl.w0 ? static_cast<T*>(sl.w0) : io.imf_m;
        io.hdst = wd ? w1 : w0;
        io.hsrc = io.rcur;
        if (SIFTING && !S.src_resid) io.hsrc = wd ? w0 : w1;
        if (MODE == TM_TRANS && !S.imf_from_resid) io.hsrc = io.hdst;  // the sift that stopped wrote it
        io.trans_imf = (MODE == TM_TRANS) && (S.imf_from_resid || wd == 1 || sl.w0);
    }
    // every stream's runs start on 32 bytes (the caller's IMF rows apart)
    const bool vec = aligned32(io.hsrc) && aligned32(io.rcur) && aligned32(MODE == TM_SIFT ? io.hdst : io.rnxt);
    const bool vec_i = vec && aligned32(io.imf_m);
    const uint32_t* ri_cur = sl.ri + (int64_t)S.kpar * C.slot_runs;
    uint32_t* ri_nxt = sl.ri + (int64_t)(S.kpar ^ 1) * C.slot_runs;
    const int np = S.kpar ^ 1;
    const int seg = rank * NW + wid;
    const int64_t pmx = knot_index(C, np, 0, seg, 0);
    const int pmd = (int)(knot_index(C, np, 1, seg, 0) - pmx);  // the minima's list from the maxima's
    const Rec<T> R0(sl.M, 0, C.kcap), R1(sl.M, 1, C.kcap);  // (R1's arrays follow R0's, kcap records on)
    // the warp's range [r0, r1): an equal share of the segment in whole runs
    // (shares in whole tiles left the last tiles' warps up to a tile behind),
    // cut into tiles of WT samples from r0 (the last one partial)
    const int nrun = (s1 - s0 + RUN - 1) / RUN;
    const int r0 = min(s1, s0 + (int)((int64_t)wid * nrun / NW) * RUN);
    const int r1 = min(s1, s0 + (int)((int64_t)(wid + 1) * nrun / NW) * RUN);
    const int tb = (r1 - r0 + WT - 1) / WT;
    // interval of the current tile's first sample, before clipping: real knots
    // before it (of the lists this step reads) + mir - 1
    int kb0 = S.pref[S.kpar][0][seg] + S.mir[0] - 1, kb1 = S.pref[S.kpar][1][seg] + S.mir[1] - 1;
    // no interval of the range is clipped at the signal's ends
    const bool inner = kb0 >= 0 && kb1 >= 0 && S.pref[S.kpar][0][seg + 1] + S.mir[0] + 1 <= S.p2[0] &&
                       S.pref[S.kpar][1][seg + 1] + S.mir[1] + 1 <= S.p2[1];
    double num = 0.0, den = 0.0;
    const bool need_sd = reads_sd(C, S);
#ifdef EEMD_TRACE
    unsigned long long scyc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    long long smark = clock64();
#define SUB(k)                                          \
    do {                                                \
        const long long now_ = clock64();               \
        scyc[k] += (unsigned long long)(now_ - smark);  \
        smark = now_;                                   \
    } while (0)
#else
#define SUB(k) \
    do {       \
    } while (0)
#endif

    // the next tile's runs and run records, in flight while a tile is
    // processed.  At 128 registers they are asked for once the values are done
    // and take the registers those leave (at the tile's start they spilled:
    // k_emd many 32-trial signals 51.8 ms against 47.4, 48 000 x 100 float32
    // 3.57 against 3.40); at 168 the earlier load covers more of the DRAM
    // latency of long signals (2^22 x 64 float64 327 ms against 335)
    constexpr bool FETCH_EARLY = !SIFTING || (sizeof(T) == 8 && NW == 4);
    T hn[RUN], rn[RUN];
    uint32_t rin = 0;
    auto fetch = [&](int j) {
        const int t = r0 + j * WT + lane * RUN;
        const int nv = max(0, min(RUN, r1 - t));
        if (needs_h) load_run<T, RUN>(io.hsrc + t, hn, nv, vec);
        if (USES_R) load_run<T, RUN>(io.rcur + t, rn, nv, vec);
        if (SIFTING) rin = nv > 0 ? ri_cur[t / RUN] : 0u;
    };

    int wcx = 0, wcy = 0;      // knots of each kind written to the warp's lists so far
    T gm1, gm2;                // next-knot values at t0-1 and t0-2 of the current tile
    uint32_t prec = 0;         // this lane's run record of the previous tile, not written yet
    gm1 = gm2 = (T)__int_as_float(0x7fc00000);  // NaN: the signal's first sample is no extremum
    if (tb > 0) {
        fetch(0);
        if (r0 > 0) {
            // the sample before the range: its value is the left neighbour of the range's first sample
            int c0 = 0, c1 = 0;
            if (SIFTING && lane == 0) {
                const uint32_t pm = __ldcg(&ri_cur[r0 / RUN - 1]);
                c0 = kb0 + 1 - S.mir[0] - (int)((pm >> (16 + RUN - 1)) & 1u);
                c1 = kb1 + 1 - S.mir[1] - (int)((pm >> (24 + RUN - 1)) & 1u);
            }
            if (lane == 0) gm1 = outside_g<T, EXACT, MODE>(C, S, d, io, R0, R1, r0 - 1, c0, c1);
            gm1 = __shfl_sync(FULL, gm1, 0);
        }
    }

    for (int j = 0; j < tb; ++j) {
        const int t0 = r0 + j * WT, tl = min(WT, r1 - t0);
        const int tj = t0 + lane * RUN;                  // first sample of this lane's run
        const int nv = max(0, min(RUN, tl - lane * RUN));  // samples of the run
        const bool whole = tl == WT;
        const int last_lane = whole ? 31 : (tl - 1) / RUN;
        T hv[RUN], rv[RUN], fv[RUN], gv[RUN];
#pragma unroll
        for (int i = 0; i < RUN; ++i) {
            hv[i] = needs_h ? hn[i] : (T)0;
            rv[i] = USES_R ? rn[i] : (T)0;
        }
        const uint32_t ri = rin;
        if (FETCH_EARLY && j + 1 < tb) fetch(j + 1);
        SUB(0);

        // ---------------- new values ----------------
        if (SIFTING) {
            unsigned kmx = (ri >> 16) & 0xffu, kmn = ri >> 24;
            int k0 = kb0 + (int)(ri & 0xffu), k1 = kb1 + (int)((ri >> 8) & 0xffu);  // the run's first intervals
            T m[RUN];  // mean envelope
            if constexpr (EXACT) {
                Iv<T> v0, v1;
                v0.k = v1.k = -1;
                int cl0 = k0 + 1 - S.mir[0], cl1 = k1 + 1 - S.mir[1];
#pragma unroll
                for (int i = 0; i < RUN; ++i) {
                    m[i] = (T)0;
                    if (i < nv) {
                        const T eu = env_at<T, EXACT>(S, v0, R0, 0, cl0, tj + i);
                        const T el = env_at<T, EXACT>(S, v1, R1, 1, cl1, tj + i);
                        m[i] = (T)0.5 * (eu + el);
                    }
                    cl0 += (kmx >> i) & 1u;
                    cl1 += (kmn >> i) & 1u;
                }
            } else {
                unsigned m0 = kmx, m1 = kmn;  // samples after which the interval changes
                if (!inner) {
                    const int hi0 = max(0, S.p2[0] - 2), hi1 = max(0, S.p2[1] - 2);  // last intervals
                    // clipped at the ends: the first knot (no mirror) starts no new interval, nor does the last
                    if (k0 < 0) m0 &= m0 - 1u;
                    if (k1 < 0) m1 &= m1 - 1u;
                    k0 = min(max(k0, 0), hi0);
                    k1 = min(max(k1, 0), hi1);
                    if (m0 && k0 + (int)__popc(m0) > hi0) m0 ^= 0x80000000u >> __clz(m0);
                    if (m1 && k1 + (int)__popc(m1) > hi1) m1 ^= 0x80000000u >> __clz(m1);
                }
                EEMD_CHECK_IV(k0, max(0, S.p2[0] - 2) - (int)__popc(m0));
                EEMD_CHECK_IV(k1, max(0, S.p2[1] - 2) - (int)__popc(m1));
                k1 += C.kcap;  // from here on an index into R0's arrays
                // offsets in the intervals; float32 counts them in integers (exact beyond 2^24 too)
                using Off = typename std::conditional<sizeof(T) == 4, int, T>::type;
                Off d0 = tj - R0.t[k0], d1 = tj - R0.t[k1];
#pragma unroll
                for (int i = 0; i < RUN; ++i) {
                    if (i > 0) {
                        const bool b0 = (m0 >> (i - 1)) & 1u, b1 = (m1 >> (i - 1)) & 1u;
                        k0 += b0;
                        k1 += b1;
                        d0 = b0 ? 1 : d0 + 1;
                        d1 = b1 ? 1 : d1 + 1;
                    }
                    const T e0 = (T)d0, e1 = (T)d1;
                    T a0, a1, a2, a3, b0, b1, b2, b3;
                    load_coef<T>(R0.c, k0, a0, a1, a2, a3);
                    load_coef<T>(R0.c, k1, b0, b1, b2, b3);
                    const T eu = fmat(e0, fmat(e0, fmat(e0, a3, a2), a1), a0);
                    const T el = fmat(e1, fmat(e1, fmat(e1, b3, b2), b1), b0);
                    m[i] = (T)0.5 * (eu + el);
                }
                if (!whole) {
#pragma unroll
                    for (int i = 0; i < RUN; ++i)
                        if (i >= nv) m[i] = (T)0;  // (hv is 0 there too: no SD terms)
                }
            }
            T tnum = (T)0, tden = (T)0;  // fast mode: this tile's SD partial sums
#pragma unroll
            for (int i = 0; i < RUN; ++i) {
                const T h = hv[i];
                fv[i] = h - m[i];
                gv[i] = (MODE == TM_LAST) ? rv[i] - fv[i] : fv[i];
                if (MODE == TM_SIFT) {
                    const T dd = (C.rules == EEMD_RULES_NUMBA) ? m[i] : h - fv[i];
                    if (EXACT) {
                        num = num + (double)dd * (double)dd;
                        den = den + (double)h * (double)h;
                    } else {
                        tnum = fmat(dd, dd, tnum);
                        tden = fmat(h, h, tden);
                    }
                }
            }
            if (MODE == TM_SIFT && !EXACT) {
                num += (double)tnum;
                den += (double)tden;
            }
            // the tile's knots: the last run's position and its own
            const int kt = (int)((ri & 0xffu) + __popc(kmx)) | ((int)(((ri >> 8) & 0xffu) + __popc(kmn)) << 16);
            const int kl = __shfl_sync(FULL, kt, last_lane);
            kb0 += kl & 0xffff;
            kb1 += kl >> 16;
            if (!FETCH_EARLY && j + 1 < tb) fetch(j + 1);
        } else {
            if (MODE == TM_INIT && C.noise_mode == EEMD_NOISE_PHILOX) {
                // runs start at even samples: one Box-Muller transform per two of them
                const double sigma = C.sigma[d.signal];
#pragma unroll
                for (int i = 0; i < RUN; i += 2) {
                    fv[i] = fv[i + 1] = (T)0;
                    if (i < nv) {
                        const double2 z = philox_normals<T>(C.seed, d.signal, d.trial, tj + i);
                        fv[i] = (T)(ldv<T>(C.x, d.x_off + tj + i) + sigma * z.x);
                        if (i + 1 < nv) fv[i + 1] = (T)(ldv<T>(C.x, d.x_off + tj + i + 1) + sigma * z.y);
                    }
                    gv[i] = fv[i];
                    gv[i + 1] = fv[i + 1];
                }
            } else {
#pragma unroll
                for (int i = 0; i < RUN; ++i) {
                    fv[i] = gv[i] = (T)0;
                    if (i < nv) plain_value<T, MODE>(C, S, d, tj + i, hv[i], rv[i], fv[i], gv[i]);
                }
            }
        }
        SUB(1);

        // ---------------- strict extrema of the new values ----------------
        // lanes decide their own samples except the tile's last one (its right
        // neighbour is the next tile's first sample): the previous tile's last
        // sample is decided now
        const T up = __shfl_up_sync(FULL, gv[RUN - 1], 1);
        const T dn = __shfl_down_sync(FULL, gv[0], 1);
        const T gfirst = __shfl_sync(FULL, gv[0], 0);
        unsigned rise = 0u, fall = 0u;  // bit i: sample i above / below the one before it
#pragma unroll
        for (int i = 0; i <= RUN; ++i) {
            const T a = (i == 0) ? (lane == 0 ? gm1 : up) : gv[(i + RUN - 1) % RUN];
            const T v = (i == RUN) ? dn : gv[i % RUN];
            if (v > a) rise |= 1u << i;
            if (v < a) fall |= 1u << i;
        }
        // samples of the run that may be knots: inside the run, not the tile's last sample
        unsigned valid = (1u << nv) - 1u;
        if (lane == last_lane) valid >>= 1;
        const unsigned nmx = rise & (fall >> 1) & valid, nmn = fall & (rise >> 1) & valid;
        // the previous tile's last sample (the same in every lane)
        const bool carry = j > 0;
        const unsigned dmx = (carry && gm1 > gm2 && gm1 > gfirst) ? 1u : 0u;
        const unsigned dmn = (carry && gm1 < gm2 && gm1 < gfirst) ? 1u : 0u;
        const int cnt = (int)__popc(nmx) | ((int)__popc(nmn) << 16);
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += x;
        }
        const int tot = __shfl_sync(FULL, inc, 31);
        const int exc = inc - cnt;
        SUB(2);

        // ---------------- writes ----------------
        const int nx = (tot & 0xffff) + (int)dmx, nn = (tot >> 16) + (int)dmn;
        if (carry) {
            // the previous tile's run records: its last sample's bit is known now
            if (lane == 31) prec |= (dmx << (16 + RUN - 1)) | (dmn << (24 + RUN - 1));
            ri_nxt[t0 / RUN - 32 + lane] = prec;
        }
        const int px = exc & 0xffff, pn = exc >> 16;  // positions within the tile
        prec = run_record(px, pn, nmx, nmn);
        if (wcx + nx > C.segcap || wcy + nn > C.segcap) {
            if (lane == 0) task_error(C, S, EEMD_E_KNOT_OVERFLOW);
        } else {
            if (lane == 31) {
                if (dmx) put_knot<T>(sl, pmx + wcx, t0 - 1, gm1);
                if (dmn) put_knot<T>(sl, pmx + pmd + wcy, t0 - 1, gm1);
            }
            if (tot) {
                // straight to the lists: a run's knots of a kind are neighbours there, and so are the lanes'
                int ox = wcx + (int)dmx + px, on = pmd + wcy + (int)dmn + pn;
                unsigned any = nmx | nmn;
                // A tile with at most two knots in every run stores them one at a time (the
                // warp's longest run bounds the steps) instead of in RUN predicated ones:
                // float32 3.323 -> 3.283 ms (48000 samples x 100 trials x 80 sifts), 5.84 ->
                // 5.73 (16 x 65536 x 8); bounds of 1 and 3 3.299, 3.287.  float64's runs of 4
                // lose by it (319 -> 344 ms, 2^22 x 64: registers) and keep the plain loop.
                if (sizeof(T) == 4 && __reduce_max_sync(FULL, (unsigned)__popc(any)) <= 2u) {
                    while (any) {
                        const int i = __ffs(any) - 1;
                        any &= any - 1u;
                        T v = gv[0];
#pragma unroll
                        for (int q = 1; q < RUN; ++q) v = i == q ? gv[q] : v;
                        const bool ax = (nmx >> i) & 1u;
                        put_knot<T>(sl, pmx + (ax ? ox : on), tj + i, v);
                        ox += ax;
                        on += !ax;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < RUN; ++i) {
                        const bool ax = (nmx >> i) & 1u, an = (nmn >> i) & 1u;
                        const int o = ax ? ox : on;
                        if (ax || an) put_knot<T>(sl, pmx + o, tj + i, gv[i]);
                        ox += ax;
                        on += an;
                    }
                }
            }
        }
        if (MODE == TM_SIFT) {
            store_run<T, RUN>(io.hdst + tj, fv, nv, vec);
        } else if (MODE == TM_LAST) {
            store_run<T, RUN>(io.imf_m + tj, fv, nv, vec_i);
            store_run<T, RUN>(io.rnxt + tj, gv, nv, vec);
        } else if (MODE == TM_TRANS) {
            store_run<T, RUN>(io.rnxt + tj, fv, nv, vec);
            if (io.trans_imf) {
                if (S.imf_from_resid) store_run<T, RUN>(io.imf_m + tj, rv, nv, vec_i);
                else store_run<T, RUN>(io.imf_m + tj, hv, nv, vec_i);
            }
        } else {
            store_run<T, RUN>(io.rnxt + tj, fv, nv, vec);
        }
        // carry to the next tile: the last sample's value and its left neighbour's
        if (whole) {
            gm2 = __shfl_sync(FULL, gv[RUN - 2], 31);
            gm1 = __shfl_sync(FULL, gv[RUN - 1], 31);
        } else {
            gm2 = (tl >= 2) ? tile_at<T, RUN>(gv, tl - 2) : gm1;
            gm1 = tile_at<T, RUN>(gv, tl - 1);
        }
        wcx += nx;
        wcy += nn;
        SUB(3);
    }
    if (tb > 0) {
        // the range's last sample r1-1: its right neighbour lies outside the range
        const int tlast = r0 + (tb - 1) * WT, last = r1 - 1 - tlast;  // last tile's start, r1-1 within it
        unsigned dmx = 0u, dmn = 0u;
        if (lane == 0 && r1 < n) {
            const T gr = outside_g<T, EXACT, MODE>(C, S, d, io, R0, R1, r1, S.pref[S.kpar][0][seg + 1],
                                                  S.pref[S.kpar][1][seg + 1]);
            dmx = (gm1 > gm2 && gm1 > gr) ? 1u : 0u;
            dmn = (gm1 < gm2 && gm1 < gr) ? 1u : 0u;
            if ((dmx && wcx >= C.segcap) || (dmn && wcy >= C.segcap)) {
                task_error(C, S, EEMD_E_KNOT_OVERFLOW);
            } else {
                if (dmx) put_knot<T>(sl, pmx + wcx, r1 - 1, gm1);
                if (dmn) put_knot<T>(sl, pmx + pmd + wcy, r1 - 1, gm1);
            }
        }
        dmx = __shfl_sync(FULL, dmx, 0);
        dmn = __shfl_sync(FULL, dmn, 0);
        if (lane == last / RUN) prec |= (dmx << (16 + last % RUN)) | (dmn << (24 + last % RUN));
        if (lane <= last / RUN) ri_nxt[tlast / RUN + lane] = prec;
        wcx += (int)dmx;
        wcy += (int)dmn;
    }
    if (MODE == TM_SIFT && need_sd) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            num += __shfl_down_sync(FULL, num, o);
            den += __shfl_down_sync(FULL, den, o);
        }
    }
    if (lane == 0) {
        S.x[q].cnt[0][wid] = wcx;
        S.x[q].cnt[1][wid] = wcy;
        if (MODE == TM_SIFT && need_sd) S.x[q].sd[wid] = make_double2(num, den);
    }
#ifdef EEMD_TRACE
    if (lane == 0) {
        for (int k = 0; k < 4; ++k) atomicAdd(&C.hdr->sweep_cycles[k], scyc[k]);
    }
#endif
#undef SUB
}

// ---------------------------------------------------------------------------
// decisions (emd_ref.py:120-153; emd_gpu.py:152-274)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void log_sift(const Ctx& C, const TaskSm& S) {
    if (C.knot_log && S.rank == 0) {
        int32_t* p = C.knot_log + (((int64_t)S.task * C.max_imf + S.imf) * C.max_sifts + S.sift) * 2;
        p[0] = S.P[0];
        p[1] = S.P[1];
    }
}

__device__ __forceinline__ void close_imf(const Ctx& C, TaskSm& S) {
    if (C.mode_sifts && S.rank == 0) C.mode_sifts[(int64_t)S.task * C.max_imf + S.imf] = S.mode_sifts_cur;
    S.nmode = S.imf + 1;
    S.imf += 1;
    S.mode_sifts_cur = 0;
}

// adopt the knots the last sweep produced (their segment prefixes are in pref[kpar ^ 1])
__device__ __forceinline__ void adopt(TaskSm& S, int cmax, int cmin) {
    S.kpar ^= 1;
    S.P[0] = cmax;
    S.P[1] = cmin;
}

__device__ __forceinline__ void imf_level(const Ctx& C, TaskSm& S, int cmax, int cmin) {
    bool stop = (cmax + cmin < C.min_extrema);
    if (C.rules == EEMD_RULES_NUMBA) stop = stop || cmax < 2 || cmin < 2;
    if (stop) { S.phase = PH_DONE; return; }
    if (S.imf >= C.max_imf) { S.phase = PH_DONE; S.flags |= 1; return; }
    S.mode_sifts_cur = 0;
    if (C.rules == EEMD_RULES_REF && (cmax < 1 || cmin < 1)) {
        // emd_ref.py:132-133: the sift loop breaks before its first sift; the IMF is the residual
        S.phase = PH_TRANS;
        S.imf_from_resid = 1;
        return;
    }
    S.phase = PH_SIFT;
    S.sift = 0;
    S.src_resid = 1;
    S.imf_from_resid = 0;
    adopt(S, cmax, cmin);
}

// the next step's mode and envelopes (mirror ends from three knots on)
__device__ __forceinline__ void set_step(const Ctx& C, TaskSm& S) {
    if (S.phase == PH_TRANS) S.mode = TM_TRANS;
    if (S.phase != PH_SIFT) return;
    S.mode = (S.sift + 1 >= C.max_sifts) ? TM_LAST : TM_SIFT;
    for (int env = 0; env < 2; ++env) {
        S.mir[env] = (C.end_mode == EEMD_END_MIRROR && S.P[env] >= 3) ? 1 : 0;
        S.p2[env] = S.P[env] + 2 * S.mir[env];
        if (S.p2[env] > C.kcap) {
            // computed from the same counts in every CTA of the cluster: all leave the task together
            raise_error(C.hdr, EEMD_E_KNOT_OVERFLOW, S.task);
            S.phase = PH_DONE;
            S.flags |= 2;
        }
    }
}

// Warp 0 gathers the knot counts of every (CTA, warp) segment through
// distributed shared memory and writes their prefixes for the new lists;
// thread 0 then takes the step decision, identical in every CTA.  Every remote
// read is one lane's: a step's critical path holds one round trip (the SD sums
// and error flags read one CTA after another cost a round trip each).
template <int NW>
__device__ void decide(const Ctx& C, TaskSm& S, cg::cluster_group& cl) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const int q = S.step & 1;
        const int nseg = S.csize * NW;
        const bool need_sd = reads_sd(C, S);
        const Xchg* X = &S.x[q];
        // segments SPL*lane .. SPL*lane + SPL-1 per lane (SPL = 3 covers the
        // 16 x 5 = 80 segments of the largest cluster of 5-warp CTAs)
        constexpr int SPL = (MAXSEG + 31) / 32;
        static_assert(SPL * 32 >= MAXSEG, "segments per lane");
        int c[2][SPL];  // [env][segment SPL*lane + k]
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            const int sg = SPL * lane + k;
            c[0][k] = c[1][k] = 0;
            if (sg < nseg) {
                const Xchg* xr = cl.map_shared_rank(X, sg / NW);
                c[0][k] = xr->cnt[0][sg % NW];
                c[1][k] = xr->cnt[1][sg % NW];
            }
        }
        // one CTA's error flag and SD sums per lane, the warps' sums as a shuffle tree adds them
        int err = 0;
        double2 v = make_double2(0.0, 0.0);
        if (lane < S.csize) {
            const Xchg* xr = cl.map_shared_rank(X, lane);
            err = xr->err;
            if (need_sd) {
                const double2 a = xr->sd[0], b = xr->sd[1], c2 = xr->sd[2], d = xr->sd[3];
                const double2 e = NW == 5 ? xr->sd[NW - 1] : make_double2(0.0, 0.0);
                v.x = ((a.x + e.x) + c2.x) + (b.x + d.x);
                v.y = ((a.y + e.y) + c2.y) + (b.y + d.y);
            }
        }
        err = __any_sync(0xffffffffu, err);
        int tot[2];
#pragma unroll
        for (int env = 0; env < 2; ++env) {
            int sum = 0;
#pragma unroll
            for (int k = 0; k < SPL; ++k) sum += c[env][k];
            int inc = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += x;
            }
            tot[env] = __shfl_sync(0xffffffffu, inc, 31);
            int* pr = S.pref[S.kpar ^ 1][env];
            int e = inc - sum;
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                if (SPL * lane + k < nseg) pr[SPL * lane + k] = e;
                e += c[env][k];
            }
            if (lane == 0) pr[nseg] = tot[env];
        }
        double num = 0.0, den = 0.0;
        if (need_sd) {
            for (int r = 0; r < S.csize; ++r) {  // in CTA order
                num += __shfl_sync(0xffffffffu, v.x, r);
                den += __shfl_sync(0xffffffffu, v.y, r);
            }
        }
        if (lane == 0) {
            const int cmax = tot[0], cmin = tot[1];
            const int mode = S.mode;
            if (err) {
                // an error of this task (recorded in the header): stop it here
                S.phase = PH_DONE;
                S.flags |= 2;
            } else if (mode == TM_SIFT) {
                log_sift(C, S);
                S.mode_sifts_cur += 1;
                S.nsift_total += 1;
                const double sdv = den > 0.0 ? num / den : 0.0;
                bool stop = need_sd && (sdv < C.tau);
                if (!stop) stop = (C.rules == EEMD_RULES_NUMBA) ? (cmax < 2 || cmin < 2) : (cmax < 1 || cmin < 1);
                if (stop) {
                    S.phase = PH_TRANS;
                    S.imf_from_resid = 0;
                } else {
                    S.sift += 1;
                    S.src_resid = 0;
                    adopt(S, cmax, cmin);
                }
            } else if (mode == TM_LAST) {
                log_sift(C, S);
                S.mode_sifts_cur += 1;
                S.nsift_total += 1;
                S.rcur ^= 1;
                close_imf(C, S);
                imf_level(C, S, cmax, cmin);
            } else if (mode == TM_TRANS) {
                S.rcur ^= 1;
                close_imf(C, S);
                imf_level(C, S, cmax, cmin);
            } else {
                S.rcur ^= 1;
                S.imf = 0;
                S.nmode = 0;
                imf_level(C, S, cmax, cmin);
            }
            S.step += 1;
            // (its last readers, of the step before, have passed a cluster barrier since)
            S.x[S.step & 1].err = 0;
            set_step(C, S);
            // every IMF ends after at most max_sifts sifts plus one closing step
            if (S.phase != PH_DONE && S.step > 2 + C.max_imf * (C.max_sifts + 1)) {
                raise_error(C.hdr, EEMD_E_TIMEOUT, S.task);
                S.phase = PH_DONE;
            }
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// k_emd: the persistent cluster kernel
// ---------------------------------------------------------------------------
template <typename T, bool EXACT, int NW>
__global__ void __launch_bounds__(32 * NW, ctas_per_sm(NW, (int)sizeof(T))) k_emd(const __grid_constant__ Ctx C) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TaskSm S;
    __shared__ int s_claim;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int csize = (int)cl.num_blocks();
    const int slot = blockIdx.x / csize;
    const int tid = threadIdx.x;
    Slot sl;
    sl.kt = C.kt + (int64_t)slot * C.slot_knots * (sizeof(T) == 4 ? 2 : 1);
    sl.ky = static_cast<T*>(C.ky) + (int64_t)slot * C.slot_knots;
    sl.M = static_cast<T*>(C.M) + (int64_t)slot * C.slot_M;
    sl.w1 = static_cast<T*>(C.w1) + (int64_t)slot * C.slot_n;
    sl.w0 = C.w0 ? static_cast<T*>(C.w0) + (int64_t)slot * C.slot_n : nullptr;
    sl.r1 = static_cast<T*>(C.r1) + (int64_t)slot * C.slot_n;
    sl.ri = C.ri + (int64_t)slot * 2 * C.slot_runs;

#ifdef EEMD_TRACE
    unsigned long long cyc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    long long tmark = clock64();
#define EEMD_PHASE(k)                                   \
    do {                                                \
        const long long now_ = clock64();               \
        cyc[k] += (unsigned long long)(now_ - tmark);   \
        tmark = now_;                                   \
    } while (0)
#else
#define EEMD_PHASE(k) \
    do {              \
    } while (0)
#endif
    for (;;) {
        if (rank == 0 && tid == 0) s_claim = atomicAdd(&C.hdr->next_task, 1);
        cl.sync();
        const int q = *cl.map_shared_rank(&s_claim, 0);
        cl.sync();
        EEMD_PHASE(6);
        if (q >= C.n_tasks) break;
        for (int r = tid; r <= MAXSEG; r += 32 * NW)
            S.pref[0][0][r] = S.pref[0][1][r] = S.pref[1][0][r] = S.pref[1][1][r] = 0;
        if (tid == 0) {
            const int task = C.order[q];
            const TaskDesc d = C.td[task];
            S.task = task;
            S.n = d.n;
            S.rank = rank;
            S.csize = csize;
            S.s0 = min(d.n, rank * d.seg);
            S.s1 = min(d.n, S.s0 + d.seg);
            S.phase = PH_INIT;
            S.imf = S.sift = S.kpar = S.src_resid = S.imf_from_resid = 0;
            S.nsift_total = S.nmode = S.mode_sifts_cur = S.flags = S.step = 0;
            S.P[0] = S.P[1] = 0;
            S.mir[0] = S.mir[1] = S.p2[0] = S.p2[1] = 0;
            S.mode = TM_INIT;
            S.x[0].err = S.x[1].err = 0;
            S.rcur = 1;  // the first step writes the residual array
            if (C.watchdog < 0 && rank == 0) {
                // watchdog test mode: a bounded wait on a flag nothing sets
                long long spins = 0;
                while (*((volatile int32_t*)&C.hdr->wd_flag) == 0) {
                    if (++spins > -C.watchdog) {
                        raise_error(C.hdr, EEMD_E_TIMEOUT, task);
                        break;
                    }
                    __nanosleep(32);
                }
            }
        }
        __syncthreads();
        while (S.phase != PH_DONE) {
            if (S.mode == TM_SIFT || S.mode == TM_LAST) {
                EEMD_PHASE(0);
                solve_task<T, EXACT, NW>(C, sl, S, smem_raw);
                EEMD_PHASE(1);
                cl.sync();  // second derivatives of every segment visible
                EEMD_PHASE(2);
            }
            switch (S.mode) {
                case TM_SIFT: sweep<T, EXACT, TM_SIFT, NW>(C, sl, S); break;
                case TM_LAST: sweep<T, EXACT, TM_LAST, NW>(C, sl, S); break;
                case TM_TRANS: sweep<T, EXACT, TM_TRANS, NW>(C, sl, S); break;
                default: sweep<T, EXACT, TM_INIT, NW>(C, sl, S); break;
            }
            EEMD_PHASE(3);
            cl.sync();  // segment results published
            EEMD_PHASE(4);
            decide<NW>(C, S, cl);
            EEMD_PHASE(5);
        }
        if (C.resid_out) {
            // this segment of the final residual
            const TaskDesc d = C.td[S.task];
            T* o = static_cast<T*>(C.resid_out) + d.noise_off;
            const T* r = S.rcur ? static_cast<const T*>(sl.r1) : static_cast<const T*>(C.resid) + d.s_off;
            for (int t = S.s0 + tid; t < S.s1; t += 32 * NW) o[t] = r[t];
        }
        if (rank == 0 && tid == 0) {
            TaskOut o;
            o.nsift = S.nsift_total;
            o.nmode = S.nmode;
            o.flags = S.flags;
            o.pad = 0;
            C.tout[S.task] = o;
            atomicAdd(&C.hdr->n_done, 1);
        }
        __syncthreads();
    }
#ifdef EEMD_TRACE
    if (tid == 0) {
        for (int k = 0; k < 8; ++k) atomicAdd(&C.hdr->phase_cycles[k], cyc[k]);
    }
#endif
#undef EEMD_PHASE
}

// ---------------------------------------------------------------------------
// k_reduce: imf_sum[s][m][t] += trial-ordered sum over the batch (emd_par.py:241-245)
// ---------------------------------------------------------------------------
// One sample per thread.  Every trial's load is independent of the others, so
// eight are in flight before their (ordered) additions; the trials that reached
// the mode are counted once per CTA, and in the common case, all of them, no
// load waits for a test.  48 000 x 100 float32, 8 modes: 105 us with one
// dependent load at a time, 45 us here; 2^22 x 64 float64, 12 modes: 5.35 and
// 3.68 ms (7 TB/s read).
constexpr int RED_UNROLL = 8;
template <typename T>
__global__ void __launch_bounds__(256) k_reduce(const SignalDesc* sdesc, const TaskDesc* td, const TaskOut* tout,
                                                const void* imfs, int trial_count, int max_imf, int imf_pad,
                                                double* imf_sum, int32_t* mode_count) {
    const int s = blockIdx.z, m = blockIdx.y;
    const SignalDesc sd = sdesc[s];
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if ((int64_t)blockIdx.x * blockDim.x >= sd.n) return;
    const TaskOut* to = tout + sd.first_task;
    int cnt = 0;
    for (int e0 = 0; e0 < trial_count; e0 += blockDim.x) {
        const int e = e0 + threadIdx.x;
        cnt += __syncthreads_count(e < trial_count && to[e].nmode > m);
    }
    if (mode_count && blockIdx.x == 0 && threadIdx.x == 0) mode_count[(int64_t)s * max_imf + m] += cnt;
    if (!imf_sum || t >= sd.n || cnt == 0) return;
    const int64_t row = row_stride<T>(sd.n, imf_pad), step = row * max_imf;  // between trials
    const T* p = static_cast<const T*>(imfs) + td[sd.first_task].imf_off + m * row + t;
    double acc = 0.0;
    if (cnt == trial_count) {
        acc = (double)p[0];
        int e = 1;
        for (; e + RED_UNROLL <= trial_count; e += RED_UNROLL) {
            T v[RED_UNROLL];
#pragma unroll
            for (int u = 0; u < RED_UNROLL; ++u) v[u] = p[(e + u) * step];
#pragma unroll
            for (int u = 0; u < RED_UNROLL; ++u) acc += (double)v[u];
        }
        for (; e < trial_count; ++e) acc += (double)p[e * step];
    } else {
        bool any = false;
        for (int e = 0; e < trial_count; ++e) {
            if (to[e].nmode > m) {
                const double v = (double)p[e * step];
                acc = any ? acc + v : v;
                any = true;
            }
        }
    }
    double* o = imf_sum + sd.sum_off + (int64_t)m * sd.n + t;
    *o = *o + acc;
}

__global__ void k_outputs(const TaskOut* tout, int n_tasks, int32_t* nsift, int32_t* nmode, int32_t* flags) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_tasks) return;
    const TaskOut o = tout[i];
    if (nsift) nsift[i] = o.nsift;
    if (nmode) nmode[i] = o.nmode;
    if (flags) flags[i] = o.flags;
}

// ---------------------------------------------------------------------------
// k_finalize: mean + residual (emd_par.py:248-250)
// ---------------------------------------------------------------------------
constexpr int FIN_BATCH = 256;  // signal descriptors per launch, passed by value
struct FinBatch {
    SignalDesc sd[FIN_BATCH];
};

template <typename T>
__global__ void k_finalize(FinBatch fb, int s_base, int max_imf, const void* x, const double* imf_sum,
                           const int32_t* mode_count, double* imf_mean, double* residual,
                           int32_t* n_modes) {
    const int sl = blockIdx.y;
    const int s = s_base + sl;
    const SignalDesc sd = fb.sd[sl];
    const int32_t* cnt = mode_count + (int64_t)s * max_imf;
    int nm = 0;
    while (nm < max_imf && cnt[nm] > 0) ++nm;
    if (n_modes && blockIdx.x == 0 && threadIdx.x == 0) n_modes[s] = nm;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= sd.n) return;
    double acc = 0.0;
    for (int m = 0; m < nm; ++m) {
        const int64_t o = sd.sum_off + (int64_t)m * sd.n + t;
        const double v = imf_sum[o] / (double)cnt[m];
        if (imf_mean) imf_mean[o] = v;
        acc = (m == 0) ? v : acc + v;
    }
    if (residual) residual[sd.r_off + t] = ldv<T>(x, sd.x_off + t) - acc;
}

}  // namespace eemd

// ===========================================================================
// host side
// ===========================================================================
using namespace eemd;

namespace {

constexpr int ASSUMED_SMS = 148;        // B200

struct Layout {
    std::vector<TaskDesc> td;
    std::vector<SignalDesc> sd;
    std::vector<int32_t> order;
    int64_t NS = 0, NIMF = 0, slot_knots = 0, slot_M = 0, slot_n = 0, slot_runs = 0;
    int B = 0, S = 0, csize = 1, slots = 1, segcap = 0, kcap = 0, scr_rows = 0, nw = NW_DEFAULT;
    bool imf_pad = false, has_w0 = false;
    size_t o_hdr, o_td, o_order, o_tout, o_sd, o_sigma, o_resid, o_imfs, o_kt, o_ky, o_M, o_w1, o_w0, o_r1, o_ri,
        o_scr;
    size_t total = 0;
};

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// records, and rows where they are padded, are read and written 32 bytes at a
// time: the arrays lie in the workspace from its first multiple of 32 on
constexpr size_t WS_ALIGN = 32;

// Clusters of c CTAs of the k_emd instance for (dtype, exact) that the
// current device can hold at once (0 if the query fails, e.g. no device).
// the k_emd instance of (storage type, exact, warps per CTA)
const void* emd_fn(int dtype, bool exact, int nw) {
    if (dtype == EEMD_F32) return nw == 5 ? (const void*)k_emd<float, false, 5> : (const void*)k_emd<float, false, 4>;
    if (exact) return (const void*)k_emd<double, true, 4>;
    return nw == 5 ? (const void*)k_emd<double, false, 5> : (const void*)k_emd<double, false, 4>;
}

int active_clusters(int dtype, bool exact, int c, int nw) {
    const void* fn = emd_fn(dtype, exact, nw);
    const size_t smem = smem_bytes(dtype == EEMD_F32 ? 4 : 8, exact, nw);
    int n = 0;
    bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
    if (ok && c > 8) ok = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (ok) {
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3((unsigned)c, 1, 1);
        cfg.blockDim = dim3((unsigned)(32 * nw), 1, 1);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)c;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        ok = cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess;
    }
    if (!ok) {
        (void)cudaGetLastError();  // a failed query leaves no sticky state for the launch checks
        n = 0;
    }
    return n;
}

// The cluster spreads one task over several SMs when there are fewer tasks
// than CTA slots.
int autotune_csize(int64_t n_tasks, int64_t nmin, int dtype, bool exact, int nw) {
    // leave a fifth of the CTA slots free: clusters must fit inside a GPC,
    // and the last clusters to be placed would otherwise wait for a second
    // wave.  Signals of a million samples or more take every slot: each CTA
    // then sweeps long ranges, and measured on 64 trials of 2^22 samples 8
    // CTAs per signal (512 CTAs) run 10 % faster than 7.
    const int64_t slots = (int64_t)ASSUMED_SMS * ctas_per_sm(nw, dtype == EEMD_F64 ? 8 : 4);
    const int64_t budget = nmin >= (1 << 20) ? slots : slots * 4 / 5;
    int c = (int)std::max<int64_t>(1, std::min<int64_t>(8, budget / std::max<int64_t>(n_tasks, 1)));
    // more tasks than slots: pairs of CTAs halve each task's time and with it
    // the last round's idle tail (1024 tasks of 65536 samples: 94.6 ms at 2
    // against 97.0 at 1)
    if (c == 1 && nmin >= (1 << 16)) c = 2;
    // signals of a million samples or more with slots to spare at 8 CTAs per
    // task (64 tasks use 512 of 592): a larger, non-portable cluster when the
    // device holds every task's cluster at once (a task waiting for a second
    // wave would double the launch)
    if (c == 8 && nmin >= (1 << 20)) {
        for (int c2 = (int)std::min<int64_t>(MAXC, slots / std::max<int64_t>(n_tasks, 1)); c2 > 8; --c2) {
            if (active_clusters(dtype, exact, c2, nw) >= n_tasks) {
                c = c2;
                break;
            }
        }
    }
    while (c > 1 && nmin / c < 2048) --c;
    return c;
}

int check_params(const eemd_params* p) {
    if (!p) return EEMD_E_BADARG;
    if (p->dtype != EEMD_F64 && p->dtype != EEMD_F32) return EEMD_E_BADARG;
    if (p->exact && p->dtype != EEMD_F64) return EEMD_E_NOTSUP;
    if (p->max_sifts < 1 || p->max_imf < 1 || p->max_imf > 4096) return EEMD_E_BADARG;
    if (p->end_mode != EEMD_END_NATURAL && p->end_mode != EEMD_END_MIRROR) return EEMD_E_BADARG;
    if (p->rules != EEMD_RULES_REF && p->rules != EEMD_RULES_NUMBA) return EEMD_E_BADARG;
    if (p->noise_mode < EEMD_NOISE_NONE || p->noise_mode > EEMD_NOISE_SCALED) return EEMD_E_BADARG;
    // warp tile: 32 lanes x 8 float32 samples or x 4 float64 samples
    const int wt = (p->dtype == EEMD_F64) ? Geo<double>::WT : Geo<float>::WT;
    if (p->tile != 0 && p->tile != wt) return EEMD_E_BADARG;
    if (p->knots_per_block < 0 || p->knots_per_block > 4096 || p->halo < 0 || p->halo > 256)
        return EEMD_E_BADARG;
    if (p->cluster_size < 0 || p->cluster_size > MAXC) return EEMD_E_BADARG;
    if (p->cta_warps != 0 && p->cta_warps != 4 && p->cta_warps != 5) return EEMD_E_BADARG;
    if (p->exact && p->cta_warps == 5) return EEMD_E_NOTSUP;  // exact mode runs 4-warp CTAs
    return EEMD_OK;
}

// pad: rows of the workspace (residuals, and IMFs kept there) start on 32
// bytes, so that a lane's run is one 256-bit access whatever the signal's
// length, and a caller's IMF rows that do not are sifted in a second slot
// scratch instead.  Without it the rows follow one another unpadded (the
// smallest workspace; runs of misaligned rows are read by element).
int make_layout(const eemd_params* p, const int64_t* lengths, int n_signals, int trial_count,
                int trial_begin, bool imfs_external, Layout& L, bool pad = true) {
    int rc = check_params(p);
    if (rc) return rc;
    if (!lengths || n_signals < 1 || trial_count < 1) return EEMD_E_BADARG;
    const int64_t n_tasks = (int64_t)n_signals * trial_count;
    if (n_tasks > (1 << 24)) return EEMD_E_BADARG;
    int64_t nmax = 0, nmin = INT64_MAX;
    for (int s = 0; s < n_signals; ++s) {
        if (lengths[s] < 3 || lengths[s] > (1LL << 30)) return EEMD_E_BADARG;
        nmax = std::max(nmax, lengths[s]);
        nmin = std::min(nmin, lengths[s]);
    }
    L.nw = p->cta_warps ? p->cta_warps : NW_DEFAULT;
    L.csize = p->cluster_size ? p->cluster_size : autotune_csize(n_tasks, nmin, p->dtype, p->exact != 0, L.nw);
    // decay halo of the seam windows: the truncation error falls like
    // (2 - sqrt 3)^S; 16 rows put it far below float32 rounding
    L.S = p->halo ? p->halo : (p->exact ? 32 : (p->dtype == EEMD_F32 ? 16 : 24));
    L.B = p->knots_per_block ? p->knots_per_block : 16;
    // a solve pass stages its windows' knots plus the halos in the warp's area:
    // exact windows carry both halos; a fast pass needs room for at least one
    // committing lane besides its ceil(S / FAST_B) right-halo lanes
    if (p->exact && 2 * L.S + L.B + 8 > WSCAP) return EEMD_E_BADARG;
    if (!p->exact && (L.S > FAST_SMAX || (L.S + FAST_B - 1) / FAST_B + 1 > std::min(32, (WSCAP_FAST - L.S - 3) / FAST_B)))
        return EEMD_E_BADARG;
    int64_t segmax = 0;
    L.td.resize(n_tasks);
    L.sd.resize(n_signals);
    const int row = (p->dtype == EEMD_F64) ? 4 : 8;  // samples of 32 bytes
    bool ragged = false;                             // the caller's IMF rows leave the 32-byte grid
    L.imf_pad = pad && !imfs_external;
    int64_t xo = 0, so = 0, ro = 0, imo = 0, sumo = 0;
    for (int s = 0; s < n_signals; ++s) {
        const int64_t n = lengths[s], np = pad ? (n + row - 1) / row * row : n;
        ragged = ragged || n % row != 0;
        SignalDesc& sd = L.sd[s];
        sd.x_off = xo;
        sd.sum_off = sumo;
        sd.r_off = xo;
        sd.n = (int32_t)n;
        sd.first_task = s * trial_count;
        sumo += (int64_t)p->max_imf * n;
        int64_t seg = (n + L.csize - 1) / L.csize;
        seg = (seg + 31) / 32 * 32;
        if ((L.csize - 1) * seg + 2 > n) return EEMD_E_BADARG;  // every segment keeps >= 2 samples
        segmax = std::max(segmax, seg);
        for (int e = 0; e < trial_count; ++e) {
            TaskDesc& d = L.td[(int64_t)s * trial_count + e];
            d.x_off = (p->noise_mode == EEMD_NOISE_PREPERTURBED) ? so : xo;
            d.s_off = ro;
            d.imf_off = imo;
            d.noise_off = so;
            d.n = (int32_t)n;
            d.signal = s;
            d.trial = trial_begin + e;
            d.seg = (int32_t)seg;
            so += n;
            ro += np;
            imo += (int64_t)p->max_imf * (L.imf_pad ? np : n);
        }
        xo += n;
    }
    // longest tasks first: the work queue hands them out in this order
    L.order.resize(n_tasks);
    std::iota(L.order.begin(), L.order.end(), 0);
    std::stable_sort(L.order.begin(), L.order.end(), [&](int a, int b) { return L.td[a].n > L.td[b].n; });
    const int run = (p->dtype == EEMD_F64) ? Geo<double>::RUN : Geo<float>::RUN;
    const int wt = 32 * run;
    // knots of one kind in one warp's range: at most half its samples (+ends)
    const int64_t tiles_per_warp = ((segmax + wt - 1) / wt + L.nw - 1) / L.nw;
    L.segcap = (int)(tiles_per_warp * wt / 2 + 2);
#ifdef EEMD_CHECKED
    // test hook of the checked build only: params.reserved > 0 shrinks the knot
    // lists' capacity so that the overflow path can be exercised
    if (p->reserved > 0 && p->reserved < L.segcap) L.segcap = p->reserved;
#endif
    L.kcap = (int)(nmax / 2 + 4);
    L.slot_n = pad ? (nmax + row - 1) / row * row : (nmax + 3) / 4 * 4;
    L.slot_runs = (nmax + run - 1) / run + 1;
    L.slots = (int)std::max<int64_t>(
        1, std::min<int64_t>(n_tasks, (int64_t)ASSUMED_SMS * ctas_per_sm(L.nw, p->dtype == EEMD_F64 ? 8 : 4) /
                                     L.csize));
    L.slot_knots = (int64_t)2 * 2 * L.csize * L.nw * L.segcap;
    // struct Rec: four coefficients and an index per knot of either envelope, every slot's on 32 bytes
    const int bm = (p->dtype == EEMD_F64) ? 8 : 4;
    L.slot_M = ((int64_t)2 * L.kcap * (4 * bm + 4) + 31) / 32 * 32 / bm;
    L.scr_rows = p->exact ? (L.B + L.S) : 0;
    L.NS = ro;
    L.NIMF = imo;
    const size_t bt = (p->dtype == EEMD_F64) ? 8 : 4;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off = align_up(off + bytes, 256);
        return o;
    };
    L.o_hdr = take(sizeof(Header));
    L.o_td = take(sizeof(TaskDesc) * n_tasks);
    L.o_order = take(sizeof(int32_t) * n_tasks);
    L.o_sd = take(sizeof(SignalDesc) * n_signals);
    L.o_tout = take(sizeof(TaskOut) * n_tasks);  // (what lies before it is uploaded in one copy)
    L.o_sigma = take(sizeof(double) * n_signals);
    L.o_resid = take(bt * L.NS);
    L.o_imfs = imfs_external ? 0 : take(bt * L.NIMF);
    L.o_kt = take(sizeof(int32_t) * L.slot_knots * L.slots);
    L.o_ky = take(bt * L.slot_knots * L.slots);
    L.o_M = take(bt * L.slot_M * L.slots);
    L.o_w1 = take(bt * L.slot_n * L.slots);
    L.has_w0 = pad && imfs_external && ragged;
    L.o_w0 = take(L.has_w0 ? bt * L.slot_n * L.slots : 0);
    L.o_r1 = take(bt * L.slot_n * L.slots);
    L.o_scr = take(sizeof(double2) * (size_t)L.scr_rows * L.slots * L.csize * 32 * L.nw);
    L.o_ri = take(sizeof(uint32_t) * 2 * L.slot_runs * L.slots + WS_ALIGN - 1);  // (the last: what the start skips)
    L.total = off;
    return EEMD_OK;
}

// Optional per-launch CUDA-event timing (eemd_run_traced): one event pair
// per kernel launch, summed per kernel kind after the final synchronise.
struct Tracer {
    eemd_kernel_times* out = nullptr;
    std::vector<cudaEvent_t> ev;
    std::vector<int> kind;
    cudaStream_t st = nullptr;
    int64_t counts[EEMD_KERNEL_KINDS] = {0};
    void begin(int k) {
        counts[k] += 1;
        if (!out) return;
        cudaEvent_t a, b;
        cudaEventCreate(&a);
        cudaEventCreate(&b);
        cudaEventRecord(a, st);
        ev.push_back(a);
        ev.push_back(b);
        kind.push_back(k);
    }
    void end() {
        if (!out) return;
        cudaEventRecord(ev.back(), st);
    }
    void finish() {
        if (!out) return;
        for (int k = 0; k < EEMD_KERNEL_KINDS; ++k) {
            out->ms[k] = 0.0;
            out->launches[k] = counts[k];
        }
        for (size_t i = 0; i < kind.size(); ++i) {
            float ms = 0.f;
            if (cudaEventElapsedTime(&ms, ev[2 * i], ev[2 * i + 1]) == cudaSuccess) out->ms[kind[i]] += ms;
        }
        for (auto e : ev) cudaEventDestroy(e);
        ev.clear();
        kind.clear();
    }
};

template <typename T, bool EXACT, int NW>
int launch_emd(const Ctx& C, const Layout& L, cudaStream_t st, Tracer& tr) {
    const size_t smem = smem_bytes((int)sizeof(T), EXACT, NW);
    if (cudaFuncSetAttribute(k_emd<T, EXACT, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return EEMD_E_CUDA;
    if (L.csize > 8 &&
        cudaFuncSetAttribute(k_emd<T, EXACT, NW>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return EEMD_E_CUDA;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(L.slots * L.csize), 1, 1);
    cfg.blockDim = dim3(32 * NW, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)L.csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    tr.begin(EEMD_K_EMD);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_emd<T, EXACT, NW>, C);
    tr.end();
    return e == cudaSuccess ? EEMD_OK : EEMD_E_CUDA;
}

template <typename T>
int run_typed(const eemd_params* p, const Layout& L, Ctx& C, double* imf_sum, int32_t* mode_count,
              int32_t* nsift, int32_t* nmode, int32_t* flags, cudaStream_t st, Tracer& tr) {
    const int64_t n_tasks = (int64_t)L.td.size();
    if (p->noise_mode == EEMD_NOISE_PHILOX) {
        tr.begin(EEMD_K_SIGMA);
        k_sigma<T><<<(int)L.sd.size(), 1024, 0, st>>>(C.sd, C.x, p->eps, const_cast<double*>(C.sigma));
        tr.end();
    }
    int rc;
    if constexpr (sizeof(T) == 8) {
        if (p->exact)
            rc = launch_emd<T, true, 4>(C, L, st, tr);  // exact mode: float64, 4-warp CTAs
        else
            rc = L.nw == 5 ? launch_emd<T, false, 5>(C, L, st, tr) : launch_emd<T, false, 4>(C, L, st, tr);
    } else {
        rc = L.nw == 5 ? launch_emd<T, false, 5>(C, L, st, tr) : launch_emd<T, false, 4>(C, L, st, tr);
    }
    if (rc) return rc;
    if (imf_sum || mode_count) {
        int64_t nmax = 0;
        for (auto& s : L.sd) nmax = std::max<int64_t>(nmax, s.n);
        dim3 g((unsigned)((nmax + 255) / 256), (unsigned)p->max_imf, (unsigned)L.sd.size());
        tr.begin(EEMD_K_REDUCE);
        k_reduce<T><<<g, 256, 0, st>>>(C.sd, C.td, C.tout, C.imfs, C.trial_count, C.max_imf, C.imf_pad, imf_sum,
                                        mode_count);
        tr.end();
    }
    if (nsift || nmode || flags) {
        tr.begin(EEMD_K_OUTPUTS);
        k_outputs<<<(int)((n_tasks + 255) / 256), 256, 0, st>>>(C.tout, (int)n_tasks, nsift, nmode, flags);
        tr.end();
    }
    return cudaGetLastError() == cudaSuccess ? EEMD_OK : EEMD_E_CUDA;
}

}  // namespace

extern "C" {

void eemd_default_params(eemd_params* p) {
    if (!p) return;
    memset(p, 0, sizeof(*p));
    p->dtype = EEMD_F64;
    p->noise_mode = EEMD_NOISE_NONE;
    p->eps = 0.2;
    p->seed = 0;
    p->tau = 0.25;
    p->max_sifts = 50;
    p->max_imf = 16;
    p->min_extrema = 4;
    p->end_mode = EEMD_END_NATURAL;
    p->rules = EEMD_RULES_REF;
    p->exact = 0;
}

int32_t eemd_version(void) { return EEMD_ABI_VERSION; }

const char* eemd_strerror(int32_t status) {
    switch (status) {
        case EEMD_OK: return "ok";
        case EEMD_E_BADARG: return "invalid argument";
        case EEMD_E_NOMEM: return "workspace too small";
        case EEMD_E_KNOT_OVERFLOW: return "knot buffer capacity exceeded";
        case EEMD_E_TIMEOUT: return "device wait gave up (watchdog)";
        case EEMD_E_CUDA: return "CUDA runtime error";
        case EEMD_E_NOTSUP: return "unsupported parameter combination";
        case EEMD_E_STATIC_CAPACITY:
            return "problem needs more scratch than the static scratch of eemd_run_static "
                   "(EEMD_STATIC_SCRATCH_BYTES); use eemd_run with a workspace";
        default: return "unknown status";
    }
}

int32_t eemd_philox_normals(uint64_t seed, int32_t signal, int32_t trial_begin, int32_t trial_count, int64_t n,
                            double* out, void* stream) {
    if (!out || signal < 0 || trial_begin < 0 || trial_count < 1 || n < 1) return EEMD_E_BADARG;
    const int64_t total = (int64_t)trial_count * n;
    const int64_t blocks = (total + 255) / 256;
    k_philox_fill<<<(unsigned)(blocks < 148 * 32 ? blocks : 148 * 32), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        seed, signal, trial_begin, trial_count, n, out);
    return cudaGetLastError() == cudaSuccess ? EEMD_OK : EEMD_E_CUDA;
}

int32_t eemd_workspace_size(const eemd_params* p, const int64_t* lengths, int32_t n_signals,
                            int32_t trial_count, int32_t imfs_external, size_t* ws_bytes) {
    if (!ws_bytes) return EEMD_E_BADARG;
    Layout L;
    int rc = make_layout(p, lengths, n_signals, trial_count, 0, imfs_external != 0, L);
    if (rc) return rc;
    *ws_bytes = L.total;
    return EEMD_OK;
}

int32_t eemd_run(const eemd_params* p, const void* x, const int64_t* lengths, int32_t n_signals,
                 int32_t trial_begin, int32_t trial_count, const void* noise, void* imfs,
                 void* resid_out, double* imf_sum, int32_t* mode_count, int32_t* nsift,
                 int32_t* nmode, int32_t* mode_sifts, int32_t* knot_log, int32_t* flags, void* ws,
                 size_t ws_bytes, void* stream) {
    return eemd_run_traced(p, x, lengths, n_signals, trial_begin, trial_count, noise, imfs, resid_out,
                           imf_sum, mode_count, nsift, nmode, mode_sifts, knot_log, flags, ws, ws_bytes,
                           stream, nullptr);
}

int32_t eemd_run_traced(const eemd_params* p, const void* x, const int64_t* lengths, int32_t n_signals,
                        int32_t trial_begin, int32_t trial_count, const void* noise, void* imfs,
                        void* resid_out, double* imf_sum, int32_t* mode_count, int32_t* nsift,
                        int32_t* nmode, int32_t* mode_sifts, int32_t* knot_log, int32_t* flags,
                        void* ws, size_t ws_bytes, void* stream, eemd_kernel_times* times) {
    Layout L;
    int rc = make_layout(p, lengths, n_signals, trial_count, trial_begin, imfs != nullptr, L);
    if (rc) return rc;
    if (!x || !ws) return EEMD_E_BADARG;
    if ((p->noise_mode == EEMD_NOISE_INJECTED || p->noise_mode == EEMD_NOISE_SCALED) && !noise)
        return EEMD_E_BADARG;
    if (ws_bytes < L.total) {
        // the same run on unpadded rows
        rc = make_layout(p, lengths, n_signals, trial_count, trial_begin, imfs != nullptr, L, false);
        if (rc) return rc;
        if (ws_bytes < L.total) return EEMD_E_NOMEM;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char* base = reinterpret_cast<char*>(align_up(reinterpret_cast<uintptr_t>(ws), WS_ALIGN));
    Ctx C;
    memset(&C, 0, sizeof(C));
    C.hdr = reinterpret_cast<Header*>(base + L.o_hdr);
    C.td = reinterpret_cast<const TaskDesc*>(base + L.o_td);
    C.order = reinterpret_cast<const int32_t*>(base + L.o_order);
    C.tout = reinterpret_cast<TaskOut*>(base + L.o_tout);
    C.sd = reinterpret_cast<const SignalDesc*>(base + L.o_sd);
    C.sigma = reinterpret_cast<const double*>(base + L.o_sigma);
    C.resid = base + L.o_resid;
    C.imfs = imfs ? imfs : (void*)(base + L.o_imfs);
    C.kt = reinterpret_cast<int32_t*>(base + L.o_kt);
    C.ky = base + L.o_ky;
    C.M = base + L.o_M;
    C.w1 = base + L.o_w1;
    C.w0 = L.has_w0 ? base + L.o_w0 : nullptr;
    C.imf_pad = L.imf_pad ? 1 : 0;
    C.resid_out = resid_out;
    C.r1 = base + L.o_r1;
    C.ri = reinterpret_cast<uint32_t*>(base + L.o_ri);
    C.scr = reinterpret_cast<double2*>(base + L.o_scr);
    C.x = x;
    C.noise = noise;
    C.knot_log = knot_log;
    C.mode_sifts = mode_sifts;
    C.slot_knots = L.slot_knots;
    C.slot_M = L.slot_M;
    C.slot_n = L.slot_n;
    C.slot_runs = L.slot_runs;
    C.segcap = L.segcap;
    C.kcap = L.kcap;
    C.n_tasks = (int32_t)L.td.size();
    C.n_signals = n_signals;
    C.trial_count = trial_count;
    C.csize = L.csize;
    C.max_sifts = p->max_sifts;
    C.max_imf = p->max_imf;
    C.min_extrema = p->min_extrema;
    C.end_mode = p->end_mode;
    C.rules = p->rules;
    C.noise_mode = p->noise_mode;
    C.B = L.B;
    C.S = L.S;
    C.scr_rows = L.scr_rows;
    C.nw = L.nw;
    C.tau = p->tau;
    C.noise_scale = p->eps;
    C.seed = p->seed;
    C.watchdog = p->watchdog != 0 ? p->watchdog : (1LL << 24);

    // the cleared header and the descriptors in one copy (a memset and three copies
    // of pageable memory each cost the call 5 to 8 us)
    std::unique_ptr<char[]> up(new (std::nothrow) char[L.o_tout]());
    if (!up) return EEMD_E_NOMEM;
    memcpy(up.get() + L.o_td, L.td.data(), sizeof(TaskDesc) * L.td.size());
    memcpy(up.get() + L.o_order, L.order.data(), sizeof(int32_t) * L.order.size());
    memcpy(up.get() + L.o_sd, L.sd.data(), sizeof(SignalDesc) * L.sd.size());
    if (cudaMemcpyAsync(base + L.o_hdr, up.get(), L.o_tout, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return EEMD_E_CUDA;
    if (knot_log) {
        const size_t nb = sizeof(int32_t) * 2 * L.td.size() * (size_t)p->max_imf * p->max_sifts;
        if (cudaMemsetAsync(knot_log, 0xff, nb, st) != cudaSuccess) return EEMD_E_CUDA;
    }
    if (mode_sifts) {
        if (cudaMemsetAsync(mode_sifts, 0, sizeof(int32_t) * L.td.size() * p->max_imf, st) != cudaSuccess)
            return EEMD_E_CUDA;
    }
    Tracer tr;
    tr.out = times;
    tr.st = st;
    rc = (p->dtype == EEMD_F64)
             ? run_typed<double>(p, L, C, imf_sum, mode_count, nsift, nmode, flags, st, tr)
             : run_typed<float>(p, L, C, imf_sum, mode_count, nsift, nmode, flags, st, tr);
    Header h;
    const bool ok = cudaMemcpyAsync(&h, C.hdr, sizeof(Header), cudaMemcpyDeviceToHost, st) == cudaSuccess;
    if (cudaStreamSynchronize(st) != cudaSuccess || !ok) return EEMD_E_CUDA;
    tr.finish();
    if (rc) return rc;
    if (h.error) return h.error;
    if (h.n_done != C.n_tasks) return EEMD_E_CUDA;
    return EEMD_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free entry point: the engine's scratch is this file-scope device
// array.  In host code `g_static_scratch` only names the symbol; its device
// address is looked up once per device with cudaGetSymbolAddress.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_static_scratch[EEMD_STATIC_SCRATCH_BYTES];

namespace {
constexpr int MAX_DEVICES = 64;
std::mutex g_static_mu;
void* g_static_addr[MAX_DEVICES] = {nullptr};
}  // namespace

extern "C" {

int32_t eemd_run_static(const eemd_params* p, const void* x, const int64_t* lengths, int32_t n_signals,
                        int32_t trial_begin, int32_t trial_count, const void* noise, void* imfs,
                        void* resid_out, double* imf_sum, int32_t* mode_count, int32_t* nsift,
                        int32_t* nmode, int32_t* mode_sifts, int32_t* knot_log, int32_t* flags,
                        void* stream) {
    Layout L;
    const int rc = make_layout(p, lengths, n_signals, trial_count, trial_begin, imfs != nullptr, L, false);
    if (rc) return rc;
    if (L.total > (size_t)EEMD_STATIC_SCRATCH_BYTES) return EEMD_E_STATIC_CAPACITY;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return EEMD_E_CUDA;
    if (dev < 0 || dev >= MAX_DEVICES) return EEMD_E_NOTSUP;
    void* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_static_mu);
        if (g_static_addr[dev] == nullptr) {
            void* addr = nullptr;
            if (cudaGetSymbolAddress(&addr, g_static_scratch) != cudaSuccess || addr == nullptr)
                return EEMD_E_CUDA;
            g_static_addr[dev] = addr;
        }
        base = g_static_addr[dev];
    }
    return eemd_run(p, x, lengths, n_signals, trial_begin, trial_count, noise, imfs, resid_out, imf_sum,
                    mode_count, nsift, nmode, mode_sifts, knot_log, flags, base,
                    (size_t)EEMD_STATIC_SCRATCH_BYTES, stream);
}

int32_t eemd_finalize(const eemd_params* p, const void* x, const int64_t* lengths, int32_t n_signals,
                      const double* imf_sum, const int32_t* mode_count, double* imf_mean, double* residual,
                      int32_t* n_modes, void* stream) {
    int rc = check_params(p);
    if (rc) return rc;
    if (!x || !lengths || n_signals < 1 || !imf_sum || !mode_count) return EEMD_E_BADARG;
    std::vector<SignalDesc> sd(n_signals);
    int64_t xo = 0, sumo = 0;
    for (int s = 0; s < n_signals; ++s) {
        if (lengths[s] < 1) return EEMD_E_BADARG;
        sd[s].x_off = xo;
        sd[s].r_off = xo;
        sd[s].sum_off = sumo;
        sd[s].n = (int32_t)lengths[s];
        sd[s].first_task = 0;
        xo += lengths[s];
        sumo += (int64_t)p->max_imf * lengths[s];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int s0 = 0; s0 < n_signals; s0 += FIN_BATCH) {
        const int ns = std::min(FIN_BATCH, n_signals - s0);
        FinBatch fb;
        memset(&fb, 0, sizeof(fb));
        int64_t bmax = 1;
        for (int i = 0; i < ns; ++i) {
            fb.sd[i] = sd[s0 + i];
            bmax = std::max<int64_t>(bmax, sd[s0 + i].n);
        }
        dim3 g((unsigned)((bmax + 255) / 256), (unsigned)ns);
        if (p->dtype == EEMD_F64)
            k_finalize<double><<<g, 256, 0, st>>>(fb, s0, p->max_imf, x, imf_sum, mode_count, imf_mean,
                                                  residual, n_modes);
        else
            k_finalize<float><<<g, 256, 0, st>>>(fb, s0, p->max_imf, x, imf_sum, mode_count, imf_mean,
                                                 residual, n_modes);
    }
    if (cudaStreamSynchronize(st) != cudaSuccess) return EEMD_E_CUDA;
    return cudaGetLastError() == cudaSuccess ? EEMD_OK : EEMD_E_CUDA;
}

}  // extern "C"
