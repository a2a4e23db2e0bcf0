// mpc_kernels.cuh -- the split-step propagator's sweeps over HBM and their helpers.
//
// Device layout of the field between sweeps ("slot layout"): the field is kept in the
// (x, y, omega) domain, omega in FFT position order.  Slots are interleaved in groups of
// SLO: element (slot s, pencil q = y*Nx + x) lives at ((s/SLO)*Nx*Ny + q)*SLO + s%SLO.
// SLO = 2 makes the t-rows of an 8-pencil tile 128 B; the default variants use SLO = 1 (rows of
// P * 8 B), which keeps every omega-plane contiguous for the plane passes.  With SLO = 1 the planes may
// be cut into blocks of YB rows, block-major: element (s, q) at (q / RB * Nt + s) * RB + q % RB with
// RB = YB * Nx pencils (RB = Nx Ny: whole planes).  A pencil tile's rows are then RB * 8 B apart instead
// of a whole plane (512 KB at 256x256: every row of a tile in another 2 MB page's quarter).
//
// Sweep 1, pencil pass (one CTA per tile of P neighbouring (x,y) pencils, all of t; mpc_step.cuh):
//   IFFT_t of -i*omega*S -> dA,  IFFT_t of S -> A,  nonlinear step N(dz) (Kerr, self-
//   steepening, ADK ionization with two affine prefix scans along t, plasma absorption and
//   defocusing, A *= exp(dz*A_nl)),  FFT_t -> S.
// Sweep 2, plane pass, the linear step factorised as (IFFT_x Rx FFT_x)(IFFT_y Ry D FFT_y):
//   either one kernel per unit of omega-planes on a thread-block cluster (FFT_y, Ry(ky) D(omega)
//   / (Nx Ny Nt), IFFT_y on columns; the columns become rows in one exchange between the
//   cluster's CTAs through distributed shared memory; FFT_x, Rx(kx), IFFT_x on rows), or two
//   kernels without clusters, the y part on column strips and the x part on row strips.
#pragma once
#include <cooperative_groups.h>
#include <type_traits>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mpc_fft.cuh"
#include "mpc_scale.h"
#include "mpc_tma.cuh"

namespace cg = cooperative_groups;

namespace mpc {

constexpr int kThreads = 512;          // threads of a one-CTA-per-SM launch (128 registers each)
constexpr int kTilePoints = 16384;     // default pencil tile: P * Nt complex points (128 KB)
// butterflies of a pencil thread unrolled together per FFT stage (the plane sweep keeps 1: its
// kernels are at the register limit)
#ifndef MPC_PENCIL_UNROLL
#define MPC_PENCIL_UNROLL 4
#endif
constexpr int kPencilUnroll = MPC_PENCIL_UNROLL;
// FP32 constants of the nonlinear step, computed on the host in FP64.
struct NLConst {
    float sst_c;     // gamma2 / (w0 fs^2), 0 when self-steepening is off
    float I_scale;   // intensity [W/m^2] per unit |a|^2
    float E_c;       // field in atomic units = sqrt(I) * E_c
    float inv_E_c;   // 1 / E_c
    float l2K1[2], l2K3[2], K5[2], K3l2e[2];  // ADK: log2 K1, log2 K3, K5, K3 log2(e) / 3
    float Kon;       // deltat / T0
    float Kuv;       // sigma_coll rho_nt v_e per unit F (v_e = e E0 / (sqrt 2 me w0))
    float K4w0;      // k0 w0^2 / (n0 rho_c)
    float w0sq;      // w0^2
    float inv_w0;    // 1 / w0
    float invI1_Kon; // Kon / I1 (I1 in eV, as the reference divides by it)
    int plasma;      // 1 = ionization and plasma terms on
    // The same step in x = |a|^2, for mpc_step.cuh (set from FP64 by nl_setup):
    float e0[2], e1[2], e2[2];  // log2 of the stage's probability per slice = e0 - e1 log2 x - e2 / sqrt x
    float kv;        // v = u / w0 per sqrt x
    float kb;        // b = kb v x / (1 + v^2)
    float x2thr;     // for every x below this the second stage flushes to zero and b < 1/2
    // and, for a step length dz (nl_set_dz): exponents per unit x, dA conj(A) and ion fraction
    float gam_dz, sst_dz, pl_dz;
    float inv_dz;
};

// Pencil tile view: line = pencil p, element (pos, p).  For P < 16 a pad of P slots every
// 2^SH positions and every 32 positions keeps the FFT stages and the per-thread t walks free
// of shared-memory bank conflicts (SH = 4 for P = 8, 3 for P = 4).  The pad depends on pos
// only through pos >> SH and pos >> 5, so a walk of CH samples from a multiple of CH has the
// same offsets everywhere, at(t0 + i, p) - at(t0, p) == walk(i), for CH = 32 and, when SH = 4,
// for CH = 16.
template <int NT, int P>
struct PencilView {
    static constexpr int NLINES = P;
    static constexpr int SH = (P < 8) ? 3 : 4;
    static constexpr __host__ __device__ __forceinline__ int at(int pos, int p) {
        if constexpr (P < 16) return pos * P + p + P * ((pos >> SH) + (pos >> 5));
        else return pos * P + p;
    }
    static constexpr __host__ __device__ __forceinline__ int walk(int i) { return at(i, 0) - at(0, 0); }
    static constexpr int SIZE = (P < 16) ? (NT * P + P * ((NT >> SH) + NT / 32)) : NT * P;
    static_assert(P >= 4, "pencil tile of at least 4 pencils");
};

enum PencilMode : int {
    PM_ENTRY_C128 = 0,  // real-space complex128 (reference layout, physical units) -> S
    PM_ENTRY_C64 = 1,   // real-space complex64 (reference layout, device units) -> S
    PM_STEP = 2,        // S -> N(dz) -> S (step_kernel)
    PM_EXIT_C128 = 3,   // S -> real-space complex128 (physical units) + per-pencil energy
    PM_EXIT_C64 = 4,    // S -> real-space complex64 (device units) + per-pencil energy
    PM_DIAG = 5,        // S -> temporal profile, spectrum and pencil energies (diag_kernel)
    PM_IONIZ = 6,       // real-space complex128 -> tau_c, freeelectrons_sp (FP64, reference layout)
};

struct PencilArgs {
    const void* in;          // input field (layout by mode)
    void* out;               // output field (may alias in)
    const float2* tw;        // W_Nt table, packed (mpc_fft.cuh Twiddles)
    const float* wpos;       // omega of each t position (FFT position order), Nt
    double* pencil_energy;   // EXIT, DIAG: sum_t |A|^2 per pencil, Nx*Ny, or null
    double* parts;           // DIAG: a row per CTA: its sums of |A|^2 per t (Nt) and |S|^2 per position (Nt)
    double* tau_out;         // IONIZ: tau_c, reference layout
    double* fe_out;          // IONIZ: freeelectrons_sp, reference layout
    unsigned int* stats;     // STEP: running maxima of the step (step_nonlinear), or null
    unsigned int* err;       // STEP: error word (KernelError)
    double in_scale;         // ENTRY: input multiplier (to device units, includes 1/Nt)
    double out_scale;        // EXIT/DIAG: output multiplier (from device units)
    int NP;                  // Nx * Ny
    int ntiles;              // NP / P
    int lrb;                 // log2 of the pencils of a row block (SLO = 1; NP when not blocked)
    NLConst nl;
};

// ---------------------------------------------------------------------------------------
// Affine-map scans of the ionization prefix (plasma.c:223-231, run forward in t).
//   R_k = (1 - b_k)(R_{k-1} + a_k) + b_k          map (B, C): R -> (1-B) R + C
//   (u, v)_{k+1} = (u_k + c2_k v_k, g_k - u_k)     map (M, o): x -> M x + o
// with a_k = W1 Kon, b_k = Wava Kon, c2_k = W2 Kon, g_k = 1 - exp(-R_k); u = ions2,
// v = ions1, both zero before the first slice; fe_sp[k] = (v_k + 2 u_k) sigma_k.
// Chunk maps are composed in FP32 inside a thread's CH points and across chunks in FP64.  Across
// chunks the R map is held as (D, C) = (1 - B, C), R -> D R + C, so that composing two maps is one
// FP64 product and one FP64 FMA (GB300 issues FP64 at 1/64 of its FP32 rate).  D keeps 1 - B to
// FP64's absolute precision (1e-16), which is what the product D R needs; B's own relative
// precision does not enter.
// ---------------------------------------------------------------------------------------
struct MapR { double D, C; };
struct MapUV { double m00, m01, m10, m11, o0, o1; };

__device__ __forceinline__ MapR compose(const MapR& first, const MapR& then) {
    MapR r;
    r.D = then.D * first.D;
    r.C = fma(then.D, first.C, then.C);
    return r;
}
__device__ __forceinline__ MapUV compose(const MapUV& f, const MapUV& t) {
    MapUV r;
    r.m00 = t.m00 * f.m00 + t.m01 * f.m10;
    r.m01 = t.m00 * f.m01 + t.m01 * f.m11;
    r.m10 = t.m10 * f.m00 + t.m11 * f.m10;
    r.m11 = t.m10 * f.m01 + t.m11 * f.m11;
    r.o0 = t.m00 * f.o0 + t.m01 * f.o1 + t.o0;
    r.o1 = t.m10 * f.o0 + t.m11 * f.o1 + t.o1;
    return r;
}
template <class M>
__device__ __forceinline__ M map_ident();
template <>
__device__ __forceinline__ MapR map_ident<MapR>() { return MapR{1.0, 0.0}; }
template <>
__device__ __forceinline__ MapUV map_ident<MapUV>() { return MapUV{1.0, 0.0, 0.0, 1.0, 0.0, 0.0}; }

template <class M>
__device__ __forceinline__ M shfl_up_map(const M& m, int off) {
    M r;
    double* dst = reinterpret_cast<double*>(&r);
    const double* src = reinterpret_cast<const double*>(&m);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(M) / sizeof(double)); i++) dst[i] = __shfl_up_sync(0xffffffffu, src[i], off);
    return r;
}

// Exclusive scan over the TPP chunk maps of each of P pencils, in place in `maps`
// (index p * TPP + c).  One warp per pencil; each lane composes TPP/32 (or 1) chunks.
template <class M, int P, int TPP>
__device__ __forceinline__ void scan_chunks(M* maps, int tid) {
    const int warp = tid >> 5, lane = tid & 31;
    constexpr int NW = P * TPP / 32;       // the CTA has one thread per chunk
    constexpr int CPL = (TPP + 31) / 32;
    for (int p = warp; p < P; p += NW) {
        M* row = maps + p * TPP;
        M acc = map_ident<M>();
        const int c0 = lane * CPL;
#pragma unroll
        for (int j = 0; j < CPL; j++)
            if (c0 + j < TPP) acc = compose(acc, row[c0 + j]);
        // inclusive warp scan of lane aggregates
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const M prev = shfl_up_map(acc, off);
            if (lane >= off) acc = compose(prev, acc);
        }
        M excl = shfl_up_map(acc, 1);
        if (lane == 0) excl = map_ident<M>();
        __syncwarp();
#pragma unroll
        for (int j = 0; j < CPL; j++) {
            if (c0 + j < TPP) {
                const M own = row[c0 + j];
                row[c0 + j] = excl;
                excl = compose(excl, own);
            }
        }
        __syncwarp();
    }
}

// Small-argument elementary functions, from their Taylor series (|x| below the stated bound;
// the CUDA library function is called outside it).  Per split step the nonlinear phase is
// < 0.25 rad and the amplitude exponent < 1/64, so the series branch is the one taken.
// 1 - exp(-x), x >= 0: alternating series to x^6/720 (relative truncation < x^6/5040 < 8e-10)
__device__ __forceinline__ float one_minus_exp_neg(float x) {
    if (x < 0.125f)
        return x * (1.0f - x * (0.5f - x * (1.0f / 6.0f - x * (1.0f / 24.0f - x * (1.0f / 120.0f - x * (1.0f / 720.0f))))));
    return 1.0f - expf(-x);
}
// exp(x): series to x^4/24 for |x| < 1/64 (truncation < |x|^5/120 < 1e-11)
__device__ __forceinline__ float exp_small(float x) {
    if (fabsf(x) < 0.015625f) return 1.0f + x * (1.0f + x * (0.5f + x * (1.0f / 6.0f + x * (1.0f / 24.0f))));
    return expf(x);
}
// sin and cos: series to x^7/7! and x^8/8! for |x| < 1/4 (truncation < 3e-11)
__device__ __forceinline__ void sincos_small(float x, float* sn, float* cs) {
    if (fabsf(x) < 0.25f) {
        const float x2 = x * x;
        *sn = x * (1.0f - x2 * (1.0f / 6.0f - x2 * (1.0f / 120.0f - x2 * (1.0f / 5040.0f))));
        *cs = 1.0f - x2 * (0.5f - x2 * (1.0f / 24.0f - x2 * (1.0f / 720.0f - x2 * (1.0f / 40320.0f))));
    } else {
        sincosf(x, sn, cs);
    }
}

// Per-point ionization coefficients of one sample (plasma.c:133-213 in FP32, A18 fix
// applied).  The ADK rates are evaluated in the log2 domain:
//   log2 W = log2 K1 + K5 (log2 K3 - log2 F) - K3 / (3 F ln 2).
// Second-stage probabilities c2 below 2^-60 per slice are flushed to zero: their whole-pencil
// effect on ions2 is < Nt 2^-60 < 2e-15, far below FP32 resolution, and a tile without any
// second-stage ionization then skips the (ions2, ions1) scan, which is exact there.
constexpr float kC2Flush = 8.673617e-19f;   // 2^-60
struct IonPoint {
    float a, b, c2;  // scan coefficients W1 Kon, Wava Kon, W2 Kon
    float sigma;     // K4 tau_c / (1 + w0^2 tau_c^2)
    float u;         // 1 / tau_c = sigma_coll rho_nt v_e
};
// SECOND = false: the second stage is known to flush to zero for every sample of the tile (the
// first walk's test), so its rate is not evaluated and c2 = 0, the value it would flush to.
template <bool SECOND = true>
__device__ __forceinline__ IonPoint ion_point(float2 a, const NLConst& c) {
    IonPoint r;
    float I = fmaf(a.x, a.x, a.y * a.y) * c.I_scale;
    if (I == 0.0f) I = 1e-30f;                   // plasma.c:136-138
    const float rs = rsqrtf(I);
    const float F = I * rs * c.E_c;              // |E| in atomic units
    const float invF = rs * c.inv_E_c;
    const float l2F = __log2f(F);
    float w[2] = {0.0f, 0.0f};
#pragma unroll
    for (int st = 0; st < (SECOND ? 2 : 1); st++) {
        const float e2 = c.l2K1[st] + c.K5[st] * (c.l2K3[st] - l2F) - c.K3l2e[st] * invF;
        w[st] = (e2 > -126.0f) ? exp2f(e2) : 0.0f;
    }
    const float u = c.Kuv * F;
    const float qw = __fdividef(c.K4w0, fmaf(u, u, c.w0sq));
    r.sigma = qw * u * c.inv_w0;
    r.u = u;
    r.a = w[0] * c.Kon;
    r.b = r.sigma * I * c.invI1_Kon;
    if constexpr (SECOND) {
        const float c2 = w[1] * c.Kon;
        r.c2 = (c2 >= kC2Flush) ? c2 : 0.0f;
    } else {
        r.c2 = 0.0f;
    }
    return r;
}

// The first walk of the ionization scan needs only a and b of each sample, and whether any
// sample of the tile may have a second-stage probability c2 at or above the flush threshold.
// That is decided on the exponent, e2 > log2(threshold / Kon) - 1, without the second exp2: a
// conservative test (a tile flagged whose c2 all flush runs the exact (ions2, ions1) scan with
// zero coefficients).
struct IonAB {
    float a, b;
    bool second;
};
__device__ __forceinline__ float ion_second_threshold(const NLConst& c) { return __log2f(kC2Flush / c.Kon) - 1.0f; }
__device__ __forceinline__ IonAB ion_point_ab(float2 a, const NLConst& c, float e2thr) {
    IonAB r;
    float I = fmaf(a.x, a.x, a.y * a.y) * c.I_scale;
    if (I == 0.0f) I = 1e-30f;                   // plasma.c:136-138
    const float rs = rsqrtf(I);
    const float F = I * rs * c.E_c;
    const float invF = rs * c.inv_E_c;
    const float l2F = __log2f(F);
    const float e1 = c.l2K1[0] + c.K5[0] * (c.l2K3[0] - l2F) - c.K3l2e[0] * invF;
    const float e2 = c.l2K1[1] + c.K5[1] * (c.l2K3[1] - l2F) - c.K3l2e[1] * invF;
    const float u = c.Kuv * F;
    const float qw = __fdividef(c.K4w0, fmaf(u, u, c.w0sq));
    r.a = ((e1 > -126.0f) ? exp2f(e1) : 0.0f) * c.Kon;
    r.b = qw * u * c.inv_w0 * I * c.invI1_Kon;
    r.second = e2 > e2thr;
    return r;
}

// Ionization outputs of a tile holding A(t) of P pencils in shared memory (natural t order): tau_c and
// freeelectrons_sp (plasma.c:118-245) in the reference layout.  Thread (p = tid % P, ch = tid / P)
// walks the CH samples t = CH ch .. CH ch + CH - 1 of pencil p.
template <int NT, int P, int CH = 32>
__device__ __forceinline__ void ioniz_tile(const float2* s, const NLConst& c, void* scan_mem, int tid, double* tau_out,
                                           double* fe_out, int q0, int NP) {
    using V = PencilView<NT, P>;
    static_assert(CH == 32 || (CH == 16 && V::SH == 4), "walk offsets need a chunk-aligned pad");
    constexpr int TPP = NT / CH;
    const int p = tid % P;
    const int ch = tid / P;
    const int t0 = ch * CH;
    const float2* w = s + V::at(t0, p);   // this thread's CH samples: w[V::walk(i)]
    MapR* mr = reinterpret_cast<MapR*>(scan_mem);
    MapUV* muv = reinterpret_cast<MapUV*>(scan_mem);
    // S1: chunk map of the R recurrence (FP32 within the chunk)
    int any2 = 0;
    {
        float B = 0.0f, C = 0.0f;
        const float e2thr = ion_second_threshold(c);
#pragma unroll 8
        for (int i = 0; i < CH; i++) {
            const IonAB ip = ion_point_ab(w[V::walk(i)], c, e2thr);
            const float Ck = fmaf(1.0f - ip.b, ip.a, ip.b);
            C = fmaf(1.0f - ip.b, C, Ck);
            B = fmaf(-B, ip.b, B + ip.b);
            any2 |= ip.second;
        }
        mr[p * TPP + ch] = MapR{1.0 - (double)B, (double)C};
    }
    any2 = __syncthreads_or(any2);
    scan_chunks<MapR, P, TPP>(mr, tid);   // carries across chunks in FP64
    __syncthreads();
    const float Rin = (float)mr[p * TPP + ch].C;
    float u = 0.0f, v = (Rin > 0.0f) ? one_minus_exp_neg(Rin) : 0.0f;
    if (any2) {
        __syncthreads();
        // S2: chunk map of the (ions2, ions1) recurrence
        float R = Rin;
        float m00 = 1.f, m01 = 0.f, m10 = 0.f, m11 = 1.f, o0 = 0.f, o1 = 0.f;
#pragma unroll 4
        for (int i = 0; i < CH; i++) {
            const IonPoint ip = ion_point<true>(w[V::walk(i)], c);
            R = fmaf(1.0f - ip.b, R + ip.a, ip.b);
            const float g = one_minus_exp_neg(R);
            const float n00 = fmaf(ip.c2, m10, m00), n01 = fmaf(ip.c2, m11, m01);
            const float no0 = fmaf(ip.c2, o1, o0), no1 = g - o0;
            m10 = -m00;
            m11 = -m01;
            m00 = n00;
            m01 = n01;
            o1 = no1;
            o0 = no0;
        }
        muv[p * TPP + ch] = MapUV{m00, m01, m10, m11, o0, o1};
        __syncthreads();
        scan_chunks<MapUV, P, TPP>(muv, tid);
        __syncthreads();
        u = (float)muv[p * TPP + ch].o0;
        v = (float)muv[p * TPP + ch].o1;
    }
    // S3: the outputs.  Tiles without second-stage ionization (any2 == 0) take the walk without the
    // second rate.
    auto walk = [&](auto second) {
        float R = Rin;
#pragma unroll 4
        for (int i = 0; i < CH; i++) {
            const IonPoint ip = ion_point<decltype(second)::value>(w[V::walk(i)], c);
            R = fmaf(1.0f - ip.b, R + ip.a, ip.b);
            const float g = one_minus_exp_neg(R);
            const float ions = fmaf(2.0f, u, v);     // state before slice t (plasma.c:238-241)
            const float nu = fmaf(ip.c2, v, u);
            v = g - u;
            u = nu;
            const size_t gi = (size_t)(t0 + i) * NP + q0 + p;
            tau_out[gi] = 1.0 / (double)ip.u;
            fe_out[gi] = (double)ions * (double)ip.sigma;
        }
    };
    if (any2) walk(std::true_type{});
    else walk(std::false_type{});
}

// Block-wide maximum of each component of v into stats[0..3] (non-negative floats, whose
// bit patterns order like the values); one atomic per component and CTA.
template <int TH>
__device__ __forceinline__ void stats_max(float4 v, unsigned int* stats, float* red, int tid) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x = fmaxf(v.x, __shfl_xor_sync(0xffffffffu, v.x, o));
        v.y = fmaxf(v.y, __shfl_xor_sync(0xffffffffu, v.y, o));
        v.z = fmaxf(v.z, __shfl_xor_sync(0xffffffffu, v.z, o));
        v.w = fmaxf(v.w, __shfl_xor_sync(0xffffffffu, v.w, o));
    }
    if ((tid & 31) == 0) reinterpret_cast<float4*>(red)[tid >> 5] = v;
    __syncthreads();
    if (tid < 4) {
        float m = 0.0f;
        for (int w = 0; w < TH / 32; w++) m = fmaxf(m, red[4 * w + tid]);
        atomicMax(&stats[tid], __float_as_uint(m));
    }
}

// ---------------------------------------------------------------------------------------
// Pencil pass
// ---------------------------------------------------------------------------------------
// Shared memory of a pencil CTA: [field tile][scan maps][W_Nt twiddles].
// One thread per CH-sample chunk of the nonlinear walk: TH = P * Nt / CH threads (CH = 16 puts
// 1024 threads, 64 registers each, in a CTA: twice the warps to hide latency).
template <int NT, int P, int SLO, int CH = 32>
struct PencilCfg {
    using View = PencilView<NT, P>;
    static constexpr int TPP = NT / CH;                 // chunks per pencil
    static constexpr int TH = P * TPP;                  // threads per CTA
    static constexpr int SMEM_FIELD = View::SIZE * 8;  // bytes
    static constexpr int SMEM_SCAN = P * TPP * (int)sizeof(MapUV);
    static constexpr int SMEM_TW = twiddle_bytes(NT);
    static constexpr int SMEM = SMEM_FIELD + SMEM_SCAN + SMEM_TW;
    static_assert(TH % 32 == 0 && TH <= 1024, "pencil CTA size");
    static_assert((P * SLO) % 2 == 0, "rows must be whole float4s");
};

// The tile of pencils that starts at q0 in the slot layout: element (position pos, pencil q0 + p) is at
// tile_base(...)[tile_elem(pos, p)].  lrb: log2 of the row block's pencils (SLO = 2: of Nx Ny).
template <int NT, int SLO, class T>
__device__ __forceinline__ T* tile_base(T* g, int q0, int lrb) {
    if constexpr (SLO == 1) return g + ((((size_t)(q0 >> lrb) * NT) << lrb) + (q0 & ((1 << lrb) - 1)));
    else return g + (size_t)q0 * SLO;
}
template <int SLO>
__device__ __forceinline__ size_t tile_elem(int pos, int p, int lrb) {
    return SLO == 1 ? ((size_t)pos << lrb) + p : ((((size_t)(pos / SLO) << lrb) + p) * SLO + pos % SLO);
}

// Element order of the two complex values of a float4 row chunk.  For SLO = 2 the pair is
// (pos 2r, pos 2r + 1) of one pencil; odd rows store them in the opposite order so that
// the four rows a warp touches fall on both halves of the shared-memory banks.
// load a slot-layout tile into shared memory
template <int NT, int P, int SLO, int TH>
__device__ __forceinline__ void load_tile(float2* s, const float2* __restrict__ g, int q0, int lrb, int tid) {
    using V = PencilView<NT, P>;
    constexpr int F4_PER_ROW = P * SLO / 2;
    constexpr int ROWS = NT / SLO;
    const float4* g4 = reinterpret_cast<const float4*>(tile_base<NT, SLO>(g, q0, lrb));
    for (int f = tid; f < ROWS * F4_PER_ROW; f += TH) {
        const int row = f / F4_PER_ROW, c = f - row * F4_PER_ROW;
        const size_t gi = (((size_t)row << lrb) * SLO) / 2 + c;
        const float4 v = __ldg(&g4[gi]);
        int pos0, p0, pos1, p1;
        if constexpr (SLO == 2) { pos0 = 2 * row; pos1 = pos0 + 1; p0 = p1 = c; }
        else { pos0 = pos1 = row; p0 = 2 * c; p1 = p0 + 1; }
        const float2 e0 = make_float2(v.x, v.y), e1 = make_float2(v.z, v.w);
        if (SLO == 2 && (row & 1)) {
            s[V::at(pos1, p1)] = e1;
            s[V::at(pos0, p0)] = e0;
        } else {
            s[V::at(pos0, p0)] = e0;
            s[V::at(pos1, p1)] = e1;
        }
    }
}

template <int NT, int P, int SLO, int TH>
__device__ __forceinline__ void store_tile(const float2* s, float2* __restrict__ g, int q0, int lrb, int tid) {
    using V = PencilView<NT, P>;
    constexpr int F4_PER_ROW = P * SLO / 2;
    constexpr int ROWS = NT / SLO;
    float4* g4 = reinterpret_cast<float4*>(tile_base<NT, SLO>(g, q0, lrb));
    for (int f = tid; f < ROWS * F4_PER_ROW; f += TH) {
        const int row = f / F4_PER_ROW, c = f - row * F4_PER_ROW;
        const size_t gi = (((size_t)row << lrb) * SLO) / 2 + c;
        int pos0, p0, pos1, p1;
        if constexpr (SLO == 2) { pos0 = 2 * row; pos1 = pos0 + 1; p0 = p1 = c; }
        else { pos0 = pos1 = row; p0 = 2 * c; p1 = p0 + 1; }
        float2 e0, e1;
        if (SLO == 2 && (row & 1)) {
            e1 = s[V::at(pos1, p1)];
            e0 = s[V::at(pos0, p0)];
        } else {
            e0 = s[V::at(pos0, p0)];
            e1 = s[V::at(pos1, p1)];
        }
        g4[gi] = make_float4(e0.x, e0.y, e1.x, e1.y);
    }
}

// The passes between real space and the slot layout and the ionization outputs (the split step is
// step_kernel, the diagnostics diag_kernel, mpc_step.cuh).
template <int NT, int P, int SLO, int MODE, int CH = 32>
__global__ void __launch_bounds__(PencilCfg<NT, P, SLO, CH>::TH, (PencilCfg<NT, P, SLO, CH>::TH >= kThreads ? 1 : 2))
    pencil_kernel(PencilArgs args) {
    using Cfg = PencilCfg<NT, P, SLO, CH>;
    using V = typename Cfg::View;
    constexpr int TH = Cfg::TH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    void* scan_mem = smem_raw + Cfg::SMEM_FIELD;
    unsigned char* tw_mem = smem_raw + Cfg::SMEM_FIELD + Cfg::SMEM_SCAN;
    const int tid = threadIdx.x;
    const int NP = args.NP;
    stage_twiddles<NT, TH>(tw_mem, args.tw, tid);
    const Twiddles tw = Twiddles::packed(tw_mem, NT);
    const IntScale os = int_scale(args.out_scale);   // EXIT
    __syncthreads();


    for (int tile = blockIdx.x; tile < args.ntiles; tile += gridDim.x) {
        const int q0 = tile * P;
        if constexpr (MODE == PM_IONIZ) {
            for (int f = tid; f < NT * P; f += TH) {
                const int t = f / P, p = f - (f / P) * P;
                const size_t gi = (size_t)t * NP + q0 + p;
                const double2 v = __ldg(&reinterpret_cast<const double2*>(args.in)[gi]);
                s[V::at(t, p)] = make_float2((float)(v.x * args.in_scale), (float)(v.y * args.in_scale));
            }
            __syncthreads();
            ioniz_tile<NT, P, CH>(s, args.nl, scan_mem, tid, args.tau_out, args.fe_out, q0, NP);
            __syncthreads();
        } else if constexpr (MODE == PM_ENTRY_C128 || MODE == PM_ENTRY_C64) {
            // real-space input, reference layout A[t*NP + q]
            for (int f = tid; f < NT * P; f += TH) {
                const int t = f / P, p = f - (f / P) * P;
                const size_t gi = (size_t)t * NP + q0 + p;
                float2 e;
                if constexpr (MODE == PM_ENTRY_C128) {
                    const double2 v = __ldg(&reinterpret_cast<const double2*>(args.in)[gi]);
                    e = make_float2((float)(v.x * args.in_scale), (float)(v.y * args.in_scale));
                } else {
                    e = cscale(__ldg(&reinterpret_cast<const float2*>(args.in)[gi]), (float)args.in_scale);
                }
                s[V::at(t, p)] = e;
            }
            __syncthreads();
            dif_all<NT, NT, V, TH, kPencilUnroll>(s, tw, tid);
            store_tile<NT, P, SLO, TH>(s, reinterpret_cast<float2*>(args.out), q0, args.lrb, tid);
            __syncthreads();
        } else if constexpr (MODE == PM_EXIT_C128 || MODE == PM_EXIT_C64) {
            load_tile<NT, P, SLO, TH>(s, reinterpret_cast<const float2*>(args.in), q0, args.lrb, tid);
            __syncthreads();
            dit_all<NT, NT, V, TH, kPencilUnroll>(s, tw, tid);
            {
                for (int f = tid; f < NT * P; f += TH) {
                    const int t = f / P, p = f - (f / P) * P;
                    const size_t gi = (size_t)t * NP + q0 + p;
                    const float2 e = s[V::at(t, p)];
                    if constexpr (MODE == PM_EXIT_C128) {
                        reinterpret_cast<double2*>(args.out)[gi] =
                            make_double2(scaled_double(e.x, args.out_scale, os), scaled_double(e.y, args.out_scale, os));
                    } else {
                        reinterpret_cast<float2*>(args.out)[gi] = cscale(e, (float)args.out_scale);
                    }
                }
                // per-pencil energy sum_t |A|^2 (physical units)
                if (args.pencil_energy) {
                    const int p = tid % P, part = tid / P;           // TH/P partial sums per pencil
                    constexpr int PARTS = TH / P;
                    float acc = 0.0f;
                    for (int t = part; t < NT; t += PARTS) {
                        const float2 e = s[V::at(t, p)];
                        acc = fmaf(e.x, e.x, fmaf(e.y, e.y, acc));
                    }
                    double* red = reinterpret_cast<double*>(scan_mem);
                    __syncthreads();
                    red[part * P + p] = (double)acc;
                    __syncthreads();
                    if (tid < P) {
                        double tot = 0.0;
                        for (int k = 0; k < PARTS; k++) tot += red[k * P + tid];
                        args.pencil_energy[q0 + tid] = tot * args.out_scale * args.out_scale;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------------------
// Plane pass
// ---------------------------------------------------------------------------------------
// These kernels start while the kernel before still runs (pdl_wait), so the field is written during their
// life, which ld.global.nc (__ldg) does not allow: it is read with __ldcg or by bulk copies.  The factor and
// lens tables are read with __ldg (a compiler may move such a load above the wait): the first plane sweep
// after their kernels is launched the ordinary way, when those have ended (PlaneArgs::overlap).  With plain
// loads for the tables the one-pass plane kernel is slower on small grids (16x16x64 15.0 -> 15.6 us).
// Linear-step factors as double-float complex numbers (x, y = high parts, z, w = low parts,
// split from FP64).  Rounded once to complex64 the same factor would be applied every step
// with the same rounding error, which adds up coherently over thousands of steps; the
// low parts remove that systematic error.
struct PlaneTables {
    const float4* Rx;   // Nx, x position order: exp(-i zd kx^2 / (2 k0))
    const float4* RyD;  // Ny * Nt, [y position][slot position]: Ry(ky) D(omega) scale
    const float4* RyDT; // the same factors slot-major, Nt * Ny: [slot position][y position]
};

struct PlaneArgs {
    const float2* in;
    float2* out;
    const float2* twx;       // W_Nx table, packed (mpc_fft.cuh Twiddles)
    const float2* twy;       // W_Ny table, packed
    PlaneTables t1;      // first (or only) linear operator
    PlaneTables t2;      // second half after the mirror lens (lens != 0)
    const float2* lensx; // exp(-i k0 x^2 / roc), real x order
    const float2* lensy;
    int lens;            // 1: L(t1) -> lens -> L(t2)
    int Nt;
    int NP;
    int nunits;          // number of cluster work units
    unsigned int* err;   // error word of the TMA-staged kernels (KernelError)
    int overlap;         // host: the sweep's first kernel may start while the kernel before it drains
};

template <int NX, int NY, int CL, int PB, int SLO>
struct PlaneCfg {
    static constexpr int RY = NY / CL;   // rows per CTA (row view)
    static constexpr int CX = NX / CL;   // columns per CTA (column view)
    static constexpr int RS = CX + 1;    // padded row stride
    static constexpr int RSZ = PB * RY * RS;  // region (one partner block), complex64
    static constexpr int SIZE = CL * RSZ;
    static constexpr int SMEM = SIZE * 8 + twiddle_bytes(NX) + twiddle_bytes(NY);
    static_assert(SLO == 1 || PB == SLO, "interleaved slots are processed together");
    static_assert((RSZ % 2) == 0, "regions are moved as float4");
};

template <int NX, int NY, int CL, int PB, int SLO>
struct RowView {
    using C = PlaneCfg<NX, NY, CL, PB, SLO>;
    static constexpr int NLINES = PB * C::RY;
    static constexpr __host__ __device__ __forceinline__ int at(int x, int l) {
        return (x / C::CX) * C::RSZ + l * C::RS + (x % C::CX);
    }
};
template <int NX, int NY, int CL, int PB, int SLO>
struct ColView {
    using C = PlaneCfg<NX, NY, CL, PB, SLO>;
    static constexpr int NLINES = PB * C::CX;
    static constexpr __host__ __device__ __forceinline__ int at(int y, int l) {
        const int pl = l / C::CX, xl = l - pl * C::CX;
        return (y / C::RY) * C::RSZ + (pl * C::RY + (y % C::RY)) * C::RS + xl;
    }
};

// Swap region g of this CTA with region `rank` of CTA g, for every g != rank.
template <int CL, int RSZ, int NTHR>
__device__ __forceinline__ void cluster_exchange(float2* s, cg::cluster_group& cluster, int rank, int tid) {
    if constexpr (CL > 1) {
        constexpr int F4 = RSZ / 2;               // float4 per region
        constexpr int KR = (CL >= 4) ? 2 : 1;     // partners per round
        constexpr int PER = (KR * F4 + NTHR - 1) / NTHR;
        cluster.sync();
        for (int k0 = 1; k0 < CL; k0 += KR) {
            float4 buf[PER];
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const int f = tid + i * NTHR;
                if (f < KR * F4) {
                    const int kk = k0 + f / F4;
                    if (kk < CL) {
                        const int g = rank ^ kk;
                        const float4* rem = reinterpret_cast<const float4*>(cluster.map_shared_rank(s, g));
                        buf[i] = rem[rank * F4 + (f % F4)];
                    }
                }
            }
            cluster.sync();
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const int f = tid + i * NTHR;
                if (f < KR * F4) {
                    const int kk = k0 + f / F4;
                    if (kk < CL) {
                        const int g = rank ^ kk;
                        reinterpret_cast<float4*>(s)[g * F4 + (f % F4)] = buf[i];
                    }
                }
            }
        }
        __syncthreads();
    }
}

// Ry(py) D(slot) (double-float) at column-view positions y (FFT position order) of line
// l = pl * CX + xl, plane pl of the unit.
template <int CX, int SLO, int PB>
struct YFactors {
    const float4* RyD;
    int Nt, unit;
    template <int R>
    __device__ __forceinline__ void operator()(float2 (&v)[R], int y0, int line) const {
        const int pl = line / CX;
        const int slot = (SLO == 1) ? unit * PB + pl : unit * SLO + pl;
        const float4* f = RyD + (size_t)y0 * Nt + slot;
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = cmul_df(v[q], __ldg(&f[(size_t)q * Nt]));
    }
};
// Rx(px) (double-float) at row-view positions x, from shared or global memory
struct XFactorsAny {
    const float4* Rx;
    template <int R>
    __device__ __forceinline__ void operator()(float2 (&v)[R], int x0, int) const {
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = cmul_df(v[q], Rx[x0 + q]);
    }
};
// Rx(px) (double-float) at row-view positions x (FFT position order).
struct XFactors {
    const float4* Rx;
    template <int R>
    __device__ __forceinline__ void operator()(float2 (&v)[R], int x0, int) const {
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = cmul_df(v[q], __ldg(&Rx[x0 + q]));
    }
};

// Move this CTA's share of a unit between global and shared memory: ROWS, the rows
// y in [rank RY, rank RY + RY) (row view, NX * 8 B contiguous per row and plane); otherwise
// the columns x in [rank CX, rank CX + CX) of every row (column view, CX * 8 B per row and
// plane).  STORE: shared -> global.  SLO == 2: one float4 holds both slots of one x.
template <int NX, int NY, int CL, int PB, int SLO, int NTHR, bool ROWS, bool STORE>
__device__ __forceinline__ void plane_move(float2* s, const float2* gin, float2* gout,
                                           int rank, int unit, int NP, int tid) {
    using C = PlaneCfg<NX, NY, CL, PB, SLO>;
    using RV = RowView<NX, NY, CL, PB, SLO>;
    using CV = ColView<NX, NY, CL, PB, SLO>;
    constexpr int W = ROWS ? NX : C::CX;    // x extent moved per row
    constexpr int NR = ROWS ? C::RY : NY;   // rows moved per plane block
    static_assert((W * SLO) % 2 == 0, "rows move as float4");
    constexpr int F4_ROW = W * SLO / 2;
    const int x0 = ROWS ? 0 : rank * C::CX;
    const int y0 = ROWS ? rank * C::RY : 0;
#pragma unroll 8
    for (int f = tid; f < PB / SLO * NR * F4_ROW; f += NTHR) {
        const int c = f % F4_ROW;
        const int r = f / F4_ROW;
        const int yr = r % NR, plb = r / NR;  // plb: plane block (SLO == 1: plane)
        const int y = y0 + yr;
        size_t gi;
        int i0, i1;
        if constexpr (SLO == 1) {
            gi = ((size_t)(unit * PB + plb) * NP + (size_t)y * NX + x0) / 2 + c;
            if constexpr (ROWS) {
                i0 = RV::at(2 * c, plb * C::RY + yr);
                i1 = RV::at(2 * c + 1, plb * C::RY + yr);
            } else {
                i0 = CV::at(y, plb * C::CX + 2 * c);
                i1 = CV::at(y, plb * C::CX + 2 * c + 1);
            }
        } else {
            gi = (size_t)unit * NP + (size_t)y * NX + x0 + c;
            if constexpr (ROWS) {
                i0 = RV::at(c, yr);
                i1 = RV::at(c, C::RY + yr);
            } else {
                i0 = CV::at(y, c);
                i1 = CV::at(y, C::CX + c);
            }
        }
        if constexpr (STORE) {
            const float2 e0 = s[i0], e1 = s[i1];
            reinterpret_cast<float4*>(gout)[gi] = make_float4(e0.x, e0.y, e1.x, e1.y);
        } else {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(gin) + gi);
            s[i0] = make_float2(v.x, v.y);
            s[i1] = make_float2(v.z, v.w);
        }
    }
}

// NTHR threads per CTA; 512 / NTHR CTAs per SM (the register file holds 512 threads at
// 128 registers).  The linear step factorises, IFFT_xy Rx Ry D FFT_xy =
// (IFFT_x Rx FFT_x)(IFFT_y Ry D FFT_y), so a unit is loaded by columns, takes its y part in
// the column view, moves to the row view in one cluster exchange, takes its x part and is
// stored by rows.  With the mirror lens: y(t1), exchange, x(t1), lens, x(t2), exchange,
// y(t2), stored by columns.
template <int NX, int NY, int CL, int PB, int SLO, int NTHR>
__global__ void __launch_bounds__(NTHR, (NTHR >= 512 ? 1 : 512 / NTHR)) plane_kernel(PlaneArgs a) {
    using C = PlaneCfg<NX, NY, CL, PB, SLO>;
    using RV = RowView<NX, NY, CL, PB, SLO>;
    using CV = ColView<NX, NY, CL, PB, SLO>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    unsigned char* twx_mem = smem_raw + C::SIZE * 8;
    unsigned char* twy_mem = twx_mem + twiddle_bytes(NX);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x;
    const int cid = blockIdx.x / CL, ncl = gridDim.x / CL;
    const int NP = a.NP;
    stage_twiddles<NX, NTHR>(twx_mem, a.twx, tid);
    stage_twiddles<NY, NTHR>(twy_mem, a.twy, tid);
    const Twiddles twx = Twiddles::packed(twx_mem, NX), twy = Twiddles::packed(twy_mem, NY);
    pdl_wait();
    __syncthreads();

    for (int unit = cid; unit < a.nunits; unit += ncl) {
        if (unit + ncl >= a.nunits) pdl_launch_next();
        plane_move<NX, NY, CL, PB, SLO, NTHR, false, false>(s, a.in, nullptr, rank, unit, NP, tid);
        __syncthreads();
        dif_op_dit<NY, NY, CV, NTHR, 1>(s, twy, tid, YFactors<C::CX, SLO, PB>{a.t1.RyD, a.Nt, unit});
        cluster_exchange<CL, C::RSZ, NTHR>(s, cluster, rank, tid);
        dif_op_dit<NX, NX, RV, NTHR, 1>(s, twx, tid, XFactors{a.t1.Rx});
        if (a.lens) {
            // mirror lens in real (x, y): exp(-i k0 (x^2 + y^2)/roc) = lensx[x] * lensy[y]
            for (int e = tid; e < PB * C::RY * NX; e += NTHR) {
                const int x = e % NX;
                const int l = e / NX;
                const int yl = l % C::RY;
                const int y = rank * C::RY + yl;
                const int idx = RV::at(x, l);
                s[idx] = cmul(s[idx], cmul(__ldg(&a.lensx[x]), __ldg(&a.lensy[y])));
            }
            __syncthreads();
            dif_op_dit<NX, NX, RV, NTHR, 1>(s, twx, tid, XFactors{a.t2.Rx});
            cluster_exchange<CL, C::RSZ, NTHR>(s, cluster, rank, tid);
            dif_op_dit<NY, NY, CV, NTHR, 1>(s, twy, tid, YFactors<C::CX, SLO, PB>{a.t2.RyD, a.Nt, unit});
            plane_move<NX, NY, CL, PB, SLO, NTHR, false, true>(s, nullptr, a.out, rank, unit, NP, tid);
        } else {
            plane_move<NX, NY, CL, PB, SLO, NTHR, true, true>(s, nullptr, a.out, rank, unit, NP, tid);
        }
        __syncthreads();
    }
    cluster.sync();
}

// ---------------------------------------------------------------------------------------
// Plane pass in two passes over HBM (no clusters), for planes that a cluster of 2-CTA-per-SM
// blocks cannot hold: the linear step's y part on column strips, then its x part on row strips
// (IFFT_xy Rx Ry D FFT_xy = (IFFT_x Rx FFT_x)(IFFT_y Ry D FFT_y)).  Slot layout SLO = 1.  Each
// CTA reads and writes only its own strip, so both passes run in place.
// ---------------------------------------------------------------------------------------
// strip of CXS columns of one omega-plane: line = column, position = y
template <int NY, int CXS>
struct StripYView {
    static constexpr int NLINES = CXS;
    static constexpr __host__ __device__ __forceinline__ int at(int y, int l) { return y * CXS + l; }
};
// strip of RYS rows: line = row, position = x, rows padded by one element (bank spread)
template <int NX, int RYS>
struct StripXView {
    static constexpr int NLINES = RYS;
    static constexpr __host__ __device__ __forceinline__ int at(int x, int l) { return l * (NX + 1) + x; }
};

template <int NX, int NY, int CXS>
struct StripYCfg {
    static constexpr int SIZE = NY * CXS;
    // [strip][the slot's NY factors Ry(y) D(slot), 16 B each][W_NY twiddles]
    static constexpr int SMEM = SIZE * 8 + NY * 16 + twiddle_bytes(NY);
    // at least 16 columns: the rows of a warp's butterfly loads then fill all 32 banks
    static_assert(CXS >= 16 && CXS % 2 == 0 && NX % CXS == 0, "whole float4 column strips");
};
template <int NX, int NY, int RYS>
struct StripXCfg {
    static constexpr int SIZE = RYS * (NX + 1);
    // rows of up to 256 points: the x factors of both tables staged in shared memory once per CTA
    static constexpr bool XSTAGE = NX <= 256;
    static constexpr int SMEM = ((SIZE * 8 + 15) / 16) * 16 + (XSTAGE ? 2 * NX * 16 : 0) + twiddle_bytes(NX);
    static_assert(NY % RYS == 0 && NX % 2 == 0, "whole row strips");
};


// Ry(y) D(slot) of the unit's slot from shared memory (staged once per unit)
struct YSmemFactors {
    const float4* f;   // NY factors of the unit's slot, shared memory
    template <int R>
    __device__ __forceinline__ void operator()(float2 (&v)[R], int y0, int) const {
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = cmul_df(v[q], f[y0 + q]);
    }
};

// Resident CTAs per SM a strip kernel is compiled for: MINB, or 512 / NTHR (128 registers).
__host__ __device__ constexpr int strip_min_blocks(int NTHR, int MINB) {
    return MINB > 0 ? MINB : (NTHR >= 512 ? 1 : 512 / NTHR);
}

// y part: units are (slot, strip of CXS columns); `second` selects the table set t2.
template <int NX, int NY, int CXS, int NTHR, int MINB = 0>
__global__ void __launch_bounds__(NTHR, strip_min_blocks(NTHR, MINB)) plane_y_kernel(PlaneArgs a, int second) {
    using C = StripYCfg<NX, NY, CXS>;
    using V = StripYView<NY, CXS>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    float4* fac = reinterpret_cast<float4*>(smem_raw + C::SIZE * 8);
    unsigned char* tw_mem = smem_raw + C::SIZE * 8 + NY * 16;
    const int tid = threadIdx.x;
    stage_twiddles<NY, NTHR>(tw_mem, a.twy, tid);
    const Twiddles tw = Twiddles::packed(tw_mem, NY);
    pdl_wait();
    __syncthreads();
    const float4* RyDT = second ? a.t2.RyDT : a.t1.RyDT;
    constexpr int STRIPS = NX / CXS;
    constexpr int F4_ROW = CXS / 2;
    const int units = a.Nt * STRIPS;
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        if (unit + (int)gridDim.x >= units) pdl_launch_next();
        const int slot = unit / STRIPS, x0 = (unit - slot * STRIPS) * CXS;
        const float4* g4 = reinterpret_cast<const float4*>(a.in) + ((size_t)slot * a.NP + x0) / 2;
        // the slot's factors, shared by the strip's CXS columns
        for (int y = tid; y < NY; y += NTHR) fac[y] = __ldg(&RyDT[(size_t)slot * NY + y]);
#pragma unroll 8
        for (int f = tid; f < NY * F4_ROW; f += NTHR) {
            const int y = f / F4_ROW, c = f - y * F4_ROW;
            reinterpret_cast<float4*>(s)[(y * CXS) / 2 + c] = __ldcg(&g4[(size_t)y * (NX / 2) + c]);
        }
        __syncthreads();
        dif_op_dit<NY, NY, V, NTHR, 1>(s, tw, tid, YSmemFactors{fac});
        float4* o4 = reinterpret_cast<float4*>(a.out) + ((size_t)slot * a.NP + x0) / 2;
#pragma unroll 8
        for (int f = tid; f < NY * F4_ROW; f += NTHR) {
            const int y = f / F4_ROW, c = f - y * F4_ROW;
            o4[(size_t)y * (NX / 2) + c] = reinterpret_cast<const float4*>(s)[(y * CXS) / 2 + c];
        }
        __syncthreads();
    }
}

// y part with TMA staging: a persistent CTA walks its units (slot, strip of CXS columns) with
// NBUF unit buffers in shared memory; warp 0 keeps NBUF - 1 units in flight as 2-D bulk tensor
// loads (box: CXS complex columns x NY rows of one omega-plane, landing in the StripYView layout)
// plus a bulk copy of the slot's NY factors Ry(y) D(slot) (the slot-major table, 16 B each) on
// the same mbarrier, and each finished unit leaves by a bulk tensor store, so no thread spends
// instructions or registers on moving the strips and every factor is read from shared memory
// (all CXS columns of a row share it).  tin / tout map the field as (2 Nx floats, rows of a block, blocks
// of a plane, slots).  A load that does not arrive within the wait limit sets *err and ends the kernel.
// Bound: HBM and the shared-memory pipe (256x256x2048 0.37 ms, 5.8 TB/s).  All 16 columns of a warp's
// rows share a twiddle, so the table is kept as float4 and an inverse stage takes one load per factor
// (plane sweep 0.710 -> 0.695 ms; 512x512x1024 1.794 -> 1.779, 256x256x512 0.188 -> 0.184).  Columns of
// 128 leave from the registers (128-byte row pieces, one barrier and one crossing of shared memory fewer:
// 128x128x1024 plane sweep 0.107 -> 0.102 ms); longer ones by a bulk store (0.695 against 0.726 ms at
// 256x256x2048, 1.779 against 1.884 at 512x512x1024, whose rows lie further apart).
template <int NX, int NY, int CXS>
struct StripYTmaCfg {
    static constexpr int UNIT_BYTES = NY * CXS * 8;
    static constexpr int FAC_BYTES = NY * 16;   // one slot's Ry(y) D(slot) factors, double-float
    static_assert(UNIT_BYTES % 128 == 0 && CXS * 8 % 16 == 0, "unit buffers of whole 128 B lines");
    static constexpr __host__ __device__ int FAC_OFF(int nbuf) { return nbuf * UNIT_BYTES; }
    static constexpr __host__ __device__ int TW_OFF(int nbuf) { return FAC_OFF(nbuf) + nbuf * FAC_BYTES; }
    static constexpr __host__ __device__ int BAR_OFF(int nbuf) { return TW_OFF(nbuf) + NY * 16; }
    static constexpr __host__ __device__ int SMEM(int nbuf) { return 128 + BAR_OFF(nbuf) + nbuf * 8 + 16; }
};

// The last stage's results of a column: position i0 + S q straight to row i0 + S q of its plane (g: the
// strip's first element)
template <int NX>
struct YColumnSink {
    static constexpr bool active = true;
    float2* g;
    template <int R>
    __device__ __forceinline__ void operator()(float2 (&v)[R], int i0, int S, int line) const {
#pragma unroll
        for (int q = 0; q < R; q++) g[(i0 + q * S) * NX + line] = v[q];
    }
};

template <int NX, int NY, int CXS, int NTHR, int NBUF>
__global__ void __launch_bounds__(NTHR, 512 / NTHR)
    plane_y_tma_kernel(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tout, PlaneArgs a,
                       int second, unsigned int* err) {
    using C = StripYTmaCfg<NX, NY, CXS>;
    using V = StripYView<NY, CXS>;
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    // unit buffers on a 128-byte boundary of the shared window (the launch adds 128 B of slack)
    unsigned char* smem_raw = smem_dyn + ((128u - (smem_addr(smem_dyn) & 127u)) & 127u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::BAR_OFF(NBUF));
    int& s_arrived = *reinterpret_cast<int*>(bars + NBUF);
    const int tid = threadIdx.x;
    constexpr int STRIPS = NX / CXS;
    constexpr bool DIRECT = NY <= 128;   // results straight from the registers (the planes are whole)
    const int units = a.Nt * STRIPS;
    const int nmine = blockIdx.x < units ? (units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (tid == 0) {
        for (int b = 0; b < NBUF; b++) mbar_init(&bars[b], 1);
        fence_mbar_init();
    }
    const Tw4 tw{reinterpret_cast<const float4*>(smem_raw + C::TW_OFF(NBUF))};
    stage_twiddles4<NY, NTHR>(reinterpret_cast<float4*>(smem_raw + C::TW_OFF(NBUF)), a.twy, tid);
    const float4* RyDT = second ? a.t2.RyDT : a.t1.RyDT;
    pdl_wait();
    __syncthreads();
    auto buf = [&](int k) { return reinterpret_cast<float2*>(smem_raw + (k % NBUF) * C::UNIT_BYTES); };
    auto fac = [&](int k) {
        return reinterpret_cast<float4*>(smem_raw + C::FAC_OFF(NBUF) + (k % NBUF) * C::FAC_BYTES);
    };
    const int warp = tid >> 5, lane = tid & 31;
    // the copies of a unit are issued by warp 0: lane 0 arms the mbarrier with the unit's bytes and
    // loads the strip, lane 1 the slot's factors
    auto issue = [&](int k) {
        const int unit = (int)blockIdx.x + k * (int)gridDim.x;
        const int slot = unit / STRIPS, x0 = (unit - slot * STRIPS) * CXS;
        if (lane == 0) mbar_arrive_expect_tx(&bars[k % NBUF], C::UNIT_BYTES + C::FAC_BYTES);
        __syncwarp();
        if (lane == 0) tma_load_4d(buf(k), &tin, 2 * x0, 0, 0, slot, &bars[k % NBUF]);
        if (lane == 1) bulk_load(fac(k), RyDT + (size_t)slot * NY, C::FAC_BYTES, &bars[k % NBUF]);
    };
    if (warp == 0)
        for (int k = 0; k < NBUF - 1 && k < nmine; k++) issue(k);
    for (int k = 0; k < nmine; k++) {
        if (k + 1 == nmine) pdl_launch_next();
        const int unit = (int)blockIdx.x + k * (int)gridDim.x;
        const int slot = unit / STRIPS, x0 = (unit - slot * STRIPS) * CXS;
        // one thread decides whether the unit arrived in time, so that the whole CTA takes the
        // same branch; then every thread observes the completed phase itself
        if (tid == 0) s_arrived = mbar_wait(&bars[k % NBUF], (uint32_t)((k / NBUF) & 1)) ? 1 : 0;
        __syncthreads();
        if (!s_arrived) {
            if (tid == 0) {
                atomicExch(err, KERR_TMA_TIMEOUT);
                // the late unit and the ones after it are still on their way into this CTA's shared memory: wait
                // (bounded) for them
                for (int j = k; j < k + NBUF - 1 && j < nmine; j++) mbar_wait(&bars[j % NBUF], (uint32_t)((j / NBUF) & 1));
                bulk_wait<0>();
            }
            return;
        }
        mbar_wait(&bars[k % NBUF], (uint32_t)((k / NBUF) & 1));   // completed: returns at once
        float2* s = buf(k);
        if constexpr (DIRECT) {
            // every thread has left unit k - 1 and fenced its accesses to that buffer
            if (warp == 0 && k + NBUF - 1 < nmine) issue(k + NBUF - 1);
            dif_op_dit<NY, NY, V, NTHR, 1, YSmemFactors, false>(s, tw, tid, YSmemFactors{fac(k)},
                                                                YColumnSink<NX>{a.out + (size_t)slot * a.NP + x0});
            fence_proxy_async_smem();   // this thread's accesses to the buffer, before a bulk load refills it
            continue;
        }
        dif_op_dit<NY, NY, V, NTHR, 1, YSmemFactors, false>(s, tw, tid, YSmemFactors{fac(k)});
        fence_proxy_async_smem();   // this thread's results, before the bulk store reads them
        __syncthreads();
        if (warp == 0) {
            if (lane == 0) {
                tma_store_4d(&tout, 2 * x0, 0, 0, slot, s);
                bulk_commit();
            }
            if (k + NBUF - 1 < nmine) {
                if (lane == 0) bulk_wait_read<1>();   // the previous unit's store has left its buffer
                issue(k + NBUF - 1);
            }
        }
    }
    if (tid == 0) bulk_wait<0>();
}

// ---- TMA-staged y pass for columns of 512 = 16 x 16 x 2 points ---------------------------------------
// As the 256-point pass, with the 32-point transforms between the outer radix-16 stages in registers:
// two lanes hold a 32-point transform (j = 0, 1 of its radix-16 stage) and do its radix-2 stages by
// shuffles, so that a unit crosses shared memory three times (outer, inner, outer) like a 256-point one.
// The operations and their order are those of dif_op_dit.  Bound: issue (54 %) and the shared-memory
// pipe; 512x512x1024 0.96 ms, 4.5 TB/s, against 1.43 ms with plain strip loads (plane_y_kernel).

// the inner part on the 16 positions pos0 + 2 q of one line, pos0 = 32 b + jj (jj = 0, 1 in lanes that
// differ in bit XOR): radix 16, radix 2, the factors f(pos), radix 2, radix 16
template <int XOR, class TW, class FAC>
__device__ __forceinline__ void inner32(float2 (&v)[16], TW tw, int jj, const FAC& fac) {
    const int t0 = tw_stage_offset(512, 32) + jj;
    const float sg = jj ? -1.0f : 1.0f;
    dft<16, false>(v);
#pragma unroll
    for (int k = 1; k < 16; k++) v[k] = tw_mul(tw, t0 + (k - 1) * 2, v[k]);
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const float2 o = make_float2(__shfl_xor_sync(~0u, v[q].x, XOR), __shfl_xor_sync(~0u, v[q].y, XOR));
        const float2 z = cmul_df(make_float2(fmaf(sg, v[q].x, o.x), fmaf(sg, v[q].y, o.y)), fac(2 * q));
        const float2 y = make_float2(__shfl_xor_sync(~0u, z.x, XOR), __shfl_xor_sync(~0u, z.y, XOR));
        v[q] = make_float2(fmaf(sg, z.x, y.x), fmaf(sg, z.y, y.y));
    }
#pragma unroll
    for (int k = 1; k < 16; k++) v[k] = tw_mulc(tw, t0 + (k - 1) * 2, v[k]);
    dft<16, true>(v);
}

// y part: units of (slot, 16 columns) of 64 KB, one 512-thread CTA per SM with three unit buffers
struct StripY512 {
    static constexpr int NY = 512, CXS = 16, NBUF = 3, NTHR = 512;
    static constexpr int UNIT_BYTES = NY * CXS * 8, FAC_BYTES = NY * 16;
    static constexpr int FAC_OFF = NBUF * UNIT_BYTES, TW_OFF = FAC_OFF + NBUF * FAC_BYTES, BAR_OFF = TW_OFF + NY * 16;
    static constexpr int SMEM = 128 + BAR_OFF + NBUF * 8 + 16;
};
template <int NX>
__global__ void __launch_bounds__(StripY512::NTHR, 1)
    plane_y512_tma_kernel(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tout, PlaneArgs a,
                          int second, unsigned int* err) {
    using C = StripY512;
    constexpr int NY = C::NY, CXS = C::CXS, NBUF = C::NBUF, STRIPS = NX / CXS;
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    unsigned char* smem_raw = smem_dyn + ((128u - (smem_addr(smem_dyn) & 127u)) & 127u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::BAR_OFF);
    int& s_arrived = *reinterpret_cast<int*>(bars + NBUF);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int units = a.Nt * STRIPS;
    const int nmine = blockIdx.x < units ? (units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (tid == 0) {
        for (int b = 0; b < NBUF; b++) mbar_init(&bars[b], 1);
        fence_mbar_init();
    }
    const Tw4 tw{reinterpret_cast<const float4*>(smem_raw + C::TW_OFF)};
    stage_twiddles4<NY, C::NTHR>(reinterpret_cast<float4*>(smem_raw + C::TW_OFF), a.twy, tid);
    const float4* RyDT = second ? a.t2.RyDT : a.t1.RyDT;
    pdl_wait();
    __syncthreads();
    auto buf = [&](int k) { return reinterpret_cast<float2*>(smem_raw + (k % NBUF) * C::UNIT_BYTES); };
    auto fac = [&](int k) { return reinterpret_cast<float4*>(smem_raw + C::FAC_OFF + (k % NBUF) * C::FAC_BYTES); };
    // a unit is one box (lane 0) and the slot's factors (lane 1)
    auto issue = [&](int k) {
        const int unit = (int)blockIdx.x + k * (int)gridDim.x;
        const int slot = unit / STRIPS, x0 = (unit - slot * STRIPS) * CXS;
        if (lane == 0) mbar_arrive_expect_tx(&bars[k % NBUF], C::UNIT_BYTES + C::FAC_BYTES);
        __syncwarp();
        if (lane == 0) tma_load_4d(buf(k), &tin, 2 * x0, 0, 0, slot, &bars[k % NBUF]);
        if (lane == 1) bulk_load(fac(k), RyDT + (size_t)slot * NY, C::FAC_BYTES, &bars[k % NBUF]);
    };
    if (warp == 0)
        for (int k = 0; k < NBUF - 1 && k < nmine; k++) issue(k);
    const int line = tid & 15, j = tid >> 4;     // outer stages: y = j + 32 q
    const int jj = (tid >> 4) & 1, b = tid >> 5; // inner part: y = 32 b + jj + 2 q
    for (int k = 0; k < nmine; k++) {
        if (k + 1 == nmine) pdl_launch_next();
        if (tid == 0) s_arrived = mbar_wait(&bars[k % NBUF], (uint32_t)((k / NBUF) & 1)) ? 1 : 0;
        __syncthreads();
        if (!s_arrived) {
            if (tid == 0) {
                atomicExch(err, KERR_TMA_TIMEOUT);
                // the late unit and the ones after it, as in plane_y_tma_kernel
                for (int i = k; i < k + NBUF - 1 && i < nmine; i++) mbar_wait(&bars[i % NBUF], (uint32_t)((i / NBUF) & 1));
                bulk_wait<0>();
            }
            return;
        }
        mbar_wait(&bars[k % NBUF], (uint32_t)((k / NBUF) & 1));   // completed: returns at once
        float2* s = buf(k);
        float2 v[16];
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = s[(j + 32 * q) * CXS + line];
        dft<16, false>(v);
#pragma unroll
        for (int i = 1; i < 16; i++) v[i] = tw_mul(tw, j + (i - 1) * 32, v[i]);
#pragma unroll
        for (int q = 0; q < 16; q++) s[(j + 32 * q) * CXS + line] = v[q];
        __syncthreads();
        const float4* f = fac(k) + 32 * b + jj;
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = s[(32 * b + jj + 2 * q) * CXS + line];
        inner32<16>(v, tw, jj, [&](int i) { return f[i]; });
#pragma unroll
        for (int q = 0; q < 16; q++) s[(32 * b + jj + 2 * q) * CXS + line] = v[q];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = s[(j + 32 * q) * CXS + line];
#pragma unroll
        for (int i = 1; i < 16; i++) v[i] = tw_mulc(tw, j + (i - 1) * 32, v[i]);
        dft<16, true>(v);
#pragma unroll
        for (int q = 0; q < 16; q++) s[(j + 32 * q) * CXS + line] = v[q];
        fence_proxy_async_smem();   // this thread's results, before the bulk stores read them
        __syncthreads();
        if (warp == 0) {
            if (lane == 0) {
                const int unit = (int)blockIdx.x + k * (int)gridDim.x;
                const int slot = unit / STRIPS, x0 = (unit - slot * STRIPS) * CXS;
                tma_store_4d(&tout, 2 * x0, 0, 0, slot, s);
                bulk_commit();
            }
            if (k + NBUF - 1 < nmine) {
                if (lane == 0) bulk_wait_read<1>();   // the previous unit's store has left its buffer
                issue(k + NBUF - 1);
            }
        }
    }
    if (tid == 0) bulk_wait<0>();
}

// ---- x part, a warp per unit -------------------------------------------------------------------------
// Rows are contiguous, so 512 complex (4 KB: one row of 512, two of 256, four of 128) are a unit that one
// warp transforms alone, 16 points per lane: outer radix-16 stage, exchange through the warp's buffer,
// inner part (radix 16, 8, or 16 x 2 by shuffles, with the factors), exchange, outer stage.  Only warp
// barriers; each warp streams its own units, bulk copies in and out, NBUF buffers deep.  A row lands at
// its natural positions; the exchange uses padded positions idx(p) of the same buffer, which are free of
// bank conflicts in both orders.  Bound: HBM, and the shared-memory pipe (94 % busy with the outer
// stages' twiddles in shared memory): a lane keeps those in registers, and 12 warps of 168 registers beat
// 16 of 128 (plane sweep 256x256x2048 0.695 -> 0.689 ms, 512x512x1024 1.779 -> 1.712, 256x256x512 0.184 ->
// 0.179, 128x128x1024 0.107 -> 0.100).  Buffers per warp, 3 against 4: 0.689 against 0.710 ms at rows of
// 256, 1.721 against 1.712 at rows of 512; 2 against 3 at rows of 128: 0.111 against 0.100.  Storing from
// the registers instead of by bulk copies: 0.704 against 0.695 and 1.801 against 1.779, not kept.
// x part alone at 512x512x1024: 0.76 ms (1.45 with plain strips in 256-thread CTAs, 1.17 with TMA boxes
// and CTA barriers).
template <int NX_>
struct XWarp {
    static constexpr int NX = NX_, M = NX / 16, ROWS = 512 / NX;
    static constexpr int PSH = NX == 512 ? 5 : NX == 256 ? 4 : 3, PAD = NX == 512 ? 2 : 1;
    static constexpr int RS = NX == 512 ? 544 : NX == 256 ? 272 : 152;   // row stride in the buffer (128: 8 mod 16)
    static constexpr int BUF = ROWS * RS * 8;
    static constexpr __host__ __device__ __forceinline__ int idx(int p) { return p + (p >> PSH) * PAD; }
    static constexpr int NFAC = idx(NX - 1) + 1;    // factors in the padded order
    static constexpr __host__ __device__ int TW_OFF(int nw, int nbuf) { return nw * nbuf * BUF + ((NFAC * 16 + 15) / 16) * 16; }
    static constexpr __host__ __device__ int BAR_OFF(int nw, int nbuf) { return TW_OFF(nw, nbuf) + ((twiddle_bytes(NX) + 15) / 16) * 16; }
    static constexpr __host__ __device__ int SMEM(int nw, int nbuf) { return BAR_OFF(nw, nbuf) + nw * nbuf * 8; }
    static_assert(NX == 128 || NX == 256 || NX == 512, "rows that fill a unit");
    static_assert(idx(NX - 1) < RS && RS * 8 % 16 == 0, "padded rows fit, bulk copies are 16-byte aligned");
};

// The outer stages' twiddles of lane j, held in registers: they are the same for every unit
template <int M>
struct XOuter {
    float2 w[15];
    float e[15];
    __device__ __forceinline__ XOuter(Twiddles tw, int j) {
#pragma unroll
        for (int k = 0; k < 15; k++) {
            w[k] = tw.w[j + k * M];
            e[k] = tw.e[j + k * M];
        }
    }
};

// IFFT_x Rx FFT_x of a warp's unit: v holds x = j + M q of row r (lane = r M + j); rx(p, i) the factor at
// position p + i of a block that starts at p.  buf: the warp's buffer, which every lane has finished reading when `v` was loaded.
template <class C, class FAC>
__device__ __forceinline__ void xwarp_linear(float2 (&v)[16], float2* buf, Twiddles tw, const XOuter<C::M>& ot, const FAC& rx, int lane) {
    constexpr int M = C::M;
    const int j = lane % M, r = lane / M;
    float2* row = buf + r * C::RS;
    dft<16, false>(v);
#pragma unroll
    for (int k = 1; k < 16; k++) v[k] = cmul(v[k], ot.w[k - 1]);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 16; q++) row[j + C::idx(M * q)] = v[q];   // j < M <= 2^PSH: idx(j + M q)
    __syncwarp();
    if constexpr (C::NX == 512) {
        const int jj = lane & 1, p = 32 * (lane >> 1);
        float2* e = buf + C::idx(p) + jj;
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = e[2 * q];
        inner32<1>(v, tw, jj, [&](int i) { return rx(p, jj + i); });
#pragma unroll
        for (int q = 0; q < 16; q++) e[2 * q] = v[q];
    } else if constexpr (C::NX == 256) {
        float2* e = row + C::idx(16 * j);   // block j of row r
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = e[q];
        dft<16, false>(v);
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = cmul_df(v[q], rx(16 * j, q));
        dft<16, true>(v);
#pragma unroll
        for (int q = 0; q < 16; q++) e[q] = v[q];
    } else {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int p = 8 * (j + 8 * h);   // blocks j and j + 8 of row r
            float2* e = row + C::idx(p);
            float2 u[8];
#pragma unroll
            for (int q = 0; q < 8; q++) u[q] = e[q];
            dft<8, false>(u);
#pragma unroll
            for (int q = 0; q < 8; q++) u[q] = cmul_df(u[q], rx(p, q));
            dft<8, true>(u);
#pragma unroll
            for (int q = 0; q < 8; q++) e[q] = u[q];
        }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = row[j + C::idx(M * q)];
#pragma unroll
    for (int k = 1; k < 16; k++) {
        const float2 u = cmulc(v[k], ot.w[k - 1]);
        v[k] = make_float2(fmaf(u.x, ot.e[k - 1], u.x), fmaf(u.y, ot.e[k - 1], u.y));
    }
    dft<16, true>(v);
}

template <int NX, int YB, int NW, int NBUF>
__global__ void __launch_bounds__(NW * 32, 1) plane_x_warp_kernel(PlaneArgs a, unsigned int* err) {
    using C = XWarp<NX>;
    extern __shared__ __align__(16) unsigned char smem_raw[];   // bulk copies: 16-byte boundaries
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float4* rx1 = reinterpret_cast<float4*>(smem_raw + NW * NBUF * C::BUF);
    unsigned char* tw_mem = smem_raw + C::TW_OFF(NW, NBUF);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::BAR_OFF(NW, NBUF)) + warp * NBUF;
    unsigned char* bufs = smem_raw + warp * NBUF * C::BUF;
    const long units = (long)a.Nt * a.NP / 512, first = (long)blockIdx.x * NW + warp, stride = (long)gridDim.x * NW;
    const int nmine = first < units ? (int)((units - 1 - first) / stride) + 1 : 0;
    if (lane == 0) {
        for (int b = 0; b < NBUF; b++) mbar_init(&bars[b], 1);
        fence_mbar_init();
    }
    stage_twiddles<NX, NW * 32>(tw_mem, a.twx, tid);
    const Twiddles tw = Twiddles::packed(tw_mem, NX);
    pdl_wait();
    for (int i = tid; i < NX; i += NW * 32) rx1[C::idx(i)] = __ldg(&a.t1.Rx[i]);
    __syncthreads();
    auto buf = [&](int k) { return reinterpret_cast<float2*>(bufs + (k % NBUF) * C::BUF); };
    auto issue = [&](int k) {   // one bulk copy per row, by the first lanes
        if (lane == 0) mbar_arrive_expect_tx(&bars[k % NBUF], 4096);
        __syncwarp();
        if (lane < C::ROWS)
            bulk_load(buf(k) + lane * C::RS, a.in + (first + k * stride) * 512 + lane * NX, NX * 8, &bars[k % NBUF]);
    };
    for (int k = 0; k < NBUF - 1 && k < nmine; k++) issue(k);
    const int j = lane % C::M, r = lane / C::M;
    const XOuter<C::M> ot(tw, j);
    for (int k = 0; k < nmine; k++) {
        if (k + 1 == nmine) pdl_launch_next();
        if (!__all_sync(~0u, mbar_wait(&bars[k % NBUF], (uint32_t)((k / NBUF) & 1)))) {
            if (lane == 0) {
                atomicExch(err, KERR_TMA_TIMEOUT);
                // the late unit and the ones after it, as in plane_y_tma_kernel
                for (int i = k; i < k + NBUF - 1 && i < nmine; i++) mbar_wait(&bars[i % NBUF], (uint32_t)((i / NBUF) & 1));
            }
            if (lane < C::ROWS) bulk_wait<0>();   // each lane's own stores
            return;
        }
        float2* s = buf(k);
        float2* row = s + r * C::RS;
        float2 v[16];
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = row[j + C::M * q];
        xwarp_linear<C>(v, s, tw, ot, [&](int p, int i) { return rx1[C::idx(p) + i]; }, lane);
        if (a.lens) {   // mirror lens in real (x, y): exp(-i k0 (x^2 + y^2)/roc) = lensx[x] * lensy[y]
            const long g = (first + k * stride) * C::ROWS + r;   // row in memory order: (block, slot, row of the block)
            const float2 ly = __ldg(&a.lensy[(int)(g / ((long)a.Nt * YB)) * YB + (int)(g % YB)]);
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = cmul(v[q], cmul(__ldg(&a.lensx[j + C::M * q]), ly));
            xwarp_linear<C>(v, s, tw, ot, [&](int p, int i) { return __ldg(&a.t2.Rx[p + i]); }, lane);
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 16; q++) row[j + C::M * q] = v[q];
        fence_proxy_async_smem();   // this lane's results, before the bulk stores read them
        __syncwarp();
        if (lane < C::ROWS) {
            bulk_store(a.out + (first + k * stride) * 512 + lane * NX, s + lane * C::RS, NX * 8);
            bulk_commit();
        }
        if (k + NBUF - 1 < nmine) {
            if (lane < C::ROWS) bulk_wait_read<1>();   // a lane refills the row that its own store read
            issue(k + NBUF - 1);
        }
    }
    if (lane < C::ROWS) bulk_wait<0>();
}

// ---- whole planes in shared memory (64 x 64) ----------------------------------------------------------
// A CTA holds a plane and applies the y part, then the x part, in one pass over HBM.  A warp takes units
// of 512 points (LPU columns, then LPU rows), 16 points per lane: outer radix-16 stage, inner radix-M
// blocks with the factors, outer stage, with warp barriers; between the y and the x part one CTA barrier.
// Each warp stores its finished rows by bulk copies and loads the next plane's into them as soon as they
// have been read, so that copies overlap the other warps' work.  Row y starts at at(y): the row stride
// and the skew leave every access of both parts free of bank conflicts, and a row has room for the x
// part's padded exchange positions idx(p).  Bound: latency (one plane per CTA at 64x64x512, four CTAs per
// SM).  18.2 us a launch at 64x64x512 against 22.6 with two planes per CTA and CTA barriers per stage
// (plane_kernel); 4 warps and 4 CTAs against 8 and 3, 8 and 4, 4 and 3: 18.2, 18.8, 19.1, 18.8 us.  (Planes
// of 128 x 128 the same way, one CTA of 16 warps per SM: 0.119 ms against 0.113 in two passes, not kept.)
struct PlaneS {
    static constexpr int N = 64, M = N / 16, LPU = 512 / N;
    static constexpr int RSTR = 88;
    static constexpr __host__ __device__ __forceinline__ int idx(int p) { return p + (p >> 2); }
    static constexpr __host__ __device__ __forceinline__ int at(int y) { return y * RSTR + 4 * (y >> 1); }
    static constexpr int SIZE = N * RSTR + 4 * ((N - 1) >> 1);        // at(N - 1) + RSTR complex values
    static constexpr int NFAC = N + ((N - 1) >> 2);                   // idx(N - 1) + 1
    // [plane][y factors of two planes][x factors, padded][twiddles][mbarrier, flag]
    static constexpr int FAC_OFF = SIZE * 8, RX_OFF = FAC_OFF + 2 * N * 16, TW_OFF = RX_OFF + NFAC * 16;
    static constexpr int BAR_OFF = TW_OFF + ((twiddle_bytes(N) + 15) / 16) * 16;
    static constexpr int SMEM = BAR_OFF + 16;
    static_assert(SIZE * 8 % 16 == 0 && RSTR * 8 % 16 == 0 && NFAC <= RSTR, "aligned rows with room for the exchange");
};

// inverse after forward transform of one line per lane group with the factors between: v holds the
// natural positions j + M q; pos(q) is the place of exchange position j + M q, blk(b) that of position
// M b of the exchange, whose neighbours are `stride(q)` away; fac(p, i) the factor at position p + i.
template <bool SEPARATE, class POS, class BLK, class STRD, class FAC>
__device__ __forceinline__ void plane_line(float2 (&v)[16], Twiddles tw, int j, const POS& pos, const BLK& blk, const STRD& strd,
                                           const FAC& fac) {
    constexpr int M = PlaneS::M;
    const float2* t = tw.w + j;
    const float* te = tw.e + j;
    dft<16, false>(v);
#pragma unroll
    for (int k = 1; k < 16; k++) v[k] = cmul(v[k], t[(k - 1) * M]);
    if constexpr (SEPARATE) __syncwarp();   // exchange places cover other lanes' natural ones
#pragma unroll
    for (int q = 0; q < 16; q++) *pos(q) = v[q];
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 16 / M; h++) {
        const int b = j + M * h;
        float2* e = blk(b);
        float2 u[M];
#pragma unroll
        for (int q = 0; q < M; q++) u[q] = e[strd(q)];
        dft<M, false>(u);
#pragma unroll
        for (int q = 0; q < M; q++) u[q] = cmul_df(u[q], fac(M * b, q));
        dft<M, true>(u);
#pragma unroll
        for (int q = 0; q < M; q++) e[strd(q)] = u[q];
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = *pos(q);
#pragma unroll
    for (int k = 1; k < 16; k++) {
        const float2 u = cmulc(v[k], t[(k - 1) * M]);
        const float e = te[(k - 1) * M];
        v[k] = make_float2(fmaf(u.x, e, u.x), fmaf(u.y, e, u.y));
    }
    dft<16, true>(v);
}

template <int NW, int MINB>
__global__ void __launch_bounds__(NW * 32, MINB) plane_smem_kernel(PlaneArgs a, unsigned int* err) {
    using C = PlaneS;
    constexpr int N = C::N, M = C::M, LPU = C::LPU, UPW = N / LPU / NW;
    static_assert(UPW * NW * LPU == N, "whole units per warp");
    extern __shared__ __align__(16) unsigned char smem_raw[];   // bulk copies: 16-byte boundaries
    float2* s = reinterpret_cast<float2*>(smem_raw);
    float4* fac = reinterpret_cast<float4*>(smem_raw + C::FAC_OFF);
    float4* rx1 = reinterpret_cast<float4*>(smem_raw + C::RX_OFF);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + C::BAR_OFF);
    int& s_arrived = *reinterpret_cast<int*>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        mbar_init(bar, NW);
        fence_mbar_init();
    }
    stage_twiddles<N, NW * 32>(smem_raw + C::TW_OFF, a.twx, tid);   // Nx = Ny: one table
    const Twiddles tw = Twiddles::packed(smem_raw + C::TW_OFF, N);
    pdl_wait();
    for (int i = tid; i < N; i += NW * 32) rx1[C::idx(i)] = __ldg(&a.t1.Rx[i]);
    __syncthreads();
    // this warp's rows of plane `slot` (and, warp 0, its y factors); the previous plane's stores of these
    // rows have been read
    auto issue = [&](int slot, int k) {
        constexpr int ROWS = UPW * LPU;
        if (lane == 0) mbar_arrive_expect_tx(bar, ROWS * N * 8 + (warp == 0 ? N * 16 : 0));
        __syncwarp();
        if (lane < ROWS) {
            const int y = warp * ROWS + lane;
            bulk_load(s + C::at(y), a.in + ((size_t)slot * N + y) * N, N * 8, bar);
        }
        if (warp == 0 && lane == 31) bulk_load(fac + (k & 1) * N, a.t1.RyDT + (size_t)slot * N, N * 16, bar);
    };
    static_assert(UPW * LPU <= 31, "rows of a warp by one lane each, the factors by another");
    int slot = blockIdx.x;
    if (slot < a.Nt) issue(slot, 0);
    // x part: rows LPU u + r, 4 rows x 4 butterflies to a half-warp; y part: columns LPU u + c
    const int jx = lane & 3, r = lane >> 2;
    const int c = lane & (LPU - 1), jy = lane / LPU;
    auto y_part = [&](const auto& f) {
#pragma unroll 1
        for (int u = 0; u < UPW; u++) {
            float2* col = s + (warp * UPW + u) * LPU + c;
            float2* own = col + C::at(jy);
            float2 v[16];
            auto pos = [&](int q) { return own + (C::at(M * q) - C::at(0)); };
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = *pos(q);
            plane_line<false>(v, tw, jy, pos, [&](int b) { return col + C::at(M * b); }, [](int q) { return C::at(q); }, f);
#pragma unroll
            for (int q = 0; q < 16; q++) *pos(q) = v[q];
        }
    };
    for (int k = 0; slot < a.Nt; k++, slot += gridDim.x) {
        if (slot + (int)gridDim.x >= a.Nt) pdl_launch_next();
        if (tid == 0) s_arrived = mbar_wait(bar, (uint32_t)(k & 1)) ? 1 : 0;
        __syncthreads();
        if (!s_arrived) {
            if (tid == 0) {
                atomicExch(err, KERR_TMA_TIMEOUT);
                mbar_wait(bar, (uint32_t)(k & 1));   // the late plane is still on its way: wait (bounded) once more
            }
            bulk_wait<0>();   // each lane's own stores
            return;
        }
        mbar_wait(bar, (uint32_t)(k & 1));   // completed: returns at once
        const float4* fk = fac + (k & 1) * N;
        y_part([&](int p, int i) { return fk[p + i]; });
        __syncthreads();
#pragma unroll 1
        for (int u = 0; u < UPW; u++) {
            const int y = (warp * UPW + u) * LPU + r;
            float2* row = s + C::at(y);
            float2 v[16];
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = row[jx + M * q];
            auto pos = [&](int q) { return row + jx + C::idx(M * q); };
            auto blk = [&](int b) { return row + C::idx(M * b); };
            auto strd = [](int q) { return q; };
            plane_line<true>(v, tw, jx, pos, blk, strd, [&](int p, int i) { return rx1[C::idx(p) + i]; });
            if (a.lens) {   // mirror lens in real (x, y): exp(-i k0 (x^2 + y^2)/roc) = lensx[x] * lensy[y]
                const float2 ly = __ldg(&a.lensy[y]);
#pragma unroll
                for (int q = 0; q < 16; q++) v[q] = cmul(v[q], cmul(__ldg(&a.lensx[jx + M * q]), ly));
                plane_line<true>(v, tw, jx, pos, blk, strd, [&](int p, int i) { return __ldg(&a.t2.Rx[p + i]); });
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 16; q++) row[jx + M * q] = v[q];
        }
        if (a.lens) {
            __syncthreads();
            const float4* f2 = a.t2.RyDT + (size_t)slot * N;
            y_part([&](int p, int i) { return __ldg(&f2[p + i]); });
            __syncthreads();
        }
        fence_proxy_async_smem();   // this lane's results, before the bulk stores read them
        __syncwarp();
        if (a.lens) __syncthreads();
        const int ROWS = UPW * LPU;
        if (lane < ROWS) {
            const int y = warp * ROWS + lane;
            bulk_store(a.out + ((size_t)slot * N + y) * N, s + C::at(y), N * 8);
            bulk_commit();
        }
        const int next = slot + gridDim.x;
        if (next < a.Nt) {
            if (lane < ROWS) bulk_wait_read<0>();
            issue(next, k + 1);
        }
    }
    bulk_wait<0>();
}

// x part: units are (slot, strip of RYS rows); with the mirror lens, x(t1), the lens, x(t2).
template <int NX, int NY, int RYS, int NTHR, int MINB = 0>
__global__ void __launch_bounds__(NTHR, strip_min_blocks(NTHR, MINB)) plane_x_kernel(PlaneArgs a) {
    using C = StripXCfg<NX, NY, RYS>;
    using V = StripXView<NX, RYS>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    float4* rx_s = reinterpret_cast<float4*>(smem_raw + ((C::SIZE * 8 + 15) / 16) * 16);
    unsigned char* tw_mem = reinterpret_cast<unsigned char*>(rx_s) + (C::XSTAGE ? 2 * NX * 16 : 0);
    const int tid = threadIdx.x;
    stage_twiddles<NX, NTHR>(tw_mem, a.twx, tid);
    const Twiddles tw = Twiddles::packed(tw_mem, NX);
    pdl_wait();
    const float4* rx1 = a.t1.Rx;
    const float4* rx2 = a.t2.Rx;
    if constexpr (C::XSTAGE) {
        for (int i = tid; i < NX; i += NTHR) {
            rx_s[i] = __ldg(&a.t1.Rx[i]);
            rx_s[NX + i] = __ldg(&a.t2.Rx[i]);
        }
        rx1 = rx_s;
        rx2 = rx_s + NX;
    }
    __syncthreads();
    constexpr int STRIPS = NY / RYS;
    constexpr int F4_ROW = NX / 2;
    const int units = a.Nt * STRIPS;
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        if (unit + (int)gridDim.x >= units) pdl_launch_next();
        const int slot = unit / STRIPS, y0 = (unit - slot * STRIPS) * RYS;
        const float4* g4 = reinterpret_cast<const float4*>(a.in) + ((size_t)slot * a.NP + (size_t)y0 * NX) / 2;
#pragma unroll 8
        for (int f = tid; f < RYS * F4_ROW; f += NTHR) {
            const int r = f / F4_ROW, c = f - r * F4_ROW;
            const float4 v = __ldcg(&g4[f]);
            s[V::at(2 * c, r)] = make_float2(v.x, v.y);
            s[V::at(2 * c + 1, r)] = make_float2(v.z, v.w);
        }
        __syncthreads();
        dif_op_dit<NX, NX, V, NTHR, 1>(s, tw, tid, XFactorsAny{rx1});
        if (a.lens) {
            for (int e = tid; e < RYS * NX; e += NTHR) {
                const int x = e % NX, r = e / NX;
                const int idx = V::at(x, r);
                s[idx] = cmul(s[idx], cmul(__ldg(&a.lensx[x]), __ldg(&a.lensy[y0 + r])));
            }
            __syncthreads();
            dif_op_dit<NX, NX, V, NTHR, 1>(s, tw, tid, XFactorsAny{rx2});
        }
        float4* o4 = reinterpret_cast<float4*>(a.out) + ((size_t)slot * a.NP + (size_t)y0 * NX) / 2;
#pragma unroll 8
        for (int f = tid; f < RYS * F4_ROW; f += NTHR) {
            const int r = f / F4_ROW, c = f - r * F4_ROW;
            const float2 e0 = s[V::at(2 * c, r)], e1 = s[V::at(2 * c + 1, r)];
            o4[f] = make_float4(e0.x, e0.y, e1.x, e1.y);
        }
        __syncthreads();
    }
}

}  // namespace mpc
