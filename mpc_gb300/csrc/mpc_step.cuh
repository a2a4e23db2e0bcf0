// mpc_step.cuh -- the split step's pencil sweep in one kernel: IFFT_t of S and of -i omega S, the
// nonlinear step, FFT_t.
//
// A tile is TP = P * Nt points (P neighbouring pencils), 16 points per thread.  The transforms are
// radix 16 (span M = Nt/16) around M-point transforms, and the work is split so that
//   - the M-point transforms (radix LL, then radix 16 where M > 16) stay inside a warp: warp w owns the
//     positions [BW w, BW w + BW) of all P pencils, loads them itself (a TMA box, one tile ahead), and
//     needs warp barriers only;
//   - the outer radix-16 stage of the inverse transforms and of the forward transform act on the same
//     points t = j + M q of one pencil, so a thread keeps its 16 samples A(t) and dA(t) conj(A(t)) in
//     registers from the end of the inverse transforms to the start of the forward one, and the
//     nonlinear step is applied there.  Only what the ionization prefix along t needs goes through
//     shared memory: the rates (b, (1 - b) a + b) of every sample out, the ion fraction back.
// Both inverse transforms run in the same passes: S is read once, the twiddles are loaded once, dA
// never leaves the SM (a tile of A, a tile of dA, in turn the exchange buffer and the next tile's
// spectrum).
//
// Bound: instruction issue and the latencies between the CTA barriers (five per tile), not HBM.  At
// 256x256x2048 (GB300, 2070 MHz) a launch takes 1.10 ms, 1.96 TB/s.  How it came there: the three-pass
// sweep before it (dA through an L2 scratch tile, the ADK terms evaluated twice, the tile read twice)
// 2.03 ms; in this form with cp.async and plain stores 1.39; planes in row blocks (mpc_shapes.cuh YB)
// 1.26; twiddles in one load 1.24; blocks as TMA boxes (a warp-wide access to 32-byte rows takes the
// load/store unit 8 to 16 cycles) 1.10.  512x512x1024: 4.05 -> 2.16 ms, 128x128x1024: 0.274 -> 0.149 ms,
// 64x64x512: 43 -> 27 us.  A prefetch of the next tile into L2 made it slower (1.29 against 1.24).
// The tile's size: mpc_shapes.cuh step_tile.
#pragma once
#include "mpc_kernels.cuh"

namespace mpc {

// ---- arithmetic -----------------------------------------------------------------------------
// The special-function unit on arguments that are normal numbers (no denormal scaling around it)
__device__ __forceinline__ float mufu_lg2(float x) { float r; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float mufu_ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float mufu_rsqrt(float x) { float r; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float mufu_rcp(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
// maximum that keeps a NaN
__device__ __forceinline__ float max_nan(float a, float b) { float r; asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r; }

// Double-float numbers (h + l, about 48 bits): the carries of the ionization prefix across chunks.
// GB300 issues FP64 at 1/64 of its FP32 rate, and every warp takes part in this scan.
struct DF { float h, l; };
__device__ __forceinline__ DF df_renorm(float h, float l) {
    const float s = h + l;
    return DF{s, l - (s - h)};
}
__device__ __forceinline__ DF df_mul(DF a, DF b) {   // two-product by FMA, cross terms to first order
    const float p = a.h * b.h;
    float e = fmaf(a.h, b.h, -p);
    e = fmaf(a.h, b.l, e);
    e = fmaf(a.l, b.h, e);
    return df_renorm(p, e);
}
__device__ __forceinline__ DF df_add(DF a, DF b) {   // two-sum of the high parts
    const float s = a.h + b.h, bb = s - a.h;
    const float e = (a.h - (s - bb)) + (b.h - bb);
    return df_renorm(s, e + (a.l + b.l));
}
// Chunk map R -> D R + C of the ionization prefix (mpc_kernels.cuh MapR), D = 1 - B
struct MapDF { DF D, C; };
__device__ __forceinline__ MapDF df_ident() { return MapDF{DF{1.0f, 0.0f}, DF{0.0f, 0.0f}}; }
__device__ __forceinline__ MapDF df_compose(const MapDF& f, const MapDF& t) {   // f first, then t
    return MapDF{df_mul(t.D, f.D), df_add(df_mul(t.D, f.C), t.C)};
}
__device__ __forceinline__ DF df_apply(const MapDF& m, DF R) { return df_add(df_mul(m.D, R), m.C); }
__device__ __forceinline__ MapDF df_up(const MapDF& m, int off) {
    return MapDF{DF{__shfl_up_sync(~0u, m.D.h, off), __shfl_up_sync(~0u, m.D.l, off)},
                 DF{__shfl_up_sync(~0u, m.C.h, off), __shfl_up_sync(~0u, m.C.l, off)}};
}
__device__ __forceinline__ MapDF df_down(const MapDF& m, int off) {
    return MapDF{DF{__shfl_down_sync(~0u, m.D.h, off), __shfl_down_sync(~0u, m.D.l, off)},
                 DF{__shfl_down_sync(~0u, m.C.h, off), __shfl_down_sync(~0u, m.C.l, off)}};
}
__device__ __forceinline__ float4 df_pack(const MapDF& m) { return make_float4(m.D.h, m.D.l, m.C.h, m.C.l); }
__device__ __forceinline__ MapDF df_unpack(float4 v) { return MapDF{DF{v.x, v.y}, DF{v.z, v.w}}; }

// ---- shape ------------------------------------------------------------------------------------
template <int NT_, int TP_>
struct StepCfg {
    static constexpr int NT = NT_, TP = TP_, P = TP / NT, TH = TP / 16, NW = TH / 32;
    static constexpr int M = NT / 16;               // span of the outer radix-16 stage
    static constexpr bool MID = M > 16;             // a radix-16 stage between it and the span-1 stage
    static constexpr int LL = MID ? M / 16 : M;     // radix of the span-1 stage
    static constexpr int BW = 512 / P;              // positions of a warp's block
    static constexpr int TPP = NT / 16;             // 16-sample chunks per pencil, one per thread
    static constexpr int LPP = P < 32 ? 32 / P : 1; // lanes of a warp that hold one pencil's chunks
    static constexpr int G = TPP / LPP;             // warps (thread groups for P >= 32) across a pencil
    using View = PencilView<NT, P>;
    static constexpr int BUF = View::SIZE * 8;      // bytes of a tile
    static constexpr int SCAN = TH * (int)sizeof(MapUV);
    static constexpr int AGG = G * P * 16;          // chunk-map aggregates
    static constexpr int TW = NT * 16;              // twiddles as (c, s, -eps, 0): one load in the inverse stages
    static constexpr int WPOS = NT * 4;
    static constexpr int NB = BW / LL;              // span-1 butterflies of a pencil in a warp's block
    // [tile][tile][scan maps][aggregates][twiddles][omega of each position][mbarriers, flag], and the
    // slack to a 128-byte boundary
    static constexpr int BARS = 2 * BUF + SCAN + AGG + TW + WPOS;
    static constexpr int SMEM = 128 + BARS + 2 * NW * 8 + 16;
    static_assert(BUF % 128 == 0 && View::at(BW, 0) * 8 % 128 == 0, "TMA boxes land on 128-byte boundaries");
    // diag_kernel: [tile][tile][energy parts][two FP64 profiles][twiddles][mbarriers, flag], and the slack
    static constexpr int DIAG_BARS = 2 * BUF + (TH + 2 * NT) * 8 + TW;
    static constexpr int DIAG_SMEM = 128 + DIAG_BARS + 2 * NW * 8 + 16;
    static_assert(NT % 16 == 0 && P >= 4 && BW >= 4 && BW % LL == 0 && BW % M == 0, "warp blocks of whole sub-transforms");
    static_assert(BUF % 16 == 0 && (SCAN % 16) == 0, "16-byte regions");
};

// ---- tile load --------------------------------------------------------------------------------
// A warp's block of a tile's spectrum into shared memory, asynchronously.  SLO = 1: 16-byte chunks of
// two pencils; SLO = 2: 8-byte elements (two positions of one pencil are adjacent in memory).
// g: the tile's first element, RS its row stride in pencils (mpc_kernels.cuh tile_elem)
// (a Stride<N> where the layout fixes it: the row offsets are then immediates)
template <size_t N>
struct Stride {
    __host__ __device__ constexpr operator size_t() const { return N; }
};
template <class C, int SLO, class STRIDE>
__device__ __forceinline__ void step_load_block(float2* s, const float2* __restrict__ g, STRIDE RS, int warp, int lane) {
    using V = typename C::View;
    if constexpr (SLO == 1) {
        constexpr int CPR = C::P / 2;   // chunks of a row; a warp's 32 lanes take 32 / CPR rows at a time
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int f = u * 32 + lane;
            const int pos = warp * C::BW + f / CPR, c = f % CPR;
            const float2* src = g + ((size_t)pos * RS + 2 * c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(s + V::at(pos, 2 * c))), "l"(src) : "memory");
        }
    } else {
#pragma unroll
        for (int u = 0; u < 16; u++) {
            const int f = u * 32 + lane;
            const int pos = warp * C::BW + 2 * (f / (2 * C::P)) + (f & 1), p = (f >> 1) % C::P;
            const float2* src = g + ((size_t)(pos / SLO) * RS + p) * SLO + pos % SLO;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_addr(s + V::at(pos, p))), "l"(src) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void step_load_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// LL consecutive values of a float table
template <int LL>
__device__ __forceinline__ void load_run(float (&w)[LL], const float* p) {
    if constexpr (LL % 4 == 0) {
#pragma unroll
        for (int i = 0; i < LL / 4; i++) {
            const float4 v = reinterpret_cast<const float4*>(p)[i];
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
    } else {
        const float2 v = *reinterpret_cast<const float2*>(p);
        w[0] = v.x; w[1] = v.y;
    }
}

// ---- the transforms' parts --------------------------------------------------------------------
// conj(w_k) factors of an inverse radix-16 stage on v (with the magnitude correction) and, without
// it, on d (mpc_fft.cuh dit_stage)
template <bool TWO>
__device__ __forceinline__ void inv_twiddle(float2 (&v)[16], float2 (&d)[16], const float4* t, int S) {
#pragma unroll
    for (int k = 1; k < 16; k++) {
        const float4 f = t[(k - 1) * S];
        const float2 w = make_float2(f.x, f.y);
        const float2 u = cmulc(v[k], w);
        v[k] = make_float2(fmaf(u.x, f.z, u.x), fmaf(u.y, f.z, u.y));
        if constexpr (TWO) d[k] = cmulc(d[k], w);
    }
}

// The warp-local inverse M-point transforms of its block: of S in `sa` in place and (SST) of
// -i omega S into `sd`.
// BOXED: the block is as its TMA box left it, element (position BW warp + LL b + q, pencil p) at
// (q NB + b) P + p of the block's first words (a warp then reads consecutive words); it is in registers
// before the results go to the tile view.
template <class C, bool SST, bool BOXED>
__device__ __forceinline__ void step_sub_inverse(float2* sa, float2* sd, const float4* tw, const float* wpos, int warp, int lane) {
    using V = typename C::View;
    constexpr int LL = C::LL;
    float2 in[16];
    if constexpr (BOXED) {
        const float2* box = sa + V::at(warp * C::BW, 0) + lane;
#pragma unroll
        for (int u = 0; u < 16 / LL; u++)
#pragma unroll
            for (int q = 0; q < LL; q++) in[u * LL + q] = box[q * C::NB * C::P + u * 32];
        __syncwarp();
    }
#pragma unroll
    for (int u = 0; u < 16 / LL; u++) {
        const int i = u * 32 + lane;
        const int line = i % C::P, pos = warp * C::BW + (i / C::P) * LL;
        const int o = V::at(pos, line);
        float2 v[LL];
#pragma unroll
        for (int q = 0; q < LL; q++) v[q] = BOXED ? in[u * LL + q] : sa[o + V::at(q, 0)];
        if constexpr (SST) {
            float w[LL];
            load_run<LL>(w, wpos + pos);
            float2 d[LL];
#pragma unroll
            for (int q = 0; q < LL; q++) d[q] = cscale(mul_mi<false>(v[q]), w[q]);
            dft<LL, true>(d);
#pragma unroll
            for (int q = 0; q < LL; q++) sd[o + V::at(q, 0)] = d[q];
        }
        dft<LL, true>(v);
#pragma unroll
        for (int q = 0; q < LL; q++) sa[o + V::at(q, 0)] = v[q];
    }
    if constexpr (C::MID) {
        __syncwarp();
        const int line = lane % C::P, g = lane / C::P;
        const int j = g % LL, pos = warp * C::BW + (g / LL) * C::M + j;
        const int o = V::at(pos, line);
        const float4* t = tw + tw_stage_offset(C::NT, C::M) + j;
        float2 v[16], d[16];
#pragma unroll
        for (int q = 0; q < 16; q++) {
            v[q] = sa[o + V::at(LL * q, 0)];
            if constexpr (SST) d[q] = sd[o + V::at(LL * q, 0)];
        }
        inv_twiddle<SST>(v, d, t, LL);
        dft<16, true>(v);
#pragma unroll
        for (int q = 0; q < 16; q++) sa[o + V::at(LL * q, 0)] = v[q];
        if constexpr (SST) {
            dft<16, true>(d);
#pragma unroll
            for (int q = 0; q < 16; q++) sd[o + V::at(LL * q, 0)] = d[q];
        }
    }
}

// The warp-local forward M-point transforms of its block of `sa`; the results go to global memory (g, RS)
// or, BOXED, into the block's first words in the order of its TMA box.
template <class C, int SLO, bool BOXED, class STRIDE>
__device__ __forceinline__ void step_sub_forward(float2* sa, const float4* tw, float2* __restrict__ g, STRIDE RS, int warp, int lane) {
    using V = typename C::View;
    constexpr int LL = C::LL;
    if constexpr (C::MID) {
        const int line = lane % C::P, gi = lane / C::P;
        const int j = gi % LL, pos = warp * C::BW + (gi / LL) * C::M + j;
        const int o = V::at(pos, line);
        const float4* t = tw + tw_stage_offset(C::NT, C::M) + j;
        float2 v[16];
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = sa[o + V::at(LL * q, 0)];
        dft<16, false>(v);
#pragma unroll
        for (int k = 1; k < 16; k++) v[k] = cmul(v[k], tw_cs(t + (k - 1) * LL));
#pragma unroll
        for (int q = 0; q < 16; q++) sa[o + V::at(LL * q, 0)] = v[q];
        __syncwarp();
    }
    float2 out[16];
#pragma unroll
    for (int u = 0; u < 16 / LL; u++) {
        const int i = u * 32 + lane;
        const int line = i % C::P, pos = warp * C::BW + (i / C::P) * LL;
        const int o = V::at(pos, line);
        float2 v[LL];
#pragma unroll
        for (int q = 0; q < LL; q++) v[q] = sa[o + V::at(q, 0)];
        dft<LL, false>(v);
        if constexpr (BOXED) {
#pragma unroll
            for (int q = 0; q < LL; q++) out[u * LL + q] = v[q];
        } else {
            // pos is a multiple of LL: element (pos + q, line) is a constant offset from (pos, line)
            float2* e = g + (SLO == 1 ? (size_t)pos * RS + line : ((size_t)(pos / SLO) * RS + line) * SLO);
#pragma unroll
            for (int q = 0; q < LL; q++) e[SLO == 1 ? (size_t)q * RS : (size_t)(q / SLO) * RS * SLO + q % SLO] = v[q];
        }
    }
    if constexpr (BOXED) {
        __syncwarp();
        float2* box = sa + V::at(warp * C::BW, 0) + lane;
#pragma unroll
        for (int u = 0; u < 16 / LL; u++)
#pragma unroll
            for (int q = 0; q < LL; q++) box[q * C::NB * C::P + u * 32] = out[u * LL + q];
    }
}

// ---- the nonlinear step in registers ------------------------------------------------------------
// R at the start of this thread's chunk, from the chunk's own map: a scan over the lanes that hold
// the pencil's chunks, then over the G warps (P >= 32: thread groups) of the pencil.
template <class C>
__device__ __forceinline__ float step_scan(MapDF own, float4* agg, int tid) {
    constexpr int P = C::P, LPP = C::LPP, G = C::G;
    const int lane = tid & 31, p = tid % P;
    const int grp = tid / (P * LPP);   // the pencil's group this chunk is in
    MapDF acc = own;
    if constexpr (LPP > 1) {
#pragma unroll
        for (int off = P; off < 32; off <<= 1) {
            const MapDF prev = df_up(acc, off);
            if (lane >= off) acc = df_compose(prev, acc);
        }
    }
    if (LPP == 1 || lane >= 32 - P) agg[grp * P + p] = df_pack(acc);
    MapDF ex = df_ident();
    if constexpr (LPP > 1) {
        ex = df_up(acc, P);
        if (lane < P) ex = df_ident();
    }
    __syncthreads();
    DF R = DF{0.0f, 0.0f};
    if constexpr (LPP > 1) {
        // the maps of the groups before this warp's, composed over the pencil's lanes in order
        constexpr int GP = (G + LPP - 1) / LPP;
        const int k = lane / P;
        MapDF m = df_ident();
#pragma unroll
        for (int i = 0; i < GP; i++) {
            const int gi = k * GP + i;
            if (gi < grp) m = df_compose(m, df_unpack(agg[gi * P + p]));
        }
#pragma unroll
        for (int off = P; off < 32; off <<= 1) {
            const MapDF then = df_down(m, off);
            m = df_compose(m, then);
        }
        R = DF{__shfl_sync(~0u, m.C.h, lane % P), __shfl_sync(~0u, m.C.l, lane % P)};
        R = df_apply(ex, R);
    } else {
        for (int gi = 0; gi < grp; gi++) R = df_apply(df_unpack(agg[gi * P + p]), R);
    }
    return R.h + R.l;
}

// 1 - exp(-x), x >= 0, of the series branch of one_minus_exp_neg
__device__ __forceinline__ float one_minus_exp_series(float x) {
    return x * (1.0f - x * (0.5f - x * (1.0f / 6.0f - x * (1.0f / 24.0f - x * (1.0f / 120.0f - x * (1.0f / 720.0f))))));
}

// A *= exp(dz A_nl) on the 16 samples t = j + M q of pencil `line` in a (natural t; own = offset of
// (j, line) in the tile view); g: dA conj(A) of the same samples (SST).  xb: the exchange buffer, whose
// entries of these samples are this thread's; xd: a second tile buffer, free once every thread of the
// CTA has entered; release(): called when this step no longer needs xd.
template <class C, bool SST, bool PLASMA, class REL>
__device__ __forceinline__ void step_nonlinear(float2 (&a)[16], float2 (&g)[16], float2* xb, float2* xd, int own, const NLConst& c,
                                               void* scan_mem, float4* agg, int tid, float4& mx, const REL& release) {
    using V = typename C::View;
    constexpr int M = C::M;
    if constexpr (PLASMA) {
        // rates of the owned samples: b = Wava Kon and (1 - b) a + b, a = W1 Kon
        float xm = 0.0f;
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const float a2 = fmaf(a[q].x, a[q].x, a[q].y * a[q].y);
            xm = fmaxf(xm, a2);
            const float x = max_nan(a2, 1e-37f);
            const float rs = mufu_rsqrt(x);
            const float ak = mufu_ex2(fmaf(-c.e2[0], rs, fmaf(-c.e1[0], mufu_lg2(x), c.e0[0])));
            const float v = c.kv * (x * rs);
            const float b = (c.kb * mufu_rcp(fmaf(v, v, 1.0f))) * (v * x);
            xb[own + V::at(M * q, 0)] = make_float2(b, fmaf(1.0f - b, ak, b));
        }
        mx.x = fmaxf(mx.x, xm);
        // second-stage ionization (or an avalanche rate b >= 1/2) anywhere in the tile?  Below x2thr its
        // probability is under the flush threshold.
        const int any2 = __syncthreads_or(xm >= c.x2thr);
        if (!any2) release();
        // this thread's chunk: 16 consecutive samples of pencil p
        const int p = tid % C::P, t0 = (tid / C::P) * 16;
        float2* w = xb + V::at(t0, p);
        float B = 0.0f, Cc = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float2 r = w[V::walk(i)];
            Cc = fmaf(1.0f - r.x, Cc, r.y);
            B = fmaf(-B, r.x, B + r.x);
        }
        const float D = 1.0f - B;
        const float Rin = step_scan<C>(MapDF{DF{D, (1.0f - D) - B}, DF{Cc, 0.0f}}, agg, tid);
        if (!any2) {
            // ion fraction before each sample: 1 - exp(-R).  With every b < 1/2, R does not decrease
            // while it is below 1, so its last value bounds the chunk's.
            float R = Rin;
            if (fmaf(D, Rin, Cc) < 0.12f) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float2 r = w[V::walk(i)];
                    w[V::walk(i)].x = one_minus_exp_series(R);
                    R = fmaf(1.0f - r.x, R, r.y);
                }
            } else {
#pragma unroll 2
                for (int i = 0; i < 16; i++) {
                    const float2 r = w[V::walk(i)];
                    w[V::walk(i)].x = one_minus_exp_neg(R);
                    R = fmaf(1.0f - r.x, R, r.y);
                }
            }
            __syncthreads();
        } else {
            // the (ions2, ions1) recurrence (mpc_kernels.cuh): c2 of every sample through xd
            MapUV* muv = reinterpret_cast<MapUV*>(scan_mem);
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const float x = max_nan(fmaf(a[q].x, a[q].x, a[q].y * a[q].y), 1e-37f);
                const float c2 = mufu_ex2(fmaf(-c.e2[1], mufu_rsqrt(x), fmaf(-c.e1[1], mufu_lg2(x), c.e0[1])));
                xd[own + V::at(M * q, 0)].x = (c2 >= kC2Flush) ? c2 : 0.0f;
            }
            __syncthreads();
            const float2* w2 = xd + V::at(t0, p);
            float R = Rin;
            float m00 = 1.f, m01 = 0.f, m10 = 0.f, m11 = 1.f, o0 = 0.f, o1 = 0.f;
#pragma unroll 2
            for (int i = 0; i < 16; i++) {
                const float c2 = w2[V::walk(i)].x;
                const float2 rk = w[V::walk(i)];
                R = fmaf(1.0f - rk.x, R, rk.y);
                const float gk = one_minus_exp_neg(R);
                const float n00 = fmaf(c2, m10, m00), n01 = fmaf(c2, m11, m01);
                const float no0 = fmaf(c2, o1, o0), no1 = gk - o0;
                m10 = -m00;
                m11 = -m01;
                m00 = n00;
                m01 = n01;
                o1 = no1;
                o0 = no0;
            }
            muv[p * C::TPP + tid / C::P] = MapUV{m00, m01, m10, m11, o0, o1};
            __syncthreads();
            scan_chunks<MapUV, C::P, C::TPP>(muv, tid);
            __syncthreads();
            // before the pencil's first sample ions1 = ions2 = 0; the composed maps start from there
            float u = (float)muv[p * C::TPP + tid / C::P].o0, v = (float)muv[p * C::TPP + tid / C::P].o1;
            R = Rin;
#pragma unroll 2
            for (int i = 0; i < 16; i++) {
                const float c2 = w2[V::walk(i)].x;
                const float2 rk = w[V::walk(i)];
                R = fmaf(1.0f - rk.x, R, rk.y);
                const float gk = one_minus_exp_neg(R);
                w[V::walk(i)].x = fmaf(2.0f, u, v);   // state before the sample (plasma.c:238-241)
                const float nu = fmaf(c2, v, u);
                v = gk - u;
                u = nu;
            }
            __syncthreads();
            release();
        }
    }
    // exponents dz Re A_nl, dz Im A_nl (into g), and their largest magnitudes
    float mre = 0.0f, mim = 0.0f;
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const float a2 = fmaf(a[q].x, a[q].x, a[q].y * a[q].y);
        float re = 0.0f, im = c.gam_dz * a2;
        if constexpr (PLASMA) {
            const float ions = xb[own + V::at(M * q, 0)].x;
            mx.y = fmaxf(mx.y, ions);
            const float x = max_nan(a2, 1e-37f);
            const float v = c.kv * (x * mufu_rsqrt(x));
            const float pl = (c.pl_dz * ions) * mufu_rcp(fmaf(v, v, 1.0f));
            re = -pl * v;
            im = im - pl;
        } else {
            mx.x = fmaxf(mx.x, a2);
        }
        if constexpr (SST) {
            re = fmaf(-3.0f * c.sst_dz, g[q].x, re);
            im = fmaf(-c.sst_dz, g[q].y, im);
        }
        g[q] = make_float2(re, im);
        mre = fmaxf(mre, fabsf(re));
        mim = fmaxf(mim, fabsf(im));
    }
    mx.z = fmaxf(mx.z, mim * c.inv_dz);
    mx.w = fmaxf(mx.w, mre * c.inv_dz);
    if (mre < 0.015625f && mim < 0.25f) {   // the series of exp_small and sincos_small
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const float re = g[q].x, im = g[q].y, i2 = im * im;
            const float amp = 1.0f + re * (1.0f + re * (0.5f + re * (1.0f / 6.0f + re * (1.0f / 24.0f))));
            const float sn = im * (1.0f - i2 * (1.0f / 6.0f - i2 * (1.0f / 120.0f - i2 * (1.0f / 5040.0f))));
            const float cs = 1.0f - i2 * (0.5f - i2 * (1.0f / 24.0f - i2 * (1.0f / 720.0f - i2 * (1.0f / 40320.0f))));
            a[q] = cmul(a[q], make_float2(amp * cs, amp * sn));
        }
    } else {
        // beyond the series: one sample at a time, through this thread's exchange entries
#pragma unroll
        for (int q = 0; q < 16; q++) xb[own + V::at(M * q, 0)] = g[q];
#pragma unroll 1
        for (int q = 0; q < 16; q++) {
            float2* e = xb + own + (V::at(M * q, 0) - V::at(0, 0));
            float sn, cs;
            const float amp = exp_small(e->x);
            sincos_small(e->y, &sn, &cs);
            *e = make_float2(amp * cs, amp * sn);
        }
#pragma unroll
        for (int q = 0; q < 16; q++) a[q] = cmul(a[q], xb[own + V::at(M * q, 0)]);
    }
}

// ---- the sweep ----------------------------------------------------------------------------------
// SLO = 1: a warp's block comes and goes as one TMA box (tin, tout: the field as (floats of a row block,
// Nt / LL, LL, row blocks)), each warp waiting for its own; no thread moves elements and the 32-byte rows
// of a tile cost the load/store unit nothing.  SLO = 2: cp.async and plain stores.
template <int NT, int TP, int SLO, int LRB, bool SST, bool PLASMA>
__global__ void __launch_bounds__(StepCfg<NT, TP>::TH, 512 / StepCfg<NT, TP>::TH)
    step_kernel(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tout, PencilArgs args) {
    using C = StepCfg<NT, TP>;
    using V = typename C::View;
    constexpr int M = C::M;
    constexpr bool BOXED = SLO == 1;
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    unsigned char* smem_raw = smem_dyn + ((128u - (smem_addr(smem_dyn) & 127u)) & 127u);
    float2* cur = reinterpret_cast<float2*>(smem_raw);
    float2* oth = reinterpret_cast<float2*>(smem_raw + C::BUF);
    void* scan_mem = smem_raw + 2 * C::BUF;
    float4* agg = reinterpret_cast<float4*>(smem_raw + 2 * C::BUF + C::SCAN);
    float4* tw = reinterpret_cast<float4*>(smem_raw + 2 * C::BUF + C::SCAN + C::AGG);
    float* wpos = reinterpret_cast<float*>(tw + NT);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::BARS);   // two per warp
    volatile int* dead = reinterpret_cast<int*>(bars + 2 * C::NW);      // a load did not arrive
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int step = gridDim.x;
    constexpr Stride<(size_t)1 << LRB> RS{};
    const float2* in = reinterpret_cast<const float2*>(args.in);
    float2* out = reinterpret_cast<float2*>(args.out);
    int tile = blockIdx.x;
    if constexpr (BOXED) {
        if (tid == 0) {
            for (int i = 0; i < 2 * C::NW; i++) mbar_init(&bars[i], 1);
            *dead = 0;
            fence_mbar_init();
        }
    }
    stage_twiddles4<NT, C::TH>(tw, args.tw, tid);
    if constexpr (SST)
        for (int i = tid; i < NT; i += C::TH) wpos[i] = __ldg(&args.wpos[i]);
    __syncthreads();
    pdl_wait();
    // load this warp's block of tile t into buffer s, the k-th load of the warp
    auto load = [&](float2* s, int t, int k) {
        if constexpr (BOXED) {
            if (lane == 0) {
                const int q0 = t * C::P;
                uint64_t* bar = &bars[2 * warp + (k & 1)];
                fence_proxy_async_smem();   // the buffer's uses so far, before the copy
                mbar_arrive_expect_tx(bar, 4096);
                tma_load_4d(s + V::at(warp * C::BW, 0), &tin, 2 * (q0 & ((1 << LRB) - 1)), warp * C::NB, 0, q0 >> LRB, bar);
            }
        } else {
            step_load_block<C, SLO>(s, tile_base<NT, SLO>(in, t * C::P, LRB), RS, warp, lane);
        }
    };
    if (tile < args.ntiles) load(cur, tile, 0);
    float4 mx = make_float4(0.f, 0.f, 0.f, 0.f);   // this thread's maxima over its tiles
    const int line = tid % C::P, j = tid / C::P;   // owned samples t = j + M q of pencil `line`
    const int own = V::at(j, line);

    for (int k = 0; tile < args.ntiles; tile += step, k++) {
        const int next = tile + step;
        auto prefetch = [&] {
            if (next < args.ntiles) load(oth, next, k + 1);
        };
        if (next >= args.ntiles) pdl_launch_next();
        if constexpr (BOXED) {
            if (!mbar_wait(&bars[2 * warp + (k & 1)], (uint32_t)((k >> 1) & 1))) {
                *dead = 1;   // the late box is still on its way into this CTA's shared memory: wait (bounded) once more
                mbar_wait(&bars[2 * warp + (k & 1)], (uint32_t)((k >> 1) & 1));
            }
            if (lane == 0) bulk_wait_read<0>();   // the last tile's store has left `oth`
        } else {
            step_load_wait();
        }
        __syncwarp();
        step_sub_inverse<C, SST, BOXED>(cur, oth, tw, wpos, warp, lane);
        __syncthreads();
        if (BOXED && *dead) {   // the same for the whole CTA
            if (tid == 0) atomicExch(args.err, KERR_TMA_TIMEOUT);
            break;
        }
        float2 a[16], g[16];
#pragma unroll
        for (int q = 0; q < 16; q++) {
            a[q] = cur[own + V::at(M * q, 0)];
            if constexpr (SST) g[q] = oth[own + V::at(M * q, 0)];
        }
        inv_twiddle<SST>(a, g, tw + j, M);
        if constexpr (SST) dft<16, true>(g);
        dft<16, true>(a);
        if constexpr (SST) {
#pragma unroll
            for (int q = 0; q < 16; q++) g[q] = cmulc(g[q], a[q]);   // dA conj(A)
        }
        step_nonlinear<C, SST, PLASMA>(a, g, cur, oth, own, args.nl, scan_mem, agg, tid, mx, prefetch);
        dft<16, false>(a);
#pragma unroll
        for (int i = 1; i < 16; i++) a[i] = cmul(a[i], tw_cs(tw + j + (i - 1) * M));
#pragma unroll
        for (int q = 0; q < 16; q++) cur[own + V::at(M * q, 0)] = a[q];
        __syncthreads();
        if constexpr (!PLASMA) prefetch();
        step_sub_forward<C, SLO, BOXED>(cur, tw, tile_base<NT, SLO>(out, tile * C::P, LRB), RS, warp, lane);
        if constexpr (BOXED) {
            fence_proxy_async_smem();   // this lane's results, before the store reads them
            __syncwarp();
            if (lane == 0) {
                const int q0 = tile * C::P;
                tma_store_4d(&tout, 2 * (q0 & ((1 << LRB) - 1)), warp * C::NB, 0, q0 >> LRB, cur + V::at(warp * C::BW, 0));
                bulk_commit();
            }
        }
        float2* sw = cur;
        cur = oth;
        oth = sw;
    }
    if (BOXED && lane == 0) bulk_wait<0>();
    if (args.stats) stats_max<C::TH>(mx, args.stats, reinterpret_cast<float*>(scan_mem), tid);
}

// ---- the diagnostics ------------------------------------------------------------------------------
// One read of the spectrum S gives the temporal profile sum_q |A(t, q)|^2, the spectrum
// sum_q |S(pos, q)|^2 and the pencil energies sum_t |A(t, q)|^2: the inverse transform of step_kernel,
// whose threads meet the same positions (lane of the span-1 stage) and the same t (outer stage) in
// every tile, so both profiles add up in registers (FP32 over runs of kDiagRun tiles, then FP64 in
// shared memory); a pencil's energy is 16 samples per thread and the lanes of a warp in FP32 (19 additions
// in a row at most), then FP64.  A CTA leaves its two profiles in a row of its own (args.parts); the rows are added in
// order afterwards (k_diag_profiles), so that identical calls give identical bits.
// Bound: the shared-memory accesses of the inverse transform and the FP64 run sums (0.17 ms would be the
// read).  At 256x256x2048 0.44 ms with the tiles as TMA boxes, 0.54 with cp.async; a temporal, a spectral
// and an exit sweep took 2.8 ms before.
constexpr int kDiagRun = 32;

template <int NT, int TP, int SLO, int LRB>
__global__ void __launch_bounds__(StepCfg<NT, TP>::TH, 512 / StepCfg<NT, TP>::TH)
    diag_kernel(const __grid_constant__ CUtensorMap tin, PencilArgs args) {
    using C = StepCfg<NT, TP>;
    using V = typename C::View;
    constexpr int M = C::M, LL = C::LL, P = C::P;
    static_assert(P < 32, "lanes of a warp share a pencil, a t and a position");
    constexpr bool BOXED = SLO == 1;   // as in step_kernel
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    unsigned char* smem_raw = smem_dyn + ((128u - (smem_addr(smem_dyn) & 127u)) & 127u);
    float2* cur = reinterpret_cast<float2*>(smem_raw);
    float2* oth = reinterpret_cast<float2*>(smem_raw + C::BUF);
    double* part = reinterpret_cast<double*>(smem_raw + 2 * C::BUF);   // energy parts of the tile's pencils
    double* tsum = part + C::TH;                                       // |A|^2 by t, |S|^2 by position
    double* ssum = tsum + NT;
    float4* tw = reinterpret_cast<float4*>(ssum + NT);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::DIAG_BARS);   // two per warp
    volatile int* dead = reinterpret_cast<int*>(bars + 2 * C::NW);           // a load did not arrive
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int step = gridDim.x;
    constexpr Stride<(size_t)1 << LRB> RS{};
    const float2* in = reinterpret_cast<const float2*>(args.in);
    int tile = blockIdx.x;
    if constexpr (BOXED) {
        if (tid == 0) {
            for (int i = 0; i < 2 * C::NW; i++) mbar_init(&bars[i], 1);
            *dead = 0;
            fence_mbar_init();
        }
        __syncthreads();
    }
    // load this warp's block of tile t into buffer s, the k-th load of the warp
    auto load = [&](float2* s, int t, int k) {
        if constexpr (BOXED) {
            if (lane == 0) {
                const int q0 = t * P;
                uint64_t* bar = &bars[2 * warp + (k & 1)];
                fence_proxy_async_smem();   // the buffer's uses so far, before the copy
                mbar_arrive_expect_tx(bar, 4096);
                tma_load_4d(s + V::at(warp * C::BW, 0), &tin, 2 * (q0 & ((1 << LRB) - 1)), warp * C::NB, 0, q0 >> LRB, bar);
            }
        } else {
            step_load_block<C, SLO>(s, tile_base<NT, SLO>(in, t * P, LRB), RS, warp, lane);
        }
    };
    if (tile < args.ntiles) load(cur, tile, 0);
    stage_twiddles4<NT, C::TH>(tw, args.tw, tid);
    for (int i = tid; i < 2 * NT; i += C::TH) tsum[i] = 0.0;
    __syncthreads();
    const int line = tid % P, j = tid / P;
    const int own = V::at(j, line);
    float ft[16], fs[16];    // running sums of the current run of tiles: |A|^2 by t, |S|^2 by position
#pragma unroll
    for (int i = 0; i < 16; i++) ft[i] = fs[i] = 0.0f;
    int run = 0;
    for (int k = 0; tile < args.ntiles; tile += step, k++) {
        const int next = tile + step;
        if constexpr (BOXED) {
            if (!mbar_wait(&bars[2 * warp + (k & 1)], (uint32_t)((k >> 1) & 1))) {
                *dead = 1;   // the late box is still on its way into this CTA's shared memory: wait (bounded) once more
                mbar_wait(&bars[2 * warp + (k & 1)], (uint32_t)((k >> 1) & 1));
            }
        } else {
            step_load_wait();
        }
        __syncwarp();
        if (next < args.ntiles) load(oth, next, k + 1);
#pragma unroll
        for (int u = 0; u < 16 / LL; u++) {
            const int i = u * 32 + lane;
            const int o = BOXED ? V::at(warp * C::BW, 0) + i : V::at(warp * C::BW + (i / P) * LL, i % P);
#pragma unroll
            for (int q = 0; q < LL; q++) {
                const float2 v = cur[o + (BOXED ? q * C::NB * P : V::at(q, 0))];
                fs[u * LL + q] = fmaf(v.x, v.x, fmaf(v.y, v.y, fs[u * LL + q]));
            }
        }
        step_sub_inverse<C, false, BOXED>(cur, oth, tw, nullptr, warp, lane);
        __syncthreads();
        if (BOXED && *dead) {   // the same for the whole CTA
            if (tid == 0) atomicExch(args.err, KERR_TMA_TIMEOUT);
            // the next tile's box is still on its way into this CTA's shared memory: wait (bounded) for it
            if (next < args.ntiles) mbar_wait(&bars[2 * warp + ((k + 1) & 1)], (uint32_t)(((k + 1) >> 1) & 1));
            break;
        }
        float2 a[16];
#pragma unroll
        for (int q = 0; q < 16; q++) a[q] = cur[own + V::at(M * q, 0)];
        inv_twiddle<false>(a, a, tw + j, M);
        dft<16, true>(a);
        float e = 0.0f;
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const float a2 = fmaf(a[q].x, a[q].x, a[q].y * a[q].y);
            ft[q] += a2;
            e += a2;
        }
        if (args.pencil_energy) {   // the pencil's M threads: the lanes of a warp, then the warps
#pragma unroll
            for (int off = P; off < 32; off <<= 1) e += __shfl_xor_sync(~0u, e, off);
            if (lane < P) part[warp * P + lane] = (double)e;
            __syncthreads();
            constexpr int K = 32 / P;   // lanes that share a pencil's parts
            if (tid < P * K) {
                double tot = 0.0;
#pragma unroll
                for (int k = tid / P; k < C::NW; k += K) tot += part[k * P + tid % P];
#pragma unroll
                for (int off = P; off < P * K; off <<= 1) tot += __shfl_xor_sync(~0u, tot, off);
                if (tid < P) args.pencil_energy[tile * P + tid] = tot * args.out_scale * args.out_scale;
            }
        }
        if (++run == kDiagRun || next >= args.ntiles) {
            run = 0;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                double t = (double)ft[i], w = (double)fs[i];
                ft[i] = fs[i] = 0.0f;
#pragma unroll
                for (int off = 1; off < P; off <<= 1) {
                    t += __shfl_xor_sync(~0u, t, off);
                    w += __shfl_xor_sync(~0u, w, off);
                }
                if (lane % P == 0) {   // one lane of the CTA owns each t and each position
                    tsum[j + M * i] += t;
                    ssum[warp * C::BW + (((i / LL) * 32 + lane) / P) * LL + i % LL] += w;
                }
            }
        }
        __syncthreads();   // every thread has read its samples (and the parts): the buffers may turn over
        float2* sw = cur;
        cur = oth;
        oth = sw;
    }
    for (int i = tid; i < 2 * NT; i += C::TH) args.parts[(size_t)blockIdx.x * (2 * NT) + i] = tsum[i];   // ssum follows tsum
}

}  // namespace mpc
