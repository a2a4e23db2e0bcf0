// mpc_noalloc.cu -- the nonlinear split-step operator for callers that cannot allocate.
//
// Some callers cannot call cudaMalloc: code that runs where allocation is not allowed or
// not safe (a host callback, a section of another library that has promised its caller
// not to allocate), processes whose device memory is handed out at start-up by a memory
// pool that owns every byte, and embedded hosts with a fixed device-memory budget.  They
// hold the field in device memory already and need the nonlinear step applied to it.
//
// mpc_nonlinear_noalloc does that without allocating anything: the tables of its kernel (twiddles,
// omega) live in the single file-scope array g_noalloc below, which every GPU that loads this library
// holds until the process exits.  Its kernel is the pencil sweep's nonlinear stage (Kerr,
// self-steepening through the spectral derivative, ADK ionization and plasma terms,
// propagation.c:164-327 and plasma.c:118-245 with the defects corrected) on a field given
// in real space, complex64, reference layout A[t*Nx*Ny + y*Nx + x], physical units.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "../../include/mpc_gpu.h"
#include "mpc_kernels.cuh"
#include "mpc_nlsetup.h"
#include "mpc_step.cuh"

namespace {

using mpc::kTilePoints;
using mpc::NLConst;

constexpr int kMaxNt = 2048;      // longest t axis supported
constexpr size_t kTwOff = 0;      // packed twiddle table (12 B per entry) in a 16 B-per-entry region
constexpr size_t kWposOff = kTwOff + (size_t)kMaxNt * 16;
constexpr size_t kNoallocBytes = kWposOff + (size_t)kMaxNt * sizeof(float);    // 40,960 B

// All tables of mpc_nonlinear_noalloc: [twiddles | omega per position]
static __device__ __align__(256) unsigned char g_noalloc[kNoallocBytes];

// omega at each FFT position, computed on the host and passed by value (8 KB of kernel
// parameters), so that no call reads host memory asynchronously
struct WposTable {
    float v[kMaxNt];
};

// Packed W_Nt table (mpc_fft.cuh Twiddles: (c, s) then -(c^2 + s^2 - 1)) and the omega of
// each FFT position, into the static array.
__global__ void k_noalloc_tables(int Nt, WposTable wp, float2* tw, float* wpos) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Nt) return;
    const int flat = mpc::tw_staged_index(Nt, k);
    double s, c;
    sincos(-2.0 * M_PI * (double)flat / (double)Nt, &s, &c);
    const float cf = flat < 0 ? 0.0f : (float)c, sf = flat < 0 ? 0.0f : (float)s;
    tw[k] = make_float2(cf, sf);
    reinterpret_cast<float*>(tw + Nt)[k] = flat < 0 ? 0.0f : (float)-((double)cf * cf + (double)sf * sf - 1.0);
    wpos[k] = wp.v[k];
}

// omega at each position of the in-place forward sweep (radices 16, ..., 16, r_last;
// pos = sum span_s k_s, freq = k_1 + r_1 k_2 + ...), from the centred omega grid w
void omega_of_positions(int Nt, const double* w, WposTable* out) {
    int bits = 0;   // Nt = 2^bits: the digits of a position are runs of its bits
    while ((1 << bits) < Nt) bits++;
    for (int k = 0; k < Nt; k++) {
        int freq = 0, mult = 0;
        for (int left = bits; left > 0;) {   // digits from the top, 4 bits each, the last one the rest
            const int r = left < 4 ? left : 4;
            left -= r;
            freq |= ((k >> left) & ((1 << r) - 1)) << mult;
            mult += r;
        }
        out->v[k] = (float)w[(freq + Nt / 2) & (Nt - 1)];
    }
}

// The nonlinear stage of the pencil sweep on a real-space complex64 field, in place, tiles and register
// layout as in step_kernel: a thread holds 16 samples t = j + M q of one pencil; FFT_t and the inverse
// transform of -i omega S / Nt go through one tile buffer, the two meeting at the span-1 stage in
// registers; dA conj(A), the nonlinear step and the store follow in registers.  The other tile buffer
// takes the next tile.
// Bound: as step_kernel (issue and barriers).  At 256x256x2048 1.27 ms a launch; the kernel before it,
// capped at 64 CTAs by a static dA scratch, took 5.3 ms.  Element-wise tile loads: 1.6 ms.
template <int NT, bool SST, bool PLASMA>
__global__ void __launch_bounds__(512, 1)
    k_nonlinear_noalloc(float2* A, int NP, int ntiles, float in_scale, float out_scale, NLConst c, const float2* tw_g,
                        const float* wpos_g, bool wide) {
    using C = mpc::StepCfg<NT, 8192>;
    using V = typename C::View;
    constexpr int M = C::M, LL = C::LL;
    static_assert(C::TH == 512, "16 samples per thread");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* xb = reinterpret_cast<float2*>(smem_raw);              // transforms and exchange
    float2* nx = reinterpret_cast<float2*>(smem_raw + C::BUF);     // the next tile's samples
    void* scan_mem = smem_raw + 2 * C::BUF;
    float4* agg = reinterpret_cast<float4*>(smem_raw + 2 * C::BUF + C::SCAN);
    float4* tw = reinterpret_cast<float4*>(smem_raw + 2 * C::BUF + C::SCAN + C::AGG);
    float* wpos = reinterpret_cast<float*>(tw + NT);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int line = tid % C::P, j = tid / C::P;
    const int own = V::at(j, line);
    // the next tile: 16-byte chunks of two pencils, or, for a field that is only 8-byte aligned, elements
    auto load = [&](int tile) {
        if (wide) {
            mpc::step_load_block<C, 1>(nx, A + (size_t)tile * C::P, (size_t)NP, warp, lane);
            return;
        }
        const float2* src = A + (size_t)j * NP + (size_t)tile * C::P + line;
#pragma unroll
        for (int q = 0; q < 16; q++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(mpc::smem_addr(nx + own + V::at(M * q, 0))),
                         "l"(src + (size_t)(M * q) * NP)
                         : "memory");
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    int tile = blockIdx.x;
    if (tile < ntiles) load(tile);
    if constexpr (SST) {
        mpc::stage_twiddles4<NT, C::TH>(tw, tw_g, tid);
        const float inv_nt = 1.0f / (float)NT;
        for (int i = tid; i < NT; i += C::TH) wpos[i] = wpos_g[i] * inv_nt;
        __syncthreads();
    }
    float4 mx = make_float4(0.f, 0.f, 0.f, 0.f);   // not reported here
    for (; tile < ntiles; tile += gridDim.x) {
        mpc::step_load_wait();
        __syncthreads();
        float2 a[16], g[16];
#pragma unroll
        for (int q = 0; q < 16; q++) a[q] = mpc::cscale(nx[own + V::at(M * q, 0)], in_scale);
        const int next = tile + gridDim.x;
        auto prefetch = [&] {
            if (next < ntiles) load(next);
        };
        if constexpr (!PLASMA && !SST) {
            __syncthreads();
            prefetch();
        }
        if constexpr (SST) {
#pragma unroll
            for (int q = 0; q < 16; q++) g[q] = a[q];
            mpc::dft<16, false>(g);
#pragma unroll
            for (int k = 1; k < 16; k++) g[k] = mpc::cmul(g[k], mpc::tw_cs(tw + j + (k - 1) * M));
#pragma unroll
            for (int q = 0; q < 16; q++) xb[own + V::at(M * q, 0)] = g[q];
            __syncthreads();
            if constexpr (!PLASMA) prefetch();   // every thread has read its samples
            const int gi = lane / C::P, jm = gi % LL;
            const int om = V::at(warp * C::BW + (gi / LL) * M + jm, lane % C::P);
            const float4* t = tw + mpc::tw_stage_offset(NT, M) + jm;
            if constexpr (C::MID) {
#pragma unroll
                for (int q = 0; q < 16; q++) g[q] = xb[om + V::at(LL * q, 0)];
                mpc::dft<16, false>(g);
#pragma unroll
                for (int k = 1; k < 16; k++) g[k] = mpc::cmul(g[k], mpc::tw_cs(t + (k - 1) * LL));
#pragma unroll
                for (int q = 0; q < 16; q++) xb[om + V::at(LL * q, 0)] = g[q];
                __syncwarp();
            }
#pragma unroll
            for (int u = 0; u < 16 / LL; u++) {
                const int i = u * 32 + lane;
                const int pos = warp * C::BW + (i / C::P) * LL;
                const int o = V::at(pos, i % C::P);
                float w[LL];
                mpc::load_run<LL>(w, wpos + pos);
                float2 v[LL];
#pragma unroll
                for (int q = 0; q < LL; q++) v[q] = xb[o + V::at(q, 0)];
                mpc::dft<LL, false>(v);
#pragma unroll
                for (int q = 0; q < LL; q++) v[q] = mpc::cscale(mpc::mul_mi<false>(v[q]), w[q]);
                mpc::dft<LL, true>(v);
#pragma unroll
                for (int q = 0; q < LL; q++) xb[o + V::at(q, 0)] = v[q];
            }
            if constexpr (C::MID) {
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 16; q++) g[q] = xb[om + V::at(LL * q, 0)];
#pragma unroll
                for (int k = 1; k < 16; k++) g[k] = mpc::cmulc(g[k], mpc::tw_cs(t + (k - 1) * LL));
                mpc::dft<16, true>(g);
#pragma unroll
                for (int q = 0; q < 16; q++) xb[om + V::at(LL * q, 0)] = g[q];
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 16; q++) g[q] = xb[own + V::at(M * q, 0)];
#pragma unroll
            for (int k = 1; k < 16; k++) g[k] = mpc::cmulc(g[k], mpc::tw_cs(tw + j + (k - 1) * M));
            mpc::dft<16, true>(g);
#pragma unroll
            for (int q = 0; q < 16; q++) g[q] = mpc::cmulc(g[q], a[q]);   // dA conj(A)
        }
        mpc::step_nonlinear<C, SST, PLASMA>(a, g, xb, nx, own, c, scan_mem, agg, tid, mx, prefetch);
        float2* dst = A + (size_t)j * NP + (size_t)tile * C::P + line;
#pragma unroll
        for (int q = 0; q < 16; q++) dst[(size_t)(M * q) * NP] = mpc::cscale(a[q], out_scale);
    }
}

struct NtKernel {
    int nt;
    // [self-steepening off, on][plasma off, on]
    void (*fn[2][2])(float2*, int, int, float, float, NLConst, const float2*, const float*, bool);
    int smem, pencils;
};
template <int NT>
constexpr NtKernel nt_kernel() {
    return NtKernel{NT,
                    {{k_nonlinear_noalloc<NT, false, false>, k_nonlinear_noalloc<NT, false, true>},
                     {k_nonlinear_noalloc<NT, true, false>, k_nonlinear_noalloc<NT, true, true>}},
                    mpc::StepCfg<NT, 8192>::SMEM, mpc::StepCfg<NT, 8192>::P};
}
const NtKernel kKernels[] = {nt_kernel<64>(), nt_kernel<256>(), nt_kernel<512>(), nt_kernel<1024>(), nt_kernel<2048>()};

// errors are reported on stderr, as the reference's functions report theirs, and as the
// status code
int noalloc_fail(int code, const char* what, cudaError_t e = cudaSuccess) {
    if (e != cudaSuccess) fprintf(stderr, "mpc_nonlinear_noalloc: %s: %s\n", what, cudaGetErrorString(e));
    else fprintf(stderr, "mpc_nonlinear_noalloc: %s\n", what);
    return code;
}

}  // namespace

extern "C" int mpc_nonlinear_noalloc(const mpc_params* p, void* A_dev, double dz, void* stream) {
    if (!p || !A_dev || !p->w) return noalloc_fail(MPC_ERR_ARG, "null argument");
    const int Nx = p->dims[0], Ny = p->dims[1], Nt = p->dims[2];
    if (Nx <= 0 || Ny <= 0 || Nt <= 0) return noalloc_fail(MPC_ERR_ARG, "dims must be positive");
    if (Nt > kMaxNt)
        return noalloc_fail(MPC_ERR_SHAPE, "Nt exceeds the static scratch of mpc_nonlinear_noalloc (at most 2048)");
    int ki = -1;
    for (int i = 0; i < (int)(sizeof(kKernels) / sizeof(kKernels[0])); i++)
        if (kKernels[i].nt == Nt) ki = i;
    if (ki < 0) return noalloc_fail(MPC_ERR_SHAPE, "Nt must be 64, 256, 512, 1024 or 2048");
    const long NP = (long)Nx * Ny;
    const int P = kTilePoints / Nt;
    if (NP % P != 0 || NP > (1L << 30))
        return noalloc_fail(MPC_ERR_SHAPE, "Nx*Ny must be a multiple of 16384/Nt");
    if (!(p->w0 > 0)) return noalloc_fail(MPC_ERR_ARG, "w0 must be positive");
    const double fs = sqrt(mpc::kHBAR * p->w0 / mpc::kIUnit);
    const mpc::NLSetup setup = mpc::nl_setup(*p, fs);
    if (p->plasm == 1 && !setup.gas_ok) return noalloc_fail(MPC_ERR_ARG, "unknown gas");
    NLConst c = setup.nl;
    mpc::nl_set_dz(setup, &c, dz, p->sst_on == 1);
    WposTable wp;
    omega_of_positions(Nt, p->w, &wp);
    // The device address of g_noalloc, looked up on every call with the caller's device current
    // (in host code the symbol is a host-side stand-in and must never be passed to a kernel);
    // the lookup allocates nothing.  The first call on a device loads this library's device code.
    void* addr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&addr, g_noalloc);
    if (e != cudaSuccess || !addr) return noalloc_fail(MPC_ERR_CUDA, "cudaGetSymbolAddress(g_noalloc)", e);
    int dev = 0, nsm = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return noalloc_fail(MPC_ERR_CUDA, "SM count", e);
    const auto fn = kKernels[ki].fn[c.sst_c != 0.0f][c.plasma];
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kKernels[ki].smem);
    if (e != cudaSuccess) return noalloc_fail(MPC_ERR_CUDA, "cudaFuncSetAttribute", e);
    unsigned char* base = static_cast<unsigned char*>(addr);
    float2* tw = reinterpret_cast<float2*>(base + kTwOff);
    float* wpos = reinterpret_cast<float*>(base + kWposOff);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_noalloc_tables<<<(Nt + 255) / 256, 256, 0, st>>>(Nt, wp, tw, wpos);
    e = cudaGetLastError();
    if (e != cudaSuccess) return noalloc_fail(MPC_ERR_CUDA, "table kernel launch", e);
    const int ntiles = (int)(NP / kKernels[ki].pencils);
    const int grid = ntiles < nsm ? ntiles : nsm;
    fn<<<grid, 512, kKernels[ki].smem, st>>>(static_cast<float2*>(A_dev), (int)NP, ntiles, (float)fs, (float)(1.0 / fs), c, tw,
                                             wpos, reinterpret_cast<uintptr_t>(A_dev) % 16 == 0);
    e = cudaGetLastError();
    if (e != cudaSuccess) return noalloc_fail(MPC_ERR_CUDA, "nonlinear kernel launch", e);
    return MPC_OK;
}
