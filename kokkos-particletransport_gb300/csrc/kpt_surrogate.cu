// Training and evaluation of the learned QLT closure (the project's own
// forward and backward kernels, FP32 SIMT; the network is tiny).
//
// Samples are drawn uniformly over the training box (feature units) with the
// keyed Philox stream; targets come from the plain slab-QLT closure in FP64
// (LegencyModel.hpp:557-645) and the driver's kappa_parallel closure
// (src/main.cpp:1177-1193).  One optimisation step: forward + backward per
// sample (activations and deltas kept in HBM), batch reductions for the
// weight gradients, then Adam.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "kpt_device.cuh"
#include "kpt_internal.h"
#include "kpt_surrogate.cuh"

namespace kpt {
namespace {

constexpr double kPiD = 3.141592653589793238462643383279502884;

// Plain slab-QLT closure (LegencyModel.hpp:557-645) with per-sample sigma^2
// and gamma_k, FP64: D_mumu, dD_mumu/dmu and the two network targets
// y0 = ln D - ln(1 - mu^2), y1 = (gk - 1) - gk reg^gk / (reg^gk + xi^gk).
__device__ void qlt_targets(double mu, double omega, double speed, double sigma2, double lc,
                            double gk, double h0, double& d, double& dd, double& y0,
                            double& y1) {
    d = 0.0;
    dd = 0.0;
    y0 = 0.0;
    y1 = 0.0;
    const double one_minus_mu2 = 1.0 - mu * mu;
    if (one_minus_mu2 <= 0.0) return;
    const double reg = fabs(mu) + h0;
    const double xi = omega * lc / speed;
    const double reg_gk = pow(reg, gk);
    const double reg_gk1 = pow(reg, gk - 1.0);
    const double denominator = reg_gk + pow(xi, gk);
    const double norm = gk * sin(kPiD / gk) / kPiD;
    const double prefactor = 0.25 * kPiD * omega * sigma2 * norm;
    d = prefactor * one_minus_mu2 * xi * reg_gk1 / denominator;
    y0 = log(prefactor * xi) + (gk - 1.0) * log(reg) - log(denominator);
    y1 = (gk - 1.0) - gk * reg_gk / denominator;
    if (d == 0.0 || mu == 0.0) return;
    const double sign = mu > 0.0 ? 1.0 : -1.0;
    dd = d * (-2.0 * mu / one_minus_mu2 + sign * ((gk - 1.0) / reg - gk * reg_gk1 / denominator));
}

// The driver's kappa_parallel closure (src/main.cpp:1177-1193).
__device__ double kappa_parallel(const SurrogateBox& box, double p, double b) {
    double k = box.kpara0;
    if (box.magnetic_dependency == 1) k *= pow(b, box.gamma_turb - 2.0);
    if (box.momentum_dependency == 1) k *= pow(p / box.p0, 3.0 - box.gamma_turb);
    return k;
}

__device__ __forceinline__ double u32_open(uint32_t r) {
    return (static_cast<double>(r) + 0.5) * 2.3283064365386963e-10;
}

// Training samples, uniform over the box in feature units (ln|mu|, ln p,
// ln|B|, ln sigma^2, gamma_k); x holds the raw features, t the targets.
__global__ void make_samples_kernel(uint64_t seed, int n, SurrogateBox box, float* x, float* t) {
    const uint2 key = seed_key(seed);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint4 r0 = philox4x32_10(make_uint4(0u, static_cast<uint32_t>(i), 0u, 7u), key);
        const uint4 r1 = philox4x32_10(make_uint4(1u, static_cast<uint32_t>(i), 0u, 7u), key);
        const uint32_t words[5] = {r0.x, r0.y, r0.z, r0.w, r1.x};
        double f[kMlpIn];
        for (int k = 0; k < kMlpIn; ++k) {
            f[k] = box.in_lo[k] + (static_cast<double>(box.in_hi[k]) - box.in_lo[k]) *
                                      u32_open(words[k]);
        }
        const double mu = exp(f[0]);
        const double p = exp(f[1]);
        const double b = exp(f[2]);
        const double sigma2 = exp(f[3]);
        const double gk = f[4];
        const double speed = box.particle_v0 * p / box.p0;
        const double omega = box.qlt_omega0 * b / sqrt(1.0 + p * p);
        double d, dd, y0, y1;
        qlt_targets(mu, omega, speed, sigma2, box.qlt_lc, gk, box.qlt_h0, d, dd, y0, y1);
        float* xi = x + static_cast<size_t>(i) * kMlpIn;
        for (int k = 0; k < kMlpIn; ++k) xi[k] = static_cast<float>(f[k]);
        float* ti = t + static_cast<size_t>(i) * kMlpOut;
        ti[0] = static_cast<float>(y0);
        ti[1] = static_cast<float>(y1);
        ti[2] = static_cast<float>(log(kappa_parallel(box, p, b)));
    }
}

// Rounding of the served network's 16-bit element type (quantization-aware
// fine-tuning): 0 none, 1 BF16 (round to nearest even), 2 FP16.
__device__ __forceinline__ float quantize(float v, int q) {
    if (q == 1) {
        uint32_t bits = __float_as_uint(v);
        bits = (bits + 0x7fffu + ((bits >> 16) & 1u)) & 0xffff0000u;
        return __uint_as_float(bits);
    }
    if (q == 2) {
        return __half2float(__float2half_rn(v));
    }
    return v;
}

__device__ __forceinline__ float normalise_input(const SurrogateBox& box, int k, float v) {
    return v * box.in_scale[k] + box.in_offset[k];
}

// ---- one optimisation step ------------------------------------------------------
// Three kernels: forward + backward (train_pass_kernel), the weight gradients
// of every chunk of kGradChunk samples (train_grad_kernel), the chunk sums and
// Adam (train_update_kernel).  Every sum runs over the same terms in the same
// order as one thread per sample (passes) or per parameter (gradients) would
// take them, each term one FMA: weights of a row in input order, samples of a
// chunk in sample order, chunks in chunk order, so the trained weights do not
// depend on the tiling.
//
// What bounds a step (batch 8192, width 64): 0.2 GFLOP of FP32 FMA is 1.4 us
// of the chip; the step is launch and latency bound, so the tiles are chosen
// to fill the SMs (256 pass blocks of 32 samples, 192 gradient blocks) rather
// than to reuse operands further, operands arrive by asynchronous copies that
// a block waits for once, and each kernel starts while the previous one
// drains.  A step takes 26 us; 115 us when a thread ran a whole sample with
// its activations in local memory and a gradient thread one column over 256
// samples from global memory.  Width 32: 61 -> 22 us.

constexpr int kPassSamples = 32;   // samples of a pass block
constexpr int kPassThreads = 256;
constexpr int kGradThreads = 256;

// Rows of H floats padded by four: 128-bit reads at a fixed column offset hit
// distinct banks for eight consecutive rows.
template <int H>
struct PassSmem {
    static constexpr int LD = H + 4;
    alignas(16) float w1[H * kMlpIn];
    alignas(16) float b1[H];
    alignas(16) float b2[H];
    alignas(16) float w3[kMlpOut * H];
    float b3[4];
    float in[kPassSamples * kMlpIn];
    float target[kPassSamples * 4];
    float dy[kPassSamples * 4];
    alignas(16) float w2[H * LD];
    alignas(16) float a1[kPassSamples * LD];
    alignas(16) float a2[kPassSamples * LD];  // activations, then deltas
};

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    v[0] = f.x;
    v[1] = f.y;
    v[2] = f.z;
    v[3] = f.w;
}

// 16 bytes from global to shared memory without a register: a block's whole
// operand set is in flight before it waits once.
__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" : : "r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// The kernels of consecutive steps are launched with programmatic dependence:
// a kernel's blocks may start while the previous kernel drains, and read or
// write nothing an earlier kernel touches before previous_done (which returns
// once the previous kernel, and so everything before it, has completed).  The
// buffers the kernels hand on therefore change while their readers are
// resident: they are plain pointers, read with ordinary loads after the wait.
// (const __restrict__ would promise data that is constant for the kernel's
// life, and allow non-coherent loads; only the training set is that.)
__device__ __forceinline__ void previous_done() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void next_may_start() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <int J>
__device__ __forceinline__ void load_row(const float* p, float (&v)[J]) {
    static_assert(J == 4 || J == 2, "H / 16 columns");
    if constexpr (J == 4) {
        load4(p, v);
    } else {
        const float2 f = *reinterpret_cast<const float2*>(p);
        v[0] = f.x;
        v[1] = f.y;
    }
}

// Forward and backward of 32 samples per block.  The two H x H products give
// each thread two samples (sg, sg + 16) times H / 16 columns; operands
// come four along the summed dimension per 128-bit read, from the weights'
// own row order in both directions.  Stores H1, H2 (activations) and G1, G2,
// GY (deltas) for the gradients.
template <int H>
__global__ void __launch_bounds__(kPassThreads)
    train_pass_kernel(const float* __restrict__ x, const float* __restrict__ t, int n,
                      uint64_t seed, int step, int batch, const SurrogateBox box,
                      const float* params, float* xb, float* h1, float* h2, float* g1, float* g2,
                      float* gy, float* loss, int quant) {
    // quant != 0: the forward sees the served network's rounding (weights,
    // inputs and activations in the 16-bit type, FP16 pre-activations too;
    // biases and accumulation FP32) and the backward passes straight
    // through it
    using M = Mlp<H>;
    using S = PassSmem<H>;
    constexpr int LD = S::LD;
    constexpr int J = H / 16;                             // columns of a thread
    constexpr int I = kPassSamples * 16 / kPassThreads;   // samples of a thread
    constexpr int SG = kPassSamples / I;                  // sample groups
    extern __shared__ __align__(16) unsigned char pass_smem[];
    S& sm = *reinterpret_cast<S*>(pass_smem);
    const int tid = threadIdx.x;
    const int b0 = blockIdx.x * kPassSamples;
    const int here = batch - b0 < kPassSamples ? batch - b0 : kPassSamples;
    next_may_start();
    // The block's samples are drawn and gathered from the fixed training set
    // before the previous step's update has to be complete.
    float in[kMlpIn] = {};
    if (tid < kPassSamples) {
        float target[kMlpOut] = {};
        if (tid < here) {
            const int b = b0 + tid;
            int i = b % n;
            if (step >= 0) {
                const uint4 r = philox4x32_10(make_uint4(static_cast<uint32_t>(b),
                                                         static_cast<uint32_t>(step), 0u, 9u),
                                              seed_key(seed));
                i = static_cast<int>(u01_f64(r.x, r.y) * n) % n;
            }
            for (int k = 0; k < kMlpIn; ++k) {
                in[k] = quantize(normalise_input(box, k, x[static_cast<size_t>(i) * kMlpIn + k]),
                                 quant);
            }
            for (int o = 0; o < kMlpOut; ++o) {
                target[o] = (t[static_cast<size_t>(i) * kMlpOut + o] - box.out_offset[o]) /
                            box.out_scale[o];
            }
        }
        for (int k = 0; k < kMlpIn; ++k) sm.in[tid * kMlpIn + k] = in[k];
        for (int o = 0; o < kMlpOut; ++o) sm.target[tid * 4 + o] = target[o];
    }
    previous_done();
    for (int k = tid; k < H * H / 4; k += kPassThreads) {
        copy16(sm.w2 + (4 * k / H) * LD + 4 * k % H, params + M::W2 + 4 * k);
    }
    for (int k = tid; k < H * kMlpIn / 4; k += kPassThreads) {
        copy16(sm.w1 + 4 * k, params + M::W1 + 4 * k);
    }
    if (tid < H / 4) {
        copy16(sm.b1 + 4 * tid, params + M::B1 + 4 * tid);
        copy16(sm.b2 + 4 * tid, params + M::B2 + 4 * tid);
    }
    if (tid < kMlpOut * H / 4) copy16(sm.w3 + 4 * tid, params + M::W3 + 4 * tid);
    if (tid < kMlpOut) sm.b3[tid] = params[M::B3 + tid];
    if (tid < here) {
        for (int k = 0; k < kMlpIn; ++k) xb[static_cast<size_t>(b0 + tid) * kMlpIn + k] = in[k];
    }
    copies_done();
    __syncthreads();
    if (quant != 0) {
        for (int k = tid; k < H * H; k += kPassThreads) {
            float& w = sm.w2[(k / H) * LD + k % H];
            w = quantize(w, quant);
        }
        for (int k = tid; k < H * kMlpIn; k += kPassThreads) sm.w1[k] = quantize(sm.w1[k], quant);
        for (int k = tid; k < kMlpOut * H; k += kPassThreads) {
            sm.w3[k] = quantize(sm.w3[k], quant);
        }
        __syncthreads();
    }
    // layer 1: sample s, columns c0, c0 + 4, ...
    {
        const int s = tid & (kPassSamples - 1);
        for (int j = tid / kPassSamples; j < H; j += kPassThreads / kPassSamples) {
            float z = sm.b1[j];
#pragma unroll
            for (int k = 0; k < kMlpIn; ++k) {
                z = fmaf(sm.w1[j * kMlpIn + k], sm.in[s * kMlpIn + k], z);
            }
            sm.a1[s * LD + j] = quantize(tanhf(quant == 2 ? quantize(z, quant) : z), quant);
        }
    }
    __syncthreads();
    const int sg = tid % SG;
    const int cg = tid / SG;  // 16 column groups
    // layer 2: columns j = cg + 16 m
    {
        float acc[I][J];
#pragma unroll
        for (int m = 0; m < J; ++m) {
#pragma unroll
            for (int i = 0; i < I; ++i) acc[i][m] = sm.b2[cg + 16 * m];
        }
#pragma unroll 4
        for (int k = 0; k < H; k += 4) {
            float a[I][4], w[J][4];
#pragma unroll
            for (int i = 0; i < I; ++i) load4(sm.a1 + (sg + SG * i) * LD + k, a[i]);
#pragma unroll
            for (int m = 0; m < J; ++m) load4(sm.w2 + (cg + 16 * m) * LD + k, w[m]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
#pragma unroll
                for (int i = 0; i < I; ++i) {
#pragma unroll
                    for (int m = 0; m < J; ++m) acc[i][m] = fmaf(w[m][e], a[i][e], acc[i][m]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < I; ++i) {
#pragma unroll
            for (int m = 0; m < J; ++m) {
                const float z = acc[i][m];
                sm.a2[(sg + SG * i) * LD + cg + 16 * m] =
                    quantize(tanhf(quant == 2 ? quantize(z, quant) : z), quant);
            }
        }
    }
    __syncthreads();
    // layer 3 and the loss: one thread per (sample, output); a warp per output
    float sq = 0.0f;
    if (tid < kMlpOut * kPassSamples) {
        const int s = tid & (kPassSamples - 1);
        const int o = tid / kPassSamples;
        float y = sm.b3[o];
#pragma unroll 4
        for (int j = 0; j < H; j += 4) {
            float a[4], w[4];
            load4(sm.a2 + s * LD + j, a);
            load4(sm.w3 + o * H + j, w);
#pragma unroll
            for (int e = 0; e < 4; ++e) y = fmaf(w[e], a[e], y);
        }
        float dy = 0.0f;
        if (s < here) {
            const float e = y - sm.target[s * 4 + o];
            sq = e * e;
            dy = 2.0f * e / static_cast<float>(batch * kMlpOut);
            gy[static_cast<size_t>(b0 + s) * kMlpOut + o] = dy;
        }
        sm.dy[s * 4 + o] = dy;
    }
    // batch loss (mean squared error in normalised units)
    for (int off = 16; off > 0; off >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, off);
    if ((tid & 31) == 0 && sq != 0.0f) {
        atomicAdd(loss, sq / static_cast<float>(batch * kMlpOut));
    }
    __syncthreads();
    // stores of the activations, deltas of layer 2 (whole rows, coalesced)
    for (int k = tid; k < kPassSamples * H; k += kPassThreads) {
        const int s = k / H;
        const int j = k % H;
        const float a2 = sm.a2[s * LD + j];
        float dh = 0.0f;
#pragma unroll
        for (int o = 0; o < kMlpOut; ++o) dh = fmaf(sm.w3[o * H + j], sm.dy[s * 4 + o], dh);
        const float dz = dh * fmaf(-a2, a2, 1.0f);
        if (s < here) {
            const size_t at = static_cast<size_t>(b0) * H + k;
            h1[at] = sm.a1[s * LD + j];
            h2[at] = a2;
            g2[at] = dz;
        }
        sm.a2[s * LD + j] = dz;
    }
    __syncthreads();
    // deltas of layer 1: columns k = J cg .. J cg + J - 1, summed over j
    {
        float acc[I][J] = {};
#pragma unroll 4
        for (int j = 0; j < H; j += 4) {
            float d[I][4], w[4][J];
#pragma unroll
            for (int i = 0; i < I; ++i) load4(sm.a2 + (sg + SG * i) * LD + j, d[i]);
#pragma unroll
            for (int e = 0; e < 4; ++e) load_row<J>(sm.w2 + (j + e) * LD + J * cg, w[e]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
#pragma unroll
                for (int i = 0; i < I; ++i) {
#pragma unroll
                    for (int m = 0; m < J; ++m) acc[i][m] = fmaf(w[e][m], d[i][e], acc[i][m]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < I; ++i) {
            const int s = sg + SG * i;
            if (s < here) {
#pragma unroll
                for (int m = 0; m < J; ++m) {
                    const float a = sm.a1[s * LD + J * cg + m];
                    g1[static_cast<size_t>(b0 + s) * H + J * cg + m] =
                        acc[i][m] * fmaf(-a, a, 1.0f);
                }
            }
        }
    }
}

// Weight and bias gradients of one chunk of samples:
//   W1 (H x 5):  sum_b G1[b][r] X[b][c];   b1[r] = sum_b G1[b][r]
//   W2 (H x H):  sum_b G2[b][r] H1[b][c];  b2[r] = sum_b G2[b][r]
//   W3 (3 x H):  sum_b GY[b][r] H2[b][c];  b3[r] = sum_b GY[b][r]
// blockIdx.y = chunk; blockIdx.x < (H / 32)^2: a 32 x 32 tile of W2 (and, in
// the first tile column, its part of b2 by a warp of its own), each thread 4
// rows x 1 column; then one block for W1 and b1 and one for W3 and b3.  The chunk's operands are
// staged in shared memory as a whole, so a block waits for memory once.
template <int H>
__host__ __device__ constexpr int grad_tiles() {
    return (H / 32) * (H / 32);
}
template <int H>
constexpr size_t grad_smem_bytes() {
    const size_t tile = 2u * kGradChunk * 32u;
    const size_t rest = kGradChunk * (H + kMlpIn);
    return (tile > rest ? tile : rest) * sizeof(float);
}
template <int H>
__global__ void __launch_bounds__(kGradThreads + 32)
    train_grad_kernel(int batch, const float* xb, const float* h1, const float* h2,
                      const float* g1, const float* g2, const float* gy, float* partial) {
    using M = Mlp<H>;
    extern __shared__ __align__(16) float grad_smem[];
    const int tid = threadIdx.x;
    const int part = static_cast<int>(blockIdx.x);
    const int b0 = blockIdx.y * kGradChunk;
    const int count = batch - b0 < kGradChunk ? batch - b0 : kGradChunk;
    float* out = partial + static_cast<size_t>(blockIdx.y) * M::Params;
    next_may_start();
    previous_done();
    if (part < grad_tiles<H>()) {
        const int r0 = part / (H / 32) * 32;
        const int c0 = part % (H / 32) * 32;
        float* d = grad_smem;
        float* in = grad_smem + kGradChunk * 32;
        for (int k = tid; k < count * 8; k += blockDim.x) {
            const int b = k >> 3;
            const int q = (k & 7) * 4;
            const size_t row = static_cast<size_t>(b0 + b) * H;
            copy16(d + b * 32 + q, g2 + row + r0 + q);
            copy16(in + b * 32 + q, h1 + row + c0 + q);
        }
        copies_done();
        __syncthreads();
        if (tid >= kGradThreads) {  // the last warp: the bias of row r0 + lane
            if (c0 == 0) {
                const int r = tid - kGradThreads;
                float bacc = 0.0f;
#pragma unroll 8
                for (int b = 0; b < count; ++b) bacc += d[b * 32 + r];
                out[M::B2 + r0 + r] = bacc;
            }
            return;
        }
        const int r = (tid >> 5) * 4;
        const int c = tid & 31;
        float acc[4] = {};
#pragma unroll 8
        for (int b = 0; b < count; ++b) {
            float dv[4];
            load4(d + b * 32 + r, dv);
            const float iv = in[b * 32 + c];
#pragma unroll
            for (int m = 0; m < 4; ++m) acc[m] = fmaf(dv[m], iv, acc[m]);
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) out[M::W2 + (r0 + r + m) * H + c0 + c] = acc[m];
        return;
    }
    // thread: hidden unit r and columns (W1) or rows (W3) g, g + G, ...
    const bool first_layer = part == grad_tiles<H>();
    constexpr int G = kGradThreads / H;
    const int r = tid & (H - 1);
    const int g = tid / H;
    float* units = grad_smem;                 // G1 or H2
    float* other = units + kGradChunk * H;    // X or GY
    const float* src = first_layer ? g1 : h2;
    for (int k = tid; k < count * H / 4; k += blockDim.x) {
        copy16(units + 4 * k, src + static_cast<size_t>(b0) * H + 4 * k);
    }
    const int width = first_layer ? kMlpIn : kMlpOut;
    const float* src2 = (first_layer ? xb : gy) + static_cast<size_t>(b0) * width;
    // a chunk's rows start on a 16-byte boundary (256 samples); the last
    // floats of a ragged chunk go one by one
    const int whole = count * width / 4;
    for (int k = tid; k < whole; k += blockDim.x) copy16(other + 4 * k, src2 + 4 * k);
    if (tid < count * width - 4 * whole) other[4 * whole + tid] = src2[4 * whole + tid];
    copies_done();
    __syncthreads();
    if (tid >= kGradThreads) {  // the last warp: b3
        const int o = tid - kGradThreads;
        if (!first_layer && o < kMlpOut) {
            float bacc = 0.0f;
#pragma unroll 8
            for (int b = 0; b < count; ++b) bacc += other[b * kMlpOut + o];
            out[M::B3 + o] = bacc;
        }
        return;
    }
    if (first_layer) {
        constexpr int N = (kMlpIn + 1 + G - 1) / G;  // column 5: the bias
        float acc[N] = {};
#pragma unroll 8
        for (int b = 0; b < count; ++b) {
            const float d = units[b * H + r];
#pragma unroll
            for (int m = 0; m < N; ++m) {
                const int c = g + m * G;
                const float v = c < kMlpIn ? other[b * kMlpIn + c] : 1.0f;
                acc[m] = fmaf(d, v, acc[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < N; ++m) {
            const int c = g + m * G;
            if (c < kMlpIn) out[M::W1 + r * kMlpIn + c] = acc[m];
            if (c == kMlpIn) out[M::B1 + r] = acc[m];
        }
    } else {
        constexpr int N = (kMlpOut + G - 1) / G;
        float acc[N] = {};
#pragma unroll 8
        for (int b = 0; b < count; ++b) {
            const float a = units[b * H + r];
#pragma unroll
            for (int m = 0; m < N; ++m) {
                const int o = g + m * G < kMlpOut ? g + m * G : 0;
                acc[m] = fmaf(other[b * kMlpOut + o], a, acc[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < N; ++m) {
            const int o = g + m * G;
            if (o < kMlpOut) out[M::W3 + o * H + r] = acc[m];
        }
    }
}

// The chunk partials of one parameter in chunk order.
__device__ __forceinline__ float chunk_sum(const float* partial, int chunks, int params, int k) {
    float sum = 0.0f;
#pragma unroll 16
    for (int ch = 0; ch < chunks; ++ch) sum += partial[static_cast<size_t>(ch) * params + k];
    return sum;
}

__global__ void grad_sum_kernel(const float* partial, int chunks, int params, float* grad) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < params) grad[k] = chunk_sum(partial, chunks, params, k);
}

// Chunk sums and Adam, one thread per parameter.
__global__ void train_update_kernel(const float* partial, int chunks, float* params, float* m,
                                    float* v, int count, float lr, float beta1, float beta2,
                                    float eps, float bias1, float bias2) {
    next_may_start();
    previous_done();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const float g = chunk_sum(partial, chunks, count, k);
    const float mk = beta1 * m[k] + (1.0f - beta1) * g;
    const float vk = beta2 * v[k] + (1.0f - beta2) * g * g;
    m[k] = mk;
    v[k] = vk;
    params[k] -= lr * (mk / bias1) / (sqrtf(vk / bias2) + eps);
}

// A launch that may overlap the end of the stream's previous kernel (the first
// kernel after a copy is ordered behind it as a whole: overlap = false).
template <typename... Params, typename... Args>
cudaError_t launch_dependent(bool overlap, void (*kernel)(Params...), dim3 grid, int threads,
                             size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attr;
    config.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// The pass and the chunk gradients of one batch (step < 0: its first samples
// in order).
template <int H>
cudaError_t launch_gradients(const SurrogateTrainLaunch& L, int step, float* loss, int quant,
                             cudaStream_t stream) {
    const int chunks = (L.batch + kGradChunk - 1) / kGradChunk;
    const cudaError_t err = launch_dependent(
        step > 0, train_pass_kernel<H>, dim3((L.batch + kPassSamples - 1) / kPassSamples), kPassThreads,
        sizeof(PassSmem<H>), stream, L.x, L.t, L.n, L.seed, step, L.batch, L.box, L.params, L.xb,
        L.h1, L.h2, L.g1, L.g2, L.gy, loss, quant);
    if (err != cudaSuccess) return err;
    return launch_dependent(true, train_grad_kernel<H>, dim3(grad_tiles<H>() + 2, chunks),
                            kGradThreads + 32, grad_smem_bytes<H>(), stream, L.batch, L.xb, L.h1,
                            L.h2, L.g1, L.g2, L.gy, L.partial);
}

// Shared memory beyond 48 KB has to be asked for once per kernel.
template <int H>
cudaError_t prepare_training() {
    cudaError_t err = cudaFuncSetAttribute(train_pass_kernel<H>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(sizeof(PassSmem<H>)));
    if (err != cudaSuccess) return err;
    return cudaFuncSetAttribute(train_grad_kernel<H>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(grad_smem_bytes<H>()));
}

// FP32 SIMT forward of normalised features -> normalised outputs.
template <int H>
__device__ void forward_fp32(const float* w, const float (&in)[kMlpIn], float (&y)[kMlpOut]) {
    using M = Mlp<H>;
    float a1[H];
    for (int j = 0; j < H; ++j) {
        float z = w[M::B1 + j];
        for (int k = 0; k < kMlpIn; ++k) z += w[M::W1 + j * kMlpIn + k] * in[k];
        a1[j] = tanhf(z);
    }
    for (int o = 0; o < kMlpOut; ++o) y[o] = w[M::B3 + o];
    for (int j = 0; j < H; ++j) {
        float z = w[M::B2 + j];
        for (int k = 0; k < H; ++k) z += w[M::W2 + j * H + k] * a1[k];
        const float a2 = tanhf(z);
        for (int o = 0; o < kMlpOut; ++o) y[o] += w[M::W3 + o * H + j] * a2;
    }
}

// Raw inputs (mu, ln p, ln|B|, sigma^2, gamma_k) -> (D_mumu, dD_mumu/dmu,
// ln kappa_parallel), FP64 out.  The network (FP32 SIMT, or a tensor-core
// engine of the push) serves inputs inside the box with |mu| >= mu_cut; the
// plain closure serves the rest.
//
// Features of input i (zeros for an idle thread and outside the box);
// returns whether the network serves it.
__device__ __forceinline__ bool eval_features(int i, bool have, const double* __restrict__ in,
                                              const SurrogateBox& box, double (&raw)[kMlpIn],
                                              float (&f)[kMlpIn]) {
    for (int k = 0; k < kMlpIn; ++k) raw[k] = 0.0;
    if (have) {
        for (int k = 0; k < kMlpIn; ++k) raw[k] = in[static_cast<size_t>(i) * kMlpIn + k];
    }
    const double mu = raw[0];
    const double feat[kMlpIn] = {log(fabs(mu)), raw[1], raw[2], log(raw[3]), raw[4]};
    bool inside = have && fabs(mu) >= box.mu_cut;
    for (int k = 0; k < kMlpIn; ++k) {
        inside = inside && feat[k] >= box.in_lo[k] && feat[k] <= box.in_hi[k];
        f[k] = static_cast<float>(feat[k]) * box.in_scale[k] + box.in_offset[k];
    }
    if (!inside) {
        for (int k = 0; k < kMlpIn; ++k) f[k] = 0.0f;
    }
    return inside;
}

// Closure values of input i from the network outputs y (or the plain
// closure outside the box), with the push's hand-over near mu_cut.
__device__ __forceinline__ void eval_store(int i, const double (&raw)[kMlpIn], bool inside,
                                           const float (&y)[kMlpOut], const SurrogateBox& box,
                                           double* __restrict__ out, int* __restrict__ served) {
    const double mu = raw[0];
    const double p = exp(raw[1]);
    const double b = exp(raw[2]);
    double d, dd, lk;
    const double speed = box.particle_v0 * p / box.p0;
    const double omega = box.qlt_omega0 * b / sqrt(1.0 + p * p);
    double pd, pdd, py0, py1;
    qlt_targets(mu, omega, speed, raw[3], box.qlt_lc, raw[4], box.qlt_h0, pd, pdd, py0, py1);
    const double plk = log(kappa_parallel(box, p, b));
    if (inside) {
        const double y0 = static_cast<double>(y[0]) * box.out_scale[0] + box.out_offset[0];
        const double y1 = static_cast<double>(y[1]) * box.out_scale[1] + box.out_offset[1];
        lk = static_cast<double>(y[2]) * box.out_scale[2] + box.out_offset[2];
        const double one_minus_mu2 = 1.0 - mu * mu;
        const double sign = mu > 0.0 ? 1.0 : -1.0;
        d = one_minus_mu2 * exp(y0);
        dd = d * (sign * y1 / (fabs(mu) + box.qlt_h0) - 2.0 * mu / one_minus_mu2);
        const double amu = fabs(mu);
        if (amu < 2.0 * box.mu_cut) {
            // the push's hand-over to the plain closure over [mu_cut, 2 mu_cut]
            const double w = (amu - box.mu_cut) / box.mu_cut;
            const double dw = sign / box.mu_cut;
            dd = pdd + w * (dd - pdd) + dw * (d - pd);
            d = pd + w * (d - pd);
            lk = log(exp(plk) + w * (exp(lk) - exp(plk)));
        }
    } else {
        d = pd;
        dd = pdd;
        lk = plk;
    }
    out[static_cast<size_t>(i) * kMlpOut + 0] = d;
    out[static_cast<size_t>(i) * kMlpOut + 1] = dd;
    out[static_cast<size_t>(i) * kMlpOut + 2] = lk;
    served[i] = inside ? 1 : 0;
}

// FP32 SIMT (MODE 0) or the warp-collective mma.sync engine (MODE 1 BF16,
// 2 FP16).  Warps stay converged (the loop bound is per warp) because the
// tensor-core path is collective.
template <int MODE, int H>
__global__ void __launch_bounds__(128) eval_kernel(int n, const double* __restrict__ in,
                                                   SurrogateBox box,
                                                   const float* __restrict__ params,
                                                   const uint2* __restrict__ block,
                                                   double* __restrict__ out,
                                                   int* __restrict__ served) {
    extern __shared__ uint2 smem[];
    if (MODE != 0) {
        load_surrogate_block<H>(block, smem);
    } else {
        float* w = reinterpret_cast<float*>(smem);
        for (int k = threadIdx.x; k < Mlp<H>::Params; k += blockDim.x) w[k] = params[k];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int base = warp * 32; base < n; base += warps * 32) {
        const int i = base + lane;
        const bool have = i < n;
        double raw[kMlpIn];
        float f[kMlpIn];
        const bool inside = eval_features(i, have, in, box, raw, f);
        float y[kMlpOut];
        if (MODE != 0) {
            mlp_warp<MODE == 2, H>(smem, f, y);
        } else {
            forward_fp32<H>(reinterpret_cast<const float*>(smem), f, y);
        }
        if (have) eval_store(i, raw, inside, y, box, out, served);
    }
}

// The tcgen05 engine: each block takes 128 inputs per trip (its rows), the
// trip count uniform over the block.
template <bool FP16, int H>
__global__ void __launch_bounds__(128) eval_tc_kernel(int n, const double* __restrict__ in,
                                                      SurrogateBox box,
                                                      const uint4* __restrict__ block,
                                                      double* __restrict__ out,
                                                      int* __restrict__ served,
                                                      unsigned int* __restrict__ timeouts) {
    extern __shared__ __align__(128) unsigned char tc_smem[];
    TcNet net = tc_setup<H>(block, tc_smem);
    tc_constants<FP16, H>(net);
    bool fail = false;
    for (int base = blockIdx.x * 128; base < n; base += gridDim.x * 128) {
        const int i = base + static_cast<int>(threadIdx.x);
        const bool have = i < n;
        double raw[kMlpIn];
        float f[kMlpIn];
        const bool inside = eval_features(i, have, in, box, raw, f);
        float y[kMlpOut];
        if (mlp_cta<FP16, H>(net, f, y, fail)) {
            break;
        }
        if (have) eval_store(i, raw, inside, y, box, out, served);
    }
    fail = __syncthreads_or(fail ? 1 : 0) != 0;
    if (fail && threadIdx.x == 0) {
        atomicAdd(timeouts, 1u);
    }
    tc_teardown<H>(net, fail);
}

// The failure path of the tcgen05 engine without a fault: every block sets
// up its network (weights, barrier, 128 TMEM columns), waits for a
// completion that nothing will signal (no MMA is issued) with `polls`
// polls, records the timeout, and tears down as a timed-out push block does
// (a second bounded wait, then the TMEM is freed).
__global__ void __launch_bounds__(128) tc_timeout_check_kernel(const uint4* __restrict__ block,
                                                               uint32_t polls,
                                                               unsigned int* __restrict__ out) {
    extern __shared__ __align__(128) unsigned char tc_smem[];
    TcNet net = tc_setup<64>(block, tc_smem);
    bool fail = !mbar_wait(net.mbar, net.phase, polls);
    net.phase ^= 1u;
    fail = __syncthreads_or(fail ? 1 : 0) != 0;
    if (fail && threadIdx.x == 0) {
        atomicAdd(out, 1u);
    }
    tc_teardown<64>(net, fail, polls);
    if (threadIdx.x == 0) {
        atomicAdd(out + 1, 1u);  // blocks that got past the teardown
    }
}

}  // namespace

cudaError_t surrogate_tc_timeout_check(const uint4* block, int blocks, uint32_t polls,
                                       unsigned int* out, cudaStream_t stream) {
    tc_timeout_check_kernel<<<blocks, 128, tc_smem_bytes<64>(), stream>>>(block, polls, out);
    return cudaGetLastError();
}

cudaError_t surrogate_make_samples(uint64_t seed, int n, const SurrogateBox& box, float* x,
                                   float* t, cudaStream_t stream) {
    const int threads = 256;
    const int blocks = (n + threads - 1) / threads < 152 * 16 ? (n + threads - 1) / threads
                                                              : 152 * 16;
    make_samples_kernel<<<blocks, threads, 0, stream>>>(seed, n, box, x, t);
    return cudaGetLastError();
}

namespace {

template <int H>
cudaError_t train_step(const SurrogateTrainLaunch& L, int step, cudaStream_t stream) {
    const cudaError_t err = launch_gradients<H>(L, step, L.loss + step,
                                                step >= L.quant_from ? L.quant : 0, stream);
    if (err != cudaSuccess) return err;
    const float t1 = static_cast<float>(step + 1);
    const float bias1 = 1.0f - powf(L.beta1, t1);
    const float bias2 = 1.0f - powf(L.beta2, t1);
    const int chunks = (L.batch + kGradChunk - 1) / kGradChunk;
    return launch_dependent(true, train_update_kernel, dim3((Mlp<H>::Params + 63) / 64), 64, 0, stream,
                            L.partial, chunks, L.params, L.m, L.v, Mlp<H>::Params, L.lr, L.beta1,
                            L.beta2, 1e-8f, bias1, bias2);
}

template <int H>
cudaError_t gradient(const SurrogateTrainLaunch& L, cudaStream_t stream) {
    cudaError_t err = prepare_training<H>();
    if (err == cudaSuccess) err = launch_gradients<H>(L, -1, L.loss, 0, stream);
    if (err != cudaSuccess) return err;
    const int chunks = (L.batch + kGradChunk - 1) / kGradChunk;
    grad_sum_kernel<<<(Mlp<H>::Params + 63) / 64, 64, 0, stream>>>(L.partial, chunks,
                                                                   Mlp<H>::Params, L.grad);
    return cudaGetLastError();
}

template <int H>
cudaError_t eval(int n, const double* inputs, const SurrogateBox& box, const SurrogateServe& sv,
                 double* out, int* served, cudaStream_t stream) {
    const int threads = 128;
    int blocks = (n + threads - 1) / threads;
    if (sv.engine == kEngineTcgen05) {
        // blocks beyond the 4 per SM whose TMEM fits wait in tcgen05.alloc
        // until a resident block frees its columns
        blocks = blocks < 1 ? 1 : (blocks > 152 * 4 ? 152 * 4 : blocks);
        const size_t smem = tc_smem_bytes<H>();
        if (box.fp16) {
            eval_tc_kernel<true, H><<<blocks, threads, smem, stream>>>(
                n, inputs, box, sv.tc_block, out, served, sv.timeouts);
        } else {
            eval_tc_kernel<false, H><<<blocks, threads, smem, stream>>>(
                n, inputs, box, sv.tc_block, out, served, sv.timeouts);
        }
        return cudaGetLastError();
    }
    blocks = blocks < 1 ? 1 : (blocks > 152 * 8 ? 152 * 8 : blocks);
    const size_t smem = Mlp<H>::SmemBytes;
    if (sv.engine == kEngineMmaSync && box.fp16) {
        eval_kernel<2, H><<<blocks, threads, smem, stream>>>(n, inputs, box, sv.params, sv.block,
                                                             out, served);
    } else if (sv.engine == kEngineMmaSync) {
        eval_kernel<1, H><<<blocks, threads, smem, stream>>>(n, inputs, box, sv.params, sv.block,
                                                             out, served);
    } else {
        eval_kernel<0, H><<<blocks, threads, Mlp<H>::Params * sizeof(float), stream>>>(
            n, inputs, box, sv.params, sv.block, out, served);
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t surrogate_prepare_training(int hidden) {
    return hidden == 64 ? prepare_training<64>() : prepare_training<32>();
}

cudaError_t surrogate_train_step(const SurrogateTrainLaunch& L, int step, cudaStream_t stream) {
    return L.box.hidden == 64 ? train_step<64>(L, step, stream) : train_step<32>(L, step, stream);
}

cudaError_t surrogate_gradient(const SurrogateTrainLaunch& L, cudaStream_t stream) {
    return L.box.hidden == 64 ? gradient<64>(L, stream) : gradient<32>(L, stream);
}

cudaError_t surrogate_eval(int n, const double* inputs, const SurrogateBox& box,
                           const SurrogateServe& serve, double* out, int* served,
                           cudaStream_t stream) {
    return box.hidden == 64 ? eval<64>(n, inputs, box, serve, out, served, stream)
                            : eval<32>(n, inputs, box, serve, out, served, stream);
}

}  // namespace kpt
