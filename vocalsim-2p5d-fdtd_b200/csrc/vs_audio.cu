// vs_audio.cu -- WAV samples of listener traces on the device.
//
// Restates results/generate_audio.py:14-42 of the reference for a batch of
// traces: audio = P / max|P| clipped to [-1, 1]; for srate_mul > 1 a
// 2nd-order Butterworth low-pass at 5050 Hz (scipy.signal.butter(2, Wn)
// with Wn = 5050 / (44100 srate_mul / 2)) applied as scipy.signal.lfilter
// applies it -- the direct form II transposed recursion in double,
//   y = b0 x + z0;  z0 = (z1 + x b1) - y a1;  z1 = x b2 - y a2,
// zero initial state -- and every srate_mul-th sample kept (filtered[::mul]);
// the samples are rounded to float32 as the WAV is written.
//
// One block per trace: the block reduces max|P|, then filters the trace in
// chunks of kAudioThreads x kAudioRun samples.  The recursion is linear in its
// state (z0, z1): a thread runs it over its kAudioRun samples from rest, a scan
// over the block (the state's transition over a run is one 2 x 2 matrix, its
// powers the scan's factors) gives every thread the state it starts from, and
// a second pass over the samples, whose quotients stayed in registers, writes
// the kept ones.  The serial chain is 2 kAudioRun + 2 log2(kAudioThreads)
// steps a chunk instead of one per sample.  The transition's powers carry the
// rounding of double, enlarged by the poles' distance from 1, which shrinks with
// srate_mul: for samples in [-1, 1] the filtered values before they are rounded
// to float are off by 8e-16 (srate_mul 2), 4e-14 (15), 2e-13 (30) and 3.5e-12
// (64), the serial recursion's by 8e-16, 4e-15, 9e-15 and 2e-14 (against 80
// bits); half an ulp of the float output is 3e-8.
#include <cuda_runtime.h>

#include <cmath>
#include <complex>
#include <string>

#include "vs_device.h"

namespace vsb {
namespace {

constexpr double kAudioCutoffHz = 5050.0;   // generate_audio.py:29
constexpr int kAudioThreads = 512;
constexpr int kAudioWarps = kAudioThreads / 32;
constexpr int kAudioRun = 16;               // samples of a thread per chunk
constexpr int kAudioPad = kAudioRun + 1;    // its shared-memory stride (bank conflicts)

struct Mat2 {
    double a, b, c, d;                      // [a b; c d]
};
struct Vec2 {
    double x, y;
};

__device__ __forceinline__ Mat2 mul(const Mat2& p, const Mat2& q) {
    return {p.a * q.a + p.b * q.c, p.a * q.b + p.b * q.d, p.c * q.a + p.d * q.c, p.c * q.b + p.d * q.d};
}
// m v + w
__device__ __forceinline__ Vec2 apply(const Mat2& m, const Vec2& v, const Vec2& w) {
    return {m.a * v.x + m.b * v.y + w.x, m.c * v.x + m.d * v.y + w.y};
}

__global__ void __launch_bounds__(kAudioThreads)
audio_kernel(const float* __restrict__ traces, int64_t n, int mul_, double b0, double b1, double b2,
             double a1, double a2, float* __restrict__ out, int64_t nout) {
    const float* x = traces + (int64_t)blockIdx.x * n;
    float* y = out + (int64_t)blockIdx.x * nout;
    __shared__ float red[kAudioWarps];
    __shared__ float tile[kAudioThreads * kAudioPad];
    __shared__ Vec2 total[kAudioWarps], start[kAudioWarps];
    __shared__ Vec2 carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr unsigned kAll = 0xffffffffu;
    float m = 0.0f;
    for (int64_t i = tid; i < n; i += kAudioThreads) m = fmaxf(m, fabsf(x[i]));
    for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(kAll, m, s));
    if (lane == 0) red[warp] = m;
    if (tid == 0) carry = {0.0, 0.0};
    __syncthreads();
    m = red[0];
    for (int w = 1; w < kAudioWarps; ++w) m = fmaxf(m, red[w]);
    const double maxp = (double)m;
    auto sample = [&](float v) {
        const double a = __ddiv_rn((double)v, maxp);
        return a < -1.0 ? -1.0 : (a > 1.0 ? 1.0 : a);     // numpy.clip: NaN stays NaN
    };
    if (mul_ == 1) {
        for (int64_t i = tid; i < n; i += kAudioThreads) y[i] = (float)sample(x[i]);
        return;
    }
    auto step = [&](double a, Vec2& z) {
        const double yi = __dadd_rn(z.x, __dmul_rn(b0, a));
        z.x = __dsub_rn(__dadd_rn(z.y, __dmul_rn(a, b1)), __dmul_rn(yi, a1));
        z.y = __dsub_rn(__dmul_rn(a, b2), __dmul_rn(yi, a2));
        return yi;
    };
    // transition of the state over one run (no input), its powers 2^k for the
    // scan of a warp, its power `lane` and that of a whole warp
    Mat2 run{-a1, 1.0, -a2, 0.0};
    for (int k = kAudioRun; k > 1; k >>= 1) run = mul(run, run);
    Mat2 pw[5], here{1.0, 0.0, 0.0, 1.0};
    for (int k = 0; k < 5; ++k) {
        pw[k] = run;
        if ((lane >> k) & 1) here = mul(here, run);
        run = mul(run, run);                // after the loop: over 32 runs
    }
    for (int64_t c0 = 0; c0 < n; c0 += kAudioThreads * kAudioRun) {
        for (int k = 0; k < kAudioRun; ++k) {
            const int i = k * kAudioThreads + tid;
            tile[i / kAudioRun * kAudioPad + i % kAudioRun] = c0 + i < n ? x[c0 + i] : 0.0f;
        }
        __syncthreads();
        double a[kAudioRun];
#pragma unroll
        for (int k = 0; k < kAudioRun; ++k) a[k] = sample(tile[tid * kAudioPad + k]);
        Vec2 z{0.0, 0.0};
#pragma unroll
        for (int k = 0; k < kAudioRun; ++k) step(a[k], z);
        // state after each thread's run, from rest at the warp's start
        for (int k = 0; k < 5; ++k) {
            const Vec2 v{__shfl_up_sync(kAll, z.x, 1 << k), __shfl_up_sync(kAll, z.y, 1 << k)};
            if (lane >= 1 << k) z = apply(pw[k], v, z);
        }
        Vec2 before{__shfl_up_sync(kAll, z.x, 1), __shfl_up_sync(kAll, z.y, 1)};
        if (lane == 0) before = {0.0, 0.0};
        if (lane == 31) total[warp] = z;
        __syncthreads();
        if (tid == 0) {
            Vec2 s = carry;
            for (int w = 0; w < kAudioWarps; ++w) {
                start[w] = s;
                s = apply(run, s, total[w]);
            }
            carry = s;
        }
        __syncthreads();
        z = apply(here, start[warp], before);
        int64_t i = c0 + (int64_t)tid * kAudioRun;
        int phase = (int)(i % mul_);
        int64_t at = (i + mul_ - 1) / mul_;
#pragma unroll
        for (int k = 0; k < kAudioRun; ++k, ++i) {
            const double yi = step(a[k], z);
            if (phase == 0 && i < n) y[at++] = (float)yi;
            if (++phase == mul_) phase = 0;
        }
    }
}

}  // namespace

// butter(2, Wn, 'low') as scipy.signal designs it: analog prototype poles
// -exp(i pi m / 4), m = -1, 1; pre-warp w = 2 fs tan(pi Wn / fs) with fs = 2;
// poles times w, gain w^2; bilinear transform (fs2 = 2 fs): poles
// (fs2 + p) / (fs2 - p), two zeros at -1, gain k / prod(fs2 - p);
// b = k [1, 2, 1], a = real(poly(poles)).
void audio_filter(int srate_mul, double b[3], double a[3]) {
    const double pi = 3.14159265358979323846;
    const double wn = kAudioCutoffHz / (44100.0 * srate_mul / 2.0);
    const double fs = 2.0, fs2 = 2.0 * fs;
    const double warped = 2.0 * fs * std::tan(pi * wn / fs);
    std::complex<double> p[2];
    for (int i = 0; i < 2; ++i) {
        const double m = i == 0 ? -1.0 : 1.0;
        p[i] = -std::exp(std::complex<double>(0.0, pi * m / 4.0)) * warped;
    }
    const double k = warped * warped;
    const std::complex<double> z0 = (fs2 + p[0]) / (fs2 - p[0]), z1 = (fs2 + p[1]) / (fs2 - p[1]);
    const double kz = k * (1.0 / ((fs2 - p[0]) * (fs2 - p[1]))).real();
    b[0] = kz; b[1] = 2.0 * kz; b[2] = kz;
    a[0] = 1.0;
    a[1] = (-(z0 + z1)).real();
    a[2] = (z0 * z1).real();
}

int audio_device(const float* traces, int ntr, int64_t n, int mul, float* out, cudaStream_t st, std::string* err) {
    double b[3], a[3];
    audio_filter(mul, b, a);
    const int64_t nout = (n + mul - 1) / mul;
    audio_kernel<<<ntr, kAudioThreads, 0, st>>>(traces, n, mul, b[0], b[1], b[2], a[1], a[2], out, nout);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        *err = std::string("vs_audio: ") + cudaGetErrorString(e);
        return VS_ERR_CUDA;
    }
    return VS_OK;
}

}  // namespace vsb
