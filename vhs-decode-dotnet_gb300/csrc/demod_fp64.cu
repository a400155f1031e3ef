// Plain FP64 block demodulator: full-length complex FFTs in global memory
// (Stockham radix-8, five passes), every kernel over a batch of blocks.  It
// restates the same per-block math as the fused FP32 kernel
// (Core/Dsp/RfDemodulator.cs:288-918) in binary64 and is the baseline the
// fused path is measured against.
//
// What bounds it is GB300's binary64 pipe (a warp instruction holds an SM's
// pipe for about 17 cycles): some 270,000 binary64 warp instructions a block,
// 15 us of the whole chip.  So a batch of blocks fills the chip (one block at
// a time left it idle: 0.54 ms a block), the twiddles come from a table of the
// same sincospi values instead of being computed in every butterfly (as much
// binary64 work as the transforms), the element-wise steps are the loads and
// stores of the transforms' first and last passes, and a last pass computes
// only what is kept: bins 0 .. N/2 of a real signal's spectrum, the real part
// of a real signal's samples.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_common.cuh"
#include "vhs_math.cuh"
#include "kernels.h"

namespace vhsd {
namespace fp64 {

constexpr int N = 32768;
constexpr int H = N / 2;

__device__ __forceinline__ double2 wN(int k, bool inv) {
    double s, c;
    sincospi(-2.0 * (double)k / (double)N, &s, &c);
    return make_double2(c, inv ? -s : s);
}

__global__ void k_twiddles(double2* tw) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < N) tw[k] = wN(k, false);
}

// What a transform's first pass reads (kSrc) and its last pass writes (kDst).
enum Src { kPlainSrc, kRf, kAnalytic, kReal, kFilter, kSub };
enum Dst { kPlainDst, kHalfDst, kRealDst, kStreamDst };
struct PassIo {
    const double2* in;         // [block][N] complex (kPlainSrc; the spectrum of kAnalytic, kFilter, kSub)
    const double* real;        // [block][N] samples (kReal)
    const int16_t* rf;         // the batch's first block in the capture (kRf)
    const float* rf32;
    const double* gain;        // [kHalf] (kAnalytic)
    const double2* h;          // [kHalf] (kFilter, kSub)
    double2* out;              // [block][N] complex
    double* real_out;          // [block][N] real parts (kRealDst), or the batch's first block in the
    int shift;                 // stitched stream (kStreamDst: samples n = s + kCut + shift)
};

template <int kSrc>
__device__ __forceinline__ double2 pass_load(const PassIo& io, int64_t b, int i) {
    const double2* in = io.in + b * N;
    if (kSrc == kRf) {
        const int64_t n = b * kStride + i;
        return make_double2(io.rf32 ? (double)io.rf32[n] : (double)io.rf[n], 0.0);
    }
    if (kSrc == kReal) return make_double2(io.real[b * N + i], 0.0);
    if (kSrc == kAnalytic) {
        // analytic spectrum: X * RfVideo * Hilbert / N  (bins > N/2 zero)
        if (i > H) return make_double2(0.0, 0.0);
        const double m = i == 0 || i == H ? io.gain[i] / N : 2.0 * io.gain[i] / N;
        return make_double2(in[i].x * m, in[i].y * m);
    }
    if (kSrc == kFilter) {
        // Hermitian spectrum D * Hfilter for bins 0..N/2 (imaginary parts of the
        // DC and Nyquist bins dropped, as a c2r inverse does), mirrored above
        // N/2, scaled 1/N
        const int kk = i <= H ? i : N - i;
        double2 v = cmul(in[kk], io.h[kk]);
        if (kk == 0 || kk == H) v.y = 0.0;
        if (i > H) v.y = -v.y;
        return make_double2(v.x / N, v.y / N);
    }
    if (kSrc == kSub) {
        // sub-deemphasis (ApplySubDeemphasisRealCore, Core/Dsp/RfDemodulator.cs:2852-2990),
        // step 1: one-sided spectrum whose inverse is the analytic signal of
        // high = irfft(D Video HighPass): x2 for 0 < k < N/2, real part at 0 and
        // N/2 (what a c2r inverse keeps), zero above; scaled 1/N
        if (i > H) return make_double2(0.0, 0.0);
        const double2 v = cmul(in[i], io.h[i]);
        if (i == 0 || i == H) return make_double2(v.x / N, 0.0);
        return make_double2(2.0 * v.x / N, 2.0 * v.y / N);
    }
    return in[i];
}

// Stockham radix-8 pass of block blockIdx.y, L = N, Ns in {1, 8, 64, 512, 4096}.
template <bool INV, int kSrc, int kDst>
__global__ void __launch_bounds__(128) k_pass8(PassIo io, const double2* __restrict__ tw, int Ns) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t b = blockIdx.y;
    const int R = 8;
    const int nbf = N / R;
    if (j >= nbf) return;
    int k = j & (Ns - 1);
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = pass_load<kSrc>(io, b, j + r * nbf);
    if (kSrc == kPlainSrc) {   // a first pass has no twiddles
#pragma unroll
        for (int r = 1; r < R; r++) {
            double2 w = tw[(k * r * (N / (Ns * R))) & (N - 1)];
            if (INV) w.y = -w.y;
            v[r] = cmul(v[r], w);
        }
    }
    dft<R, INV>(v);
    int dst = (j - k) * R + k;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = dst + r * Ns;
        if (kDst == kPlainDst) io.out[b * N + i] = v[r];
        // the last pass: i = j + r N / 8
        if (kDst == kHalfDst && (r < R / 2 || (r == R / 2 && j == 0))) io.out[b * N + i] = v[r];
        if (kDst == kRealDst) io.real_out[b * N + i] = v[r].x;
        if (kDst == kStreamDst) {
            const int s = i - kCut - io.shift;
            if (s >= 0 && s < kStride) io.real_out[b * kStride + s] = v[r].x;
        }
    }
}

// One transform of `nb` blocks: first pass from io's source, x and y in turn,
// the last pass to io's destination (the complex result, if any, in y).
template <bool INV, int kSrc, int kDst>
void fft(PassIo io, double2* x, double2* y, const double2* tw, int nb, cudaStream_t s) {
    const dim3 grid(N / 8 / 128, nb);
    PassIo p = io;
    p.out = y;
    k_pass8<INV, kSrc, kPlainDst><<<grid, 128, 0, s>>>(p, tw, 1);
    p.in = y; p.out = x;
    k_pass8<INV, kPlainSrc, kPlainDst><<<grid, 128, 0, s>>>(p, tw, 8);
    p.in = x; p.out = y;
    k_pass8<INV, kPlainSrc, kPlainDst><<<grid, 128, 0, s>>>(p, tw, 64);
    p.in = y; p.out = x;
    k_pass8<INV, kPlainSrc, kPlainDst><<<grid, 128, 0, s>>>(p, tw, 512);
    p.in = x; p.out = y;
    k_pass8<INV, kPlainSrc, kDst><<<grid, 128, 0, s>>>(p, tw, 4096);
}

// demod (float polynomial atan2 of the double analytic signal), the block's
// spike flag and its spike mask (d > diff_max; a warp holds 32 consecutive n)
__global__ void k_demod(const double2* z, double* d, float fs, double diff_max, int* flag, unsigned* mask) {
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t b = blockIdx.y;
    z += b * N;
    double v = 0.0;
    if (n > 0) {
        float th = vhs_atan2((float)z[n].y, (float)z[n].x);
        float tp = vhs_atan2((float)z[n - 1].y, (float)z[n - 1].x);
        v = (double)vhs_freq_diff(th, tp, fs);
    }
    d[b * N + n] = v;
    const unsigned m = __ballot_sync(0xffffffffu, v > diff_max);
    if ((n & 31) == 0) mask[b * (N / 32) + (n >> 5)] = m;
    if (n >= 20 && n < N - 20 && v > diff_max) atomicOr(flag + b, 1);
}

// diff demod (analytic first difference), only when the block has spikes
__global__ void k_diff_demod(const double2* z, double* dd, float fs, const int* flag) {
    const int64_t blk = blockIdx.y;
    if (!flag[blk]) return;
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    z += blk * N;
    dd += blk * N;
    double v = 0.0;
    if (n >= 1) {
        double2 a = z[n], b = z[n - 1];
        float th = vhs_atan2((float)(a.y - b.y), (float)(a.x - b.x));
        float tp;
        if (n >= 2) {
            double2 c = z[n - 2];
            tp = vhs_atan2((float)(b.y - c.y), (float)(b.x - c.x));
        } else {
            tp = vhs_atan2(0.0f, 0.0f);
        }
        v = (double)vhs_freq_diff(th, tp, fs);
    }
    dd[n] = v;
}

// ReplaceSpikes (Core/Dsp/RfDemodulator.cs:966-1001) on one warp, spike set
// taken from the demod before replacement.
__global__ void __launch_bounds__(32) k_replace_spikes(double* d, const double* dd, int* flag,
                                                       const unsigned* mask) {
    const int64_t blk = blockIdx.x;
    if (!flag[blk]) return;
    d += blk * N;
    dd += blk * N;
    mask += blk * (N / 32);
    int lane = threadIdx.x;
    for (int base = 0; base < N / 32; base += 32) {
        const unsigned mine = mask[base + lane];
        unsigned words = __ballot_sync(0xffffffffu, mine != 0u);
        while (words) {
            const int w = __ffs(words) - 1;
            words &= words - 1;
            unsigned m = __shfl_sync(0xffffffffu, mine, w);
            while (m) {
                int b = __ffs(m) - 1;
                m &= m - 1;
                int i0 = (base + w) * 32 + b;
                int st = max(i0 - 8, 0), en = min(i0 + 30, N - 1);
                if (st >= en) continue;
                double mdd = -INFINITY, md = -INFINITY;
                for (int k = st + lane; k < en; k += 32) { mdd = fmax(mdd, dd[k]); md = fmax(md, d[k]); }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    mdd = fmax(mdd, __shfl_xor_sync(0xffffffffu, mdd, o));
                    md = fmax(md, __shfl_xor_sync(0xffffffffu, md, o));
                }
                if (mdd < md) for (int k = st + lane; k < en; k += 32) d[k] = dd[k];
                __syncwarp();
            }
        }
    }
    if (lane == 0) flag[blk] = 0;
}

// float32 envelope filtfilt (SosFilter.ApplyForwardBackwardFloat32,
// Core/Dsp/SosFilter.cs:300-540) of raw[n] = |float(Re z[n-4])| (circular
// roll by 4), in float32 like the reference, as a parallel scan: one CTA of
// 32 warps, warp w covers samples [1024 w, 1024 w + 1024) as four rows of 256
// (8 consecutive samples per lane, lanes joined by an affine warp scan).  The
// state entering a warp's range comes from a 256-sample halo started at zero
// (the first-order filter's memory c^256 is below 1e-12); at the block edges
// the recursion starts from zero instead of the reference's padded
// steady-state start, which only touches samples the overlap-save cut drops.
struct EnvAff { float a, b; };
__device__ __forceinline__ EnvAff env_then(EnvAff first, EnvAff second) {
    return EnvAff{second.a * first.a, fmaf(second.a, first.b, second.b)};
}
__device__ __forceinline__ EnvAff env_scan(EnvAff v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float pa = __shfl_up_sync(0xffffffffu, v.a, o), pb = __shfl_up_sync(0xffffffffu, v.b, o);
        if (lane >= o) v = env_then(EnvAff{pa, pb}, v);
    }
    return v;
}
__device__ __forceinline__ EnvAff env_scan_rev(EnvAff v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float pa = __shfl_down_sync(0xffffffffu, v.a, o), pb = __shfl_down_sync(0xffffffffu, v.b, o);
        if (lane + o < 32) v = env_then(EnvAff{pa, pb}, v);
    }
    return v;
}

// The kept samples go to the stitched stream (rows lie wholly inside or
// outside the kept range).
__global__ void __launch_bounds__(1024) k_envelope(const double2* z, float* work, double* env, float b0,
                                                   float b1, float a1) {
    z += (int64_t)blockIdx.x * N;
    work += (int64_t)blockIdx.x * N;
    env += (int64_t)blockIdx.x * kStride - kCut;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = warp * 1024;
    const float cc = -a1, gk = b1 - a1 * b0;
    float c8 = cc;
#pragma unroll
    for (int k = 1; k < 8; k++) c8 *= cc;
    auto raw = [&](int n) { return fabsf((float)z[(n - 4) & (N - 1)].x); };
    float yv[32];
    float carry = 0.0f;
    if (n0 >= 256) {
        float st = 0.0f;
        for (int k = 0; k < 8; k++) st = fmaf(cc, st, gk * raw(n0 - 256 + lane * 8 + k));
        EnvAff inc = env_scan(EnvAff{c8, st}, lane);
        carry = __shfl_sync(0xffffffffu, inc.b, 31);
    }
    for (int row = 0; row < 4; row++) {
        int ms = n0 + row * 256 + lane * 8;
        float ev[8], st = 0.0f;
        for (int k = 0; k < 8; k++) { ev[k] = raw(ms + k); st = fmaf(cc, st, gk * ev[k]); }
        EnvAff inc = env_scan(EnvAff{c8, st}, lane);
        float pb = __shfl_up_sync(0xffffffffu, inc.b, 1), pa = __shfl_up_sync(0xffffffffu, inc.a, 1);
        float zz = lane == 0 ? carry : fmaf(pa, carry, pb);
        for (int k = 0; k < 8; k++) { yv[row * 8 + k] = fmaf(b0, ev[k], zz); zz = fmaf(cc, zz, gk * ev[k]); }
        carry = __shfl_sync(0xffffffffu, zz, 31);
        for (int k = 0; k < 8; k++) work[ms + k] = yv[row * 8 + k];
    }
    __syncthreads();
    const int nend = n0 + 1024;
    carry = 0.0f;
    if (nend + 256 <= N) {
        float st = 0.0f;
        for (int k = 7; k >= 0; k--) st = fmaf(cc, st, gk * work[nend + lane * 8 + k]);
        EnvAff inc = env_scan_rev(EnvAff{c8, st}, lane);
        carry = __shfl_sync(0xffffffffu, inc.b, 0);
    }
    for (int row = 3; row >= 0; row--) {
        int ms = n0 + row * 256 + lane * 8;
        float st = 0.0f;
        for (int k = 7; k >= 0; k--) st = fmaf(cc, st, gk * yv[row * 8 + k]);
        EnvAff inc = env_scan_rev(EnvAff{c8, st}, lane);
        float nb = __shfl_down_sync(0xffffffffu, inc.b, 1), na = __shfl_down_sync(0xffffffffu, inc.a, 1);
        float zz = lane == 31 ? carry : fmaf(na, carry, nb);
        for (int k = 7; k >= 0; k--) {
            float y = yv[row * 8 + k];
            if (ms >= kCut && ms < kCut + kStride) env[ms + k] = (double)fmaf(b0, y, zz);
            zz = fmaf(cc, zz, gk * y);
        }
        carry = __shfl_sync(0xffffffffu, zz, 0);
    }
}

struct Aff64 { double a, b; };
__device__ __forceinline__ Aff64 aff64_then(Aff64 first, Aff64 second) {
    return Aff64{second.a * first.a, fma(second.a, first.b, second.b)};
}
__device__ __forceinline__ Aff64 aff64_scan(Aff64 v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        double pa = __shfl_up_sync(0xffffffffu, v.a, o), pb = __shfl_up_sync(0xffffffffu, v.b, o);
        if (lane >= o) v = aff64_then(Aff64{pa, pb}, v);
    }
    return v;
}
__device__ __forceinline__ Aff64 aff64_scan_rev(Aff64 v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        double pa = __shfl_down_sync(0xffffffffu, v.a, o), pb = __shfl_down_sync(0xffffffffu, v.b, o);
        if (lane + o < 32) v = aff64_then(Aff64{pa, pb}, v);
    }
    return v;
}

__device__ __forceinline__ double sub_gain64(double amp, const SubDeemph64& s) {
    amp = fmax(0.0, amp) * s.scale1;
    amp = pow(amp, s.exponent) * s.scale2;
    if (s.logistic_rate > 0.0) amp *= 1.0 / (1.0 + exp(-s.logistic_rate * (amp - s.logistic_mid)));
    return amp;
}

// Sub-deemphasis step 2: amp[n] = |a[n]| * 2 / deviation.
__global__ void k_sub_mag(const double2* a, double* amp, SubDeemph64 sub) {
    int64_t n = blockIdx.x * blockDim.x + threadIdx.x + (int64_t)blockIdx.y * N;
    amp[n] = hypot(a[n].x, a[n].y) * sub.inv_half_dev;
}

// Steps 3-4: first-order low-pass filtfilt of amp in binary64, one warp (one
// CTA) per 1024-sample range, 32 ranges per block: the range is four rows of
// 256 (8 consecutive samples per lane) joined by affine warp scans, and the
// state entering it comes from the 1024 samples before it (after it, backward)
// started at zero, where the filter's memory c^1024 is below 1e-40; at the
// block edges the recursion starts from zero instead of the padded
// steady-state start, which only moves samples the overlap-save cut drops.
// Forward: amp -> fwd.  Backward: fwd -> out.
template <bool BACKWARD>
__global__ void __launch_bounds__(32) k_sub_filt(const double* in, double* out, SubDeemph64 sub) {
    const int lane = threadIdx.x;
    const int n0 = blockIdx.x * 1024;
    in += (int64_t)blockIdx.y * N;
    out += (int64_t)blockIdx.y * N;
    const double cc = -sub.a1, gk = sub.b1 - sub.a1 * sub.b0, b0 = sub.b0;
    double c8 = cc;
#pragma unroll
    for (int k = 1; k < 8; k++) c8 *= cc;
    double carry = 0.0;
    if (!BACKWARD) {
        if (n0 >= 1024) {
            for (int hr = 0; hr < 4; hr++) {
                int ms = n0 - 1024 + hr * 256 + lane * 8;
                double ev[8], st = 0.0;
                for (int k = 0; k < 8; k++) { ev[k] = in[ms + k]; st = fma(cc, st, gk * ev[k]); }
                Aff64 inc = aff64_scan(Aff64{c8, st}, lane);
                double pb = __shfl_up_sync(0xffffffffu, inc.b, 1), pa = __shfl_up_sync(0xffffffffu, inc.a, 1);
                double z = lane == 0 ? carry : fma(pa, carry, pb);
                for (int k = 0; k < 8; k++) z = fma(cc, z, gk * ev[k]);
                carry = __shfl_sync(0xffffffffu, z, 31);
            }
        }
        for (int row = 0; row < 4; row++) {
            int ms = n0 + row * 256 + lane * 8;
            double ev[8], st = 0.0;
            for (int k = 0; k < 8; k++) { ev[k] = in[ms + k]; st = fma(cc, st, gk * ev[k]); }
            Aff64 inc = aff64_scan(Aff64{c8, st}, lane);
            double pb = __shfl_up_sync(0xffffffffu, inc.b, 1), pa = __shfl_up_sync(0xffffffffu, inc.a, 1);
            double z = lane == 0 ? carry : fma(pa, carry, pb);
            for (int k = 0; k < 8; k++) { out[ms + k] = fma(b0, ev[k], z); z = fma(cc, z, gk * ev[k]); }
            carry = __shfl_sync(0xffffffffu, z, 31);
        }
    } else {
        const int nend = n0 + 1024;
        if (nend + 1024 <= N) {
            for (int hr = 3; hr >= 0; hr--) {
                int ms = nend + hr * 256 + lane * 8;
                double ev[8], st = 0.0;
                for (int k = 7; k >= 0; k--) { ev[k] = in[ms + k]; st = fma(cc, st, gk * ev[k]); }
                Aff64 inc = aff64_scan_rev(Aff64{c8, st}, lane);
                double nb = __shfl_down_sync(0xffffffffu, inc.b, 1), na = __shfl_down_sync(0xffffffffu, inc.a, 1);
                double z = lane == 31 ? carry : fma(na, carry, nb);
                for (int k = 7; k >= 0; k--) z = fma(cc, z, gk * ev[k]);
                carry = __shfl_sync(0xffffffffu, z, 0);
            }
        }
        for (int row = 3; row >= 0; row--) {
            int ms = n0 + row * 256 + lane * 8;
            double ev[8], st = 0.0;
            for (int k = 7; k >= 0; k--) { ev[k] = in[ms + k]; st = fma(cc, st, gk * ev[k]); }
            Aff64 inc = aff64_scan_rev(Aff64{c8, st}, lane);
            double nb = __shfl_down_sync(0xffffffffu, inc.b, 1), na = __shfl_down_sync(0xffffffffu, inc.a, 1);
            double z = lane == 31 ? carry : fma(na, carry, nb);
            for (int k = 7; k >= 0; k--) { out[ms + k] = fma(b0, ev[k], z); z = fma(cc, z, gk * ev[k]); }
            carry = __shfl_sync(0xffffffffu, z, 0);
        }
    }
}

// Step 5, elementwise, into the stitched stream: video[n] - (Re a[n] (1 - map(amp[n])) + Re a[n] static_factor).
__global__ void k_sub_apply(const double2* a, const double* amp, const double* video, double* out, SubDeemph64 sub) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= kStride) return;
    const int64_t n = (int64_t)blockIdx.y * N + s + kCut;
    double h = a[n].x;
    double g = sub_gain64(amp[n], sub);
    double v = video[n];
    v -= h * (1.0 - g) + h * sub.static_factor;
    out[(int64_t)blockIdx.y * kStride + s] = v;
}

}  // namespace fp64

cudaError_t make_fp64_twiddles(double2* tw, cudaStream_t s) {
    fp64::k_twiddles<<<fp64::N / 256, 256, 0, s>>>(tw);
    return cudaGetLastError();
}

cudaError_t launch_demod_fp64(const PlainDemodParams& p, cudaStream_t s) {
    using namespace fp64;
    const int nb = p.nblocks;
    if (nb <= 0) return cudaSuccess;
    if (nb > 65535) return cudaErrorInvalidValue;
    const dim3 every(N / 256, nb), kept((kStride + 255) / 256, nb);
    const size_t all = (size_t)nb * N;
    double2* w0 = p.work;
    double2* w1 = p.work + all;
    double2* w2 = p.work + 2 * all;
    double* d = p.dwork;
    double* dd = p.dwork + all;
    double* video = p.dwork + 2 * all;
    const int64_t first = p.first_block * kStride;
    PassIo io{};
    io.rf = p.rf ? p.rf + first : nullptr;
    io.rf32 = p.rf_f32 ? p.rf_f32 + first : nullptr;
    fft<false, kRf, kHalfDst>(io, w1, w0, p.twiddle, nb, s);           // X in w0
    io.in = w0;
    io.gain = p.rf_video;
    fft<true, kAnalytic, kPlainDst>(io, w2, w1, p.twiddle, nb, s);     // z in w1
    k_demod<<<every, 256, 0, s>>>(w1, d, (float)p.fs, p.diff_max, p.flag, p.mask);
    k_diff_demod<<<every, 256, 0, s>>>(w1, dd, (float)p.fs, p.flag);
    k_replace_spikes<<<nb, 32, 0, s>>>(d, dd, p.flag, p.mask);
    k_envelope<<<nb, 1024, 0, s>>>(w1, p.fwork, p.env_out + first, (float)p.env_b0, (float)p.env_b1, (float)p.env_a1);
    io.real = d;
    fft<false, kReal, kHalfDst>(io, w1, w0, p.twiddle, nb, s);         // D in w0
    io.h = p.video;
    io.real_out = p.sub.high ? video : p.video_out + first;
    if (p.sub.high) fft<true, kFilter, kRealDst>(io, w2, w1, p.twiddle, nb, s);
    else fft<true, kFilter, kStreamDst>(io, w2, w1, p.twiddle, nb, s);
    if (p.sub.high) {
        io.h = p.sub.high;
        fft<true, kSub, kPlainDst>(io, w2, w1, p.twiddle, nb, s);      // analytic high part in w1
        k_sub_mag<<<every, 256, 0, s>>>(w1, dd, p.sub);
        k_sub_filt<false><<<dim3(N / 1024, nb), 32, 0, s>>>(dd, d, p.sub);
        k_sub_filt<true><<<dim3(N / 1024, nb), 32, 0, s>>>(d, dd, p.sub);
        k_sub_apply<<<kept, 256, 0, s>>>(w1, dd, video, p.video_out + first, p.sub);
    }
    io.h = p.sync;
    io.real_out = p.sync_out + first;
    io.shift = 32;
    fft<true, kFilter, kStreamDst>(io, w2, w1, p.twiddle, nb, s);
    return cudaGetLastError();
}

}  // namespace vhsd
