// Low-pass filtering of trace planes for the multiscale misfit
// (lowpass / adj_lowpass, PyFWI src/PyFWI/fwi_tools.py:1188-1258, applied by
// cost_preparation / adj_cost_preparation, :1153-1273).
//
// The reference pads every trace with 512 zeros, takes its FFT, multiplies
// it by h and by conj(h) (h the frequency response of a Butterworth design)
// and keeps the first nt samples of the real inverse FFT; its "adjoint"
// applies conj(h) and h, the same product.  Along time that is the
// symmetric Toeplitz operator y[t] = sum_s g[|t - s|] x[s] (t, s < nt), g the
// real inverse FFT of conj(h) h on nt + 512 points.  Embedded in a circulant
// of nfft >= 2 nt - 1 points (a power of two) the operator is diagonal in
// Fourier space with a real spectrum C (the response is real and even), so
// each trace is filtered by one forward FFT, a product with C and one inverse
// FFT.  The host builds C (with the 1/nfft of the inverse folded in) and the
// twiddle table once per cutoff.
//
// A CTA filters up to four pairs of adjacent traces of one plane: trace 2p goes
// in the real part and trace 2p+1 in the imaginary part of one complex
// signal (C is real and even, so the two stay apart).  A signal is transformed
// in one to four passes of radix 2 to 16.  In a pass a thread holds the points
// of a butterfly in registers; between passes they lie in shared memory, each
// pass in place: decimation in frequency from samples read from memory to a
// digit-reversed spectrum, the product with C in the last pass's registers, and
// the same passes backwards (conjugate twiddles) to the first nt samples, which
// go straight to memory.  FP32 arithmetic throughout.
//
// What bounds it: a radix-2 transform (24 sweeps over shared memory for 4096
// points, a barrier each) took 842 us for 8000 traces of 2000 samples, 20 us of
// which are the memory traffic; four sweeps are left here, and it takes 117 us.
#include "pyfwi_b200.h"

#include <cuda_runtime.h>

#include <cstdint>

void pyfwi_set_error(const char *msg);

namespace {

constexpr int MAX_LOGN = 14;
// Threads of a CTA: from 4096 points on the signals of one CTA fill an SM, and 512 threads keep it busier (119 us
// against 134 for 8000 traces of 2000 samples); below, more CTAs do (50 against 53 us for 8000 of 1000).
__host__ __device__ constexpr int fft_threads(int l) { return l < 12 ? 256 : 512; }

int fail(int code, const char *msg)
{
    pyfwi_set_error(msg);
    return code;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ float2 cmulc(float2 a, float2 b)  // a * conj(b)
{
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// Passes of a transform of 2^l points and the radix (as a power of two) of each.
__host__ __device__ constexpr int n_pass(int l) { return (l + 3) / 4; }
__host__ __device__ constexpr int pass_bits(int l, int i) { return l / n_pass(l) + (i < l % n_pass(l)); }
__host__ __device__ constexpr int bits_before(int l, int i) { return i == 0 ? 0 : bits_before(l, i - 1) + pass_bits(l, i - 1); }

// Place of point p of a signal: one free place after every 16 and every 256
// points, so that neither contiguous butterflies nor strided ones share banks.
__host__ __device__ constexpr int place(int p) { return p + (p >> 4) + (p >> 8); }
// Places of a signal; the pairs' samples are read and written together, so the
// signals start 16 / pairs places apart modulo the 16 float2 of the banks.
__host__ __device__ constexpr int signal_places(int n, int pairs) { return (place(n) + 15) / 16 * 16 + 16 / pairs % 16; }

// a * exp(-+ i pi / 2)
template <bool INV>
__device__ __forceinline__ float2 quarter(float2 a) { return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x); }

template <bool INV>
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d)
{
    const float2 s = a + c, t = a - c, u = b + d, v = quarter<INV>(b - d);
    a = s + u;
    b = t + v;
    c = s - u;
    d = t - v;
}

// Discrete Fourier transform of 2^B points in registers, in and out in natural
// order: for 8 and 16, transforms of four over the points of each residue, the
// twiddles between, and transforms over the residues.
template <int B, bool INV>
__device__ __forceinline__ void dft(float2 (&x)[1 << B])
{
    if constexpr (B == 1) {
        const float2 a = x[0];
        x[0] = a + x[1];
        x[1] = a - x[1];
    } else if constexpr (B == 2) {
        dft4<INV>(x[0], x[1], x[2], x[3]);
    } else {
        constexpr float C1 = 0.923879532511286756f, S1 = 0.382683432365089772f, H = 0.707106781186547524f;  // cos, sin pi / 8; sqrt 1/2
        constexpr int NB = 1 << (B - 2);
#pragma unroll
        for (int b = 0; b < NB; ++b) dft4<INV>(x[b], x[NB + b], x[2 * NB + b], x[3 * NB + b]);
        // x[NB c + b] times exp(-+ 2 pi i b c / 2^B)
        auto turn = [](float2 v, float c, float s) { return INV ? cmulc(v, make_float2(c, -s)) : cmul(v, make_float2(c, -s)); };
        constexpr int U = B == 4 ? 1 : 2;  // sixteenths of a turn per b c
#pragma unroll
        for (int b = 1; b < NB; ++b)
#pragma unroll
            for (int c = 1; c < 4; ++c) {
                float2 &v = x[NB * c + b];
                switch (U * b * c) {
                    case 1: v = turn(v, C1, S1); break;
                    case 2: v = turn(v, H, H); break;
                    case 3: v = turn(v, S1, C1); break;
                    case 4: v = quarter<INV>(v); break;
                    case 6: v = turn(v, -H, H); break;
                    case 9: v = turn(v, -C1, -S1); break;
                }
            }
        float2 y[1 << B];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float2 r[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) r[b] = x[NB * c + b];
            dft<B - 2, INV>(r);
#pragma unroll
            for (int d = 0; d < NB; ++d) y[c + 4 * d] = r[d];
        }
#pragma unroll
        for (int k = 0; k < (1 << B); ++k) x[k] = y[k];
    }
}

// exp(-2 pi i k / N) from the table of the first half turn.
template <int LOGN>
__device__ __forceinline__ float2 root(const float2 *tw, int k)
{
    constexpr int HALF = 1 << (LOGN - 1);
    const float2 w = __ldg(tw + (k & (HALF - 1)));
    return k & HALF ? make_float2(-w.x, -w.y) : w;
}

// Points k > 0 times at(k) or its conjugate.  Each factor is a table value: products of fewer of them cost
// accuracy (1.50e-7 against 1.39e-7 for 2000 samples).
template <int B, bool INV, class At>
__device__ __forceinline__ void twiddle(float2 (&x)[1 << B], At at)
{
#pragma unroll
    for (int k = 1; k < (1 << B); ++k) x[k] = INV ? cmulc(x[k], at(k)) : cmul(x[k], at(k));
}

// Places of the twiddles of the passes between the first and pass i.
__host__ __device__ constexpr int roots_before(int l, int i)
{
    return i <= 1 ? 0 : roots_before(l, i - 1) + (1 << (l - bits_before(l, i - 1)));
}

// filter: [0, nfft) the real spectrum C, then nfft/2 twiddles
// exp(-2 pi i j / nfft) as (cos, sin) pairs.
template <int LOGN>
struct Transform {
    static constexpr int N = 1 << LOGN;
    float2 *sig;
    int pairs, places;
    const float *spec;
    const float2 *tw;
    float2 *roots;  // [middle pass][k][j]: its twiddles, read without conflicts by consecutive threads

    template <int I>
    __device__ __forceinline__ void fill() const
    {
        if constexpr (I < n_pass(LOGN) - 1) {
            constexpr int LM = LOGN - bits_before(LOGN, I), SUB = 1 << (LM - pass_bits(LOGN, I));
            for (int e = threadIdx.x; e < 1 << LM; e += fft_threads(LOGN))
                roots[roots_before(LOGN, I) + e] = root<LOGN>(tw, ((e / SUB) * (e % SUB)) << (LOGN - LM));
            fill<I + 1>();
        }
    }

    // A pass between the first and the last, in shared memory.
    template <int I, bool INV>
    __device__ __forceinline__ void middle() const
    {
        constexpr int B = pass_bits(LOGN, I), r = 1 << B, LM = LOGN - bits_before(LOGN, I), SUB = 1 << (LM - B);
        for (int e = threadIdx.x; e < pairs * (N / r); e += fft_threads(LOGN)) {
            const int p = e / (N / r), q = e % (N / r), j = q % SUB, o = (q / SUB << LM) + j;
            float2 *s = sig + p * places;
            float2 x[r];
#pragma unroll
            for (int m = 0; m < r; ++m) x[m] = s[place(o + m * SUB)];
            auto at = [&](int k) { return roots[roots_before(LOGN, I) + k * SUB + j]; };
            if (INV) twiddle<B, true>(x, at);
            dft<B, INV>(x);
            if (!INV) twiddle<B, false>(x, at);
#pragma unroll
            for (int m = 0; m < r; ++m) s[place(o + m * SUB)] = x[m];
        }
        __syncthreads();
    }

    // The last forward pass, the filter and the first inverse pass of r points: the spectrum's points f0 + k N / r.
    template <int B>
    __device__ __forceinline__ void filter(float2 (&x)[1 << B], int f0) const
    {
        dft<B, false>(x);
#pragma unroll
        for (int k = 0; k < (1 << B); ++k) {
            const float c = __ldg(spec + f0 + k * (N >> B));
            x[k] = make_float2(x[k].x * c, x[k].y * c);
        }
        dft<B, true>(x);
    }

    __device__ __forceinline__ void last() const
    {
        constexpr int NP = n_pass(LOGN), B = pass_bits(LOGN, NP - 1), r = 1 << B;
        // consecutive threads take consecutive frequencies
        for (int e = threadIdx.x; e < pairs * (N / r); e += fft_threads(LOGN)) {
            const int p = e / (N / r), f0 = e % (N / r);
            int o = 0;  // its digits the other way round
#pragma unroll
            for (int i = 0; i < NP - 1; ++i)
                o = o << pass_bits(LOGN, i) | (f0 >> bits_before(LOGN, i) & ((1 << pass_bits(LOGN, i)) - 1));
            float2 *s = sig + p * places;
            float2 x[r];
#pragma unroll
            for (int m = 0; m < r; ++m) x[m] = s[place(o * r + m)];
            filter<B>(x, f0);
#pragma unroll
            for (int m = 0; m < r; ++m) s[place(o * r + m)] = x[m];
        }
        __syncthreads();
    }

    template <int I>
    __device__ __forceinline__ void inside() const
    {
        if constexpr (I < n_pass(LOGN) - 1) {
            middle<I, false>();
            inside<I + 1>();
            middle<I, true>();
        } else {
            last();
        }
    }
};

// VEC: two adjacent traces are one aligned float2.
template <int LOGN, bool VEC>
__global__ void __launch_bounds__(fft_threads(LOGN)) lowpass_fft_kernel(const float *filter, int pairs, const float *in,
                                                                      float *out, int nt, long long ncols)
{
    extern __shared__ float2 sig[];
    constexpr int N = 1 << LOGN, NP = n_pass(LOGN), B = pass_bits(LOGN, 0), r = 1 << B, SUB = N / r;
    const Transform<LOGN> T{sig, pairs, signal_places(N, pairs), filter,
                            reinterpret_cast<const float2 *>(filter + N), sig + pairs * signal_places(N, pairs)};
    const long long plane = (long long)nt * ncols, c0 = (long long)blockIdx.x * 2 * pairs;
    const float *src = in + blockIdx.y * plane;
    float *dst = out + blockIdx.y * plane;

    auto load = [&](float2 (&x)[r], int j, long long c) {
#pragma unroll
        for (int m = 0; m < r; ++m) {
            const int t = j + m * SUB;
            x[m] = make_float2(0.f, 0.f);
            if ((m < r / 2 || r == 2) && t < nt) {  // 2 nt - 1 <= N: the upper half is zero
                const float *v = src + (long long)t * ncols + c;
                if (VEC) {
                    x[m] = __ldg(reinterpret_cast<const float2 *>(v));
                } else {
                    x[m].x = __ldg(v);
                    if (c + 1 < ncols) x[m].y = __ldg(v + 1);
                }
            }
        }
    };
    auto store = [&](const float2 (&x)[r], int j, long long c) {
#pragma unroll
        for (int m = 0; m < r; ++m) {
            const int t = j + m * SUB;
            if ((m < r / 2 || r == 2) && t < nt) {
                float *v = dst + (long long)t * ncols + c;
                if (VEC) {
                    *reinterpret_cast<float2 *>(v) = x[m];
                } else {
                    v[0] = x[m].x;
                    if (c + 1 < ncols) v[1] = x[m].y;
                }
            }
        }
    };
    if constexpr (NP > 2) T.template fill<1>();
    // consecutive threads take consecutive pairs of a row
    for (int e = threadIdx.x; e < pairs * SUB; e += fft_threads(LOGN)) {
        const int p = e % pairs, j = e / pairs;
        const long long c = c0 + 2 * p;
        float2 x[r];
        if (c < ncols)
            load(x, j, c);
        else
#pragma unroll
            for (int m = 0; m < r; ++m) x[m] = make_float2(0.f, 0.f);
        if constexpr (NP == 1) {
            T.template filter<B>(x, 0);
            if (c < ncols) store(x, j, c);
        } else {
            dft<B, false>(x);
            twiddle<B, false>(x, [&](int k) { return root<LOGN>(T.tw, k * j); });
            float2 *s = sig + p * T.places;
#pragma unroll
            for (int m = 0; m < r; ++m) s[place(j + m * SUB)] = x[m];
        }
    }
    if constexpr (NP > 1) {
        __syncthreads();
        T.template inside<1>();
        for (int e = threadIdx.x; e < pairs * SUB; e += fft_threads(LOGN)) {
            const int p = e % pairs, j = e / pairs;
            const long long c = c0 + 2 * p;
            if (c >= ncols) continue;
            const float2 *s = sig + p * T.places;
            float2 x[r];
#pragma unroll
            for (int m = 0; m < r; ++m) x[m] = s[place(j + m * SUB)];
            twiddle<B, true>(x, [&](int k) { return root<LOGN>(T.tw, k * j); });
            dft<B, true>(x);
            store(x, j, c);
        }
    }
}

struct Job {
    const float *filter, *in;
    float *out;
    int nt;
    long long ncols;
    int planes;
    cudaStream_t stream;
};

template <int LOGN>
cudaError_t launch(const Job &a, int nfft)
{
    if (nfft != 1 << LOGN) {
        if constexpr (LOGN < MAX_LOGN)
            return launch<LOGN + 1>(a, nfft);
        else
            return cudaErrorInvalidValue;
    } else {
        // four pairs of traces fill a 32-byte sector of a row; as many as fit in shared memory
        constexpr int pairs = LOGN <= 12 ? 4 : LOGN == 13 ? 2 : 1;
        const long long ctas = (a.ncols + 2 * pairs - 1) / (2 * pairs);
        if (ctas > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
        const size_t places = (size_t)pairs * signal_places(nfft, pairs) + roots_before(LOGN, n_pass(LOGN) - 1);
        const size_t smem = n_pass(LOGN) == 1 ? 0 : places * sizeof(float2);
        const bool vec = a.ncols % 2 == 0 && reinterpret_cast<uintptr_t>(a.in) % 8 == 0 &&
                         reinterpret_cast<uintptr_t>(a.out) % 8 == 0;
        auto kern = vec ? lowpass_fft_kernel<LOGN, true> : lowpass_fft_kernel<LOGN, false>;
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<dim3((unsigned)ctas, (unsigned)a.planes), fft_threads(LOGN), smem, a.stream>>>(a.filter, pairs, a.in, a.out,
                                                                                         a.nt, a.ncols);
        return cudaGetLastError();
    }
}

}  // namespace

extern "C" int pyfwi_lowpass(const float *filter, int32_t nfft, const float *in, float *out, int32_t nt,
                             int64_t ncols, int32_t n_planes, void *stream)
{
    if (!filter || !in || !out || nt < 1 || ncols < 0 || n_planes < 0)
        return fail(PYFWI_E_INVALID, "pyfwi_lowpass: bad argument");
    if (nfft < 2 || (nfft & (nfft - 1)) || nfft > 1 << MAX_LOGN || nfft < 2 * nt - 1)
        return fail(PYFWI_E_INVALID, "pyfwi_lowpass: nfft must be a power of two with 2*nt - 1 <= nfft <= 16384");
    const long long plane = (long long)nt * ncols;
    if (out < in + plane * n_planes && in < out + plane * n_planes)
        return fail(PYFWI_E_INVALID, "pyfwi_lowpass: in and out overlap");
    if (ncols == 0 || n_planes == 0) return PYFWI_OK;
    if (n_planes > 65535) return fail(PYFWI_E_INVALID, "pyfwi_lowpass: more than 65535 planes");
    const long long ctas = (ncols + 1) / 2;  // at most
    if (ctas > 0x7fffffffLL) return fail(PYFWI_E_INVALID, "pyfwi_lowpass: too many traces per plane");
    const cudaError_t e = launch<1>({filter, in, out, nt, ncols, n_planes, static_cast<cudaStream_t>(stream)}, nfft);
    if (e != cudaSuccess) return fail(PYFWI_E_CUDA, cudaGetErrorString(e));
    return PYFWI_OK;
}
