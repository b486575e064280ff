// ktm_prep.cu -- trace preparation on the device: the rho (half-derivative)
// pre-filter of scripts/ktmApplyRhoFilter.m, the sqrt(t) weight fold, per-trace
// scaling, FP16/BF16 quantisation and packing for the fast migration kernel.
//
// With the rho filter on, a PAIR of real traces x and y goes through ONE complex FFT as
// z = x + i y: every rho filter is Hermitian (H(-w) = conj H(w),
// ktmApplyRhoFilter.m:39-58), so filtering z and taking real and imaginary parts gives
// the two filtered traces.  The Nyquist bin, where the script's filter is not Hermitian
// (2.5D), is the one place this needs care: real(ifft(H X)) only sees Re(H) there, so
// Re(H) is what is applied.  M = 2^ceil(log2 tracePts) <= 16384.
//
// The FFT (prep_kernel): M / 16 threads hold 16 values each in registers and run radix-16
// passes (a last one of radix 2, 4 or 8 where log2 M is not a multiple of 4).  The forward
// transform is decimated in frequency, so its spectrum comes out in digit-reversed order,
// the filter is applied there, and the inverse, decimated in time, takes it as it is: no
// reordering pass, and the last forward and first inverse pass meet in registers.  The
// first pass reads global memory (lane t: samples t + j M/16, coalesced) and the last one
// ends with the same samples in registers, which are folded, scaled and stored from there.
// In between, 2 (passes - 1) exchanges go through shared memory; value n lies at word
// n ^ ((n >> 4) & 15), which gives 16 neighbouring lanes 16 different 8-byte banks at
// every pass's stride.  CTAs stay for several pairs and keep tables of the
// twiddles (sincospif each), the filter and the fold weights in shared memory.
// What bounds it: issue and the FP32 pipe, about 1700 instructions a thread and pair, 62 % of
// the issue slots busy at 16 warps per SM.  62,500 traces of 1501 samples, 3D
// filter to FP16: 297 us, where the radix-2 transform in shared memory (22 passes with a
// barrier each, double-precision filter) took 2581; 4 bytes read and 2 written per sample
// would take 86.  Without a filter the same kernel keeps the samples in registers between
// the maximum and the store: 102 us, against 217 for a second read from cache.
//
// Output record of trace k (ktmPrepareTraces in include/ktm.h):
//   out[k][j] = Q(x'_j / s_k), x'_j = filtered x_j (times sqrt(j dt) when
//   prefold), 0 < j < tracePts; out[k][0] = out[k][j >= tracePts] = 0.
//   s_k = max|x'| (BF16), max|x'| / 32768 (F16), 1 (F32).
#include "ktm_ibm.cuh"
#include "ktm_pair.cuh"

#include <algorithm>

namespace ktm {
namespace {

constexpr int kMaxFft = 16384;

struct PrepArgs {
    int ntr, nt, inStride, pitch;
    float dt;
    const float* in;
    int ibm;                 // 1: in holds IBM-32 words
    int rho, scriptOrder, prefold, fmt;
    void* out;
    float* scale;
    float wHi, wLo;          // 2 pi / dt (pi / dt for the 2.5D filter) in two floats
};

__device__ __forceinline__ void to_sample(float& d, float v) { d = v; }
__device__ __forceinline__ void to_sample(__half& d, float v) { d = __float2half_rn(v); }
__device__ __forceinline__ void to_sample(__nv_bfloat16& d, float v) { d = __float2bfloat16_rn(v); }

// s_k from the trace's absolute maximum
__device__ __forceinline__ float trace_scale(int fmt, float m)
{
    if (fmt == KTM_FMT_F32 || !(m > 0.0f)) return 1.0f;
    return fmt == KTM_FMT_F16 ? m / 32768.0f : m;
}

// output slot of trace k (the script's rotation for odd traceNo: out[q] = in[(q+1) mod n])
__device__ __forceinline__ int out_slot(const PrepArgs& a, int k)
{
    return a.scriptOrder && (a.ntr & 1) && a.ntr > 1 ? (k + a.ntr - 1) % a.ntr : k;
}

// ------------------------------------------------------------------- FFT ---
__device__ __forceinline__ float2 cadd(float2 a, float2 b)
{
    float2 r;
    dev::upk(dev::add2(dev::pk(a.x, a.y), dev::pk(b.x, b.y)), r.x, r.y);
    return r;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b)
{
    float2 r;
    dev::upk(dev::sub2(dev::pk(a.x, a.y), dev::pk(b.x, b.y)), r.x, r.y);
    return r;
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 conj_if(float2 a, bool c) { return make_float2(a.x, c ? -a.y : a.y); }

// X[k] = sum_j z[j] e^{-+2 pi i jk/4} in place (INV: +)
template <bool INV>
__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d)
{
    const float2 s = cadd(a, c), t = csub(a, c), u = cadd(b, d), v = csub(b, d);
    a = cadd(s, u);
    c = csub(s, u);
    // t -+ i v
    b = INV ? make_float2(t.x - v.y, t.y + v.x) : make_float2(t.x + v.y, t.y - v.x);
    d = INV ? make_float2(t.x + v.y, t.y - v.x) : make_float2(t.x - v.y, t.y + v.x);
}

// e^{-2 pi i n / 16}
__device__ __forceinline__ constexpr float2 w16(int n)
{
    constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f, h = 0.70710678118654752f;
    constexpr float cs[16] = {1, c1, h, s1, 0, -s1, -h, -c1, -1, -c1, -h, -s1, 0, s1, h, c1};
    return float2{cs[n & 15], cs[(n + 4) & 15]};
}

// R-point transform in place; X[m] ends at z[slot<R>(m)]
template <int R>
__device__ __forceinline__ constexpr int slot(int m)
{
    return R == 16 ? 4 * (m & 3) + (m >> 2) : R == 8 ? 2 * (m & 3) + (m >> 2) : m;
}
template <int R, bool INV>
__device__ __forceinline__ void dft(float2* z)
{
    if constexpr (R == 2) {
        const float2 a = z[0], b = z[1];
        z[0] = cadd(a, b);
        z[1] = csub(a, b);
    } else if constexpr (R == 4) {
        dft4<INV>(z[0], z[1], z[2], z[3]);
    } else if constexpr (R == 8) {
#pragma unroll
        for (int i = 0; i < 2; i++) dft4<INV>(z[i], z[i + 2], z[i + 4], z[i + 6]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 a = z[2 * k], b = k ? cmul(z[2 * k + 1], conj_if(w16(2 * k), INV)) : z[1];
            z[2 * k] = cadd(a, b);
            z[2 * k + 1] = csub(a, b);
        }
    } else if constexpr (R == 16) {
#pragma unroll
        for (int i = 0; i < 4; i++) dft4<INV>(z[i], z[i + 4], z[i + 8], z[i + 12]);
#pragma unroll
        for (int k = 1; k < 4; k++)
#pragma unroll
            for (int i = 1; i < 4; i++) z[i + 4 * k] = cmul(z[i + 4 * k], conj_if(w16(i * k), INV));
#pragma unroll
        for (int k = 0; k < 4; k++) dft4<INV>(z[4 * k], z[4 * k + 1], z[4 * k + 2], z[4 * k + 3]);
    }
}

// Word of value n.  The map is linear over XOR, so value at + m s of a pass (m s in bits
// that are zero in `at`) lies at (swz(at) ^ low bits) + high bits of swz(m s): constants.
__host__ __device__ __forceinline__ constexpr int swz(int n) { return n ^ ((n >> 4) & 15); }
__device__ __forceinline__ constexpr int at_plus(int swzAt, int ms)
{
    return (swzAt ^ (swz(ms) & 15)) + (swz(ms) & ~15);
}

template <int LOGM, bool FILTER>
struct FftShape {
    static constexpr int M = 1 << LOGM;
    static constexpr int E = M < 16 ? M : 16;            // values per thread
    static constexpr int T = M / E;                       // threads per pair
    static constexpr int kPasses = LOGM <= 4 ? 1 : (LOGM + 3) / 4;
    static constexpr int kLast = LOGM == 0 ? 1 : 1 << ((LOGM - 1) % 4 + 1);   // last radix
    static constexpr int kPairs = T >= 128 ? 1 : 128 / T; // pairs of traces per CTA
    static constexpr int kThreads = T * kPairs;
    // 16 warps of 128 registers per SM with the transform (where a CTA is not larger): 20 warps
    // of 96 take 300 us instead of 297 for 62,500 traces of 1501 samples; 32 warps without it
    static constexpr int kCtasPerSm = kThreads >= 1024 ? 1 : (FILTER ? 512 : 1024) / kThreads;
    static constexpr bool kTables = LOGM <= 13;           // all tables fit beside z, at 16384 that of |H|
    // twiddles w_N^(i m), m = 1 .. 15, of every radix-16 pass: 15 (M/16 + M/256 + ...)
    static constexpr int kTwiddles = kPasses == 1 ? 0 : 15 * (T + (kPasses > 2 ? T / 16 : 0) + (kPasses > 3 ? T / 256 : 0));
    static constexpr size_t kSmem = FILTER ? (size_t)kPairs * M * 8 + (size_t)M * 4 + (kTables ? (size_t)M * 4 + kTwiddles * 8 : 0)
                                           : kTables ? (size_t)M * 4 : 0;
};

// Size of H at FFT bin k, as ktmApplyRhoFilter.m:33 pairs omega = 2 pi kk / Dr with the
// shifted spectrum (kk = k - M for k >= M/2): 2D |w|; 2.5D sqrt|w| e^{i pi/4 sgn w}, both
// parts of size sqrt(|w| / 2); 3D i w, zero at Nyquist.  |w| is the sum of two floats, and the
// approximate root takes one Newton step against both: 6 million sizes (dt from 1e-5 to 1 s, k to
// 8192, roots 2^-22 off) are the doubles of the formula rounded once; 4 % of the 2.5D ones are not if
// the root is taken of |w| already rounded.
template <int M>
__device__ __forceinline__ float rho_size(const PrepArgs& a, int k)
{
    const int kk = k < (M >> 1) ? k : k - M;
    const float f = fabsf((float)kk), w = fmaf(f, a.wHi, f * a.wLo);
    if (a.rho == KTM_RHO_25D) {
        const float hi = __fmul_rn(f, a.wHi), lo = fmaf(f, a.wLo, fmaf(f, a.wHi, -hi));
        const float y = dev::rsqrt_approx(hi), s = hi * y;
        return f > 0.0f ? fmaf(fmaf(-s, s, hi) + lo, 0.5f * y, s) : 0.0f;
    }
    return a.rho == KTM_RHO_3D && k == (M >> 1) ? 0.0f : w;
}

template <int LOGM, bool FILTER>
__global__ void __launch_bounds__(FftShape<LOGM, FILTER>::kThreads, FftShape<LOGM, FILTER>::kCtasPerSm) prep_kernel(PrepArgs a)
{
    using S = FftShape<LOGM, FILTER>;
    constexpr int M = S::M, E = S::E, T = S::T, R = S::kLast, G = E / R, P = S::kPasses;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // the warps' maxima: two sets in turn where the barrier before they are read is the only
    // one of a round, so that a warp in the next round writes none that is still to be read;
    // the transform's barriers keep the rounds apart
    __shared__ float2 red[FILTER ? 1 : 2][S::kThreads / 32 + 1];
    int set = 0;
    const int t = threadIdx.x % T, sub = threadIdx.x / T;
    float2* zs = reinterpret_cast<float2*>(smem_raw) + (size_t)sub * M;
    // z of each pair, twiddles, |H| [E][T], fold weights [M]
    float2* twTab = reinterpret_cast<float2*>(smem_raw) + (FILTER ? S::kPairs * M : 0);
    float* hTab = reinterpret_cast<float*>(twTab + (FILTER && S::kTables ? S::kTwiddles : 0));
    float* wTab = hTab + (FILTER ? M : 0);

    // frequency of the last forward pass's output m of group g: the hexadecimal digits of
    // the position in reverse, m the most significant
    auto bin = [&](int g, int m) {
        int k = m, d = g;
#pragma unroll
        for (int q = 0; q < P - 1; q++) {
            k = 16 * k + (d & 15);
            d >>= 4;
        }
        return k;
    };
    // e^{-2 pi i x / M}: the exponent in turns is exact
    auto turn = [&](int x) {
        float sn, cs;
        sincospif(2.0f / (float)M * (float)x, &sn, &cs);
        return make_float2(cs, -sn);
    };
    // z[m] *= w_N^(i m), N = 16 s, of pass q (conj: its conjugate); ord: value m lies at slot(m)
    auto twiddle = [&](float2* z, int q, bool conj, bool ord) {
        const int s = (M >> (4 * q)) / 16, i = t % s;
        const float2* tab = twTab + 15 * (q > 0 ? T : 0) + 15 * (q > 1 ? T / 16 : 0) + i;
#pragma unroll
        for (int m = 1; m < 16; m++) {
            const float2 w = S::kTables ? tab[(m - 1) * s] : turn((i << (4 * q)) * m);
            float2& v = z[ord ? slot<16>(m) : m];
            v = cmul(v, conj_if(w, conj));
        }
    };
    if (FILTER || S::kTables) {
        if (FILTER && S::kTables) {
            int o = 0;
#pragma unroll
            for (int q = 0; q + 1 < P; q++) {
                const int s = (M >> (4 * q)) / 16;
                for (int v = threadIdx.x; v < 15 * s; v += S::kThreads) twTab[o + v] = turn(((v % s) << (4 * q)) * (v / s + 1));
                o += 15 * s;
            }
        }
        for (int v = threadIdx.x; v < M; v += S::kThreads) {
            const int u = v / T, g = v % T + T * (u / R);
            if (FILTER) hTab[v] = rho_size<M>(a, bin(g, u % R));
            if (S::kTables) wTab[v] = (FILTER ? 1.0f / (float)M : 1.0f) * (a.prefold ? sqrtf((float)v * a.dt) : 1.0f);
        }
        __syncthreads();
    }
    // real and imaginary part of H in units of its size
    const float re = a.rho == KTM_RHO_3D ? 0.0f : 1.0f, im = a.rho == KTM_RHO_2D ? 0.0f : 1.0f;
    const int pairs = (a.ntr + 1) / 2;
    for (int base = blockIdx.x * S::kPairs; base < pairs; base += gridDim.x * S::kPairs) {
        const int k0 = 2 * (base + sub);
        const bool one = k0 < a.ntr, two = k0 + 1 < a.ntr;
        const float* x = a.in + (size_t)k0 * a.inStride;
        float2 z[E];
        // z = x + i y, zero padded to M (fft(trace', M), :37)
        const int ntx = one ? a.nt - t : 0, nty = two ? a.nt - t : 0;
        x += t;
        if (a.ibm) {
            const uint32_t* w = reinterpret_cast<const uint32_t*>(x);
            bool other = false;
#pragma unroll
            for (int j = 0; j < E; j++) {
                z[j].x = dev::ibm32_usual(T * j < ntx ? w[T * j] : 0u, other);
                z[j].y = dev::ibm32_usual(T * j < nty ? w[a.inStride + T * j] : 0u, other);
            }
            if (other) {
#pragma unroll
                for (int j = 0; j < E; j++) {
                    if (T * j < ntx) z[j].x = dev::ibm32_any(w[T * j]);
                    if (T * j < nty) z[j].y = dev::ibm32_any(w[a.inStride + T * j]);
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < E; j++) {
                z[j].x = T * j < ntx ? x[T * j] : 0.0f;
                z[j].y = T * j < nty ? x[a.inStride + T * j] : 0.0f;
            }
        }
        if constexpr (FILTER) {
            // forward radix-16 passes
#pragma unroll
            for (int q = 0; q + 1 < P; q++) {
                const int N = M >> (4 * q), s = N / 16, at = swz(t / s * N + t % s);
                if (q > 0) {
#pragma unroll
                    for (int j = 0; j < 16; j++) z[j] = zs[at_plus(at, j * s)];
                }
                dft<16, false>(z);
                twiddle(z, q, false, true);
#pragma unroll
                for (int m = 0; m < 16; m++) zs[at_plus(at, m * s)] = z[slot<16>(m)];
                __syncthreads();
            }
            // last forward pass, filter, first inverse pass: groups t + T u of R values
#pragma unroll
            for (int u = 0; u < G; u++) {
                const int g = t + T * u, at = swz(g * R);
                float2 v[R], f[R];
#pragma unroll
                for (int j = 0; j < R; j++) v[j] = P > 1 ? zs[at_plus(at, j)] : z[u * R + j];
                dft<R, false>(v);
#pragma unroll
                for (int m = 0; m < R; m++) {
                    // bin m M / R + (bins of g): negative frequencies from m = R / 2 on, where bin
                    // M / 2 (Nyquist, g = 0) keeps the real part alone
                    const float h = hTab[(u * R + m) * T + t];
                    const float i = 2 * m < R ? im : 2 * m == R && g == 0 ? 0.0f : -im;
                    const float2 x = v[slot<R>(m)];
                    const float px = h * x.x, py = h * x.y;
                    f[m] = make_float2(re * px - i * py, i * px + re * py);
                }
                dft<R, true>(f);
#pragma unroll
                for (int j = 0; j < R; j++) {
                    if (P > 1) zs[at_plus(at, j)] = f[slot<R>(j)];
                    else z[u * R + j] = f[slot<R>(j)];
                }
            }
            // inverse radix-16 passes
#pragma unroll
            for (int q = P - 2; q >= 0; q--) {
                const int N = M >> (4 * q), s = N / 16, at = swz(t / s * N + t % s);
                __syncthreads();
                float2 v[16];
#pragma unroll
                for (int m = 0; m < 16; m++) v[m] = zs[at_plus(at, m * s)];
                twiddle(v, q, true, false);
                dft<16, true>(v);
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    if (q > 0) zs[at_plus(at, j * s)] = v[slot<16>(j)];
                    else z[j] = v[slot<16>(j)];
                }
            }
        }
        // sample window, 1 / M and weight fold, absmax
        float mx = 0.0f, my = 0.0f;
#pragma unroll
        for (int j = 0; j < E; j++) {
            const int n = t + T * j;
            const bool in = n < a.nt && (j > 0 || t > 0);
            const float w = S::kTables ? wTab[n] : (FILTER ? 1.0f / (float)M : 1.0f) * (a.prefold ? sqrtf((float)n * a.dt) : 1.0f);
            z[j].x = in ? z[j].x * w : 0.0f;
            z[j].y = in ? z[j].y * w : 0.0f;
            mx = fmaxf(mx, fabsf(z[j].x));
            my = fmaxf(my, fabsf(z[j].y));
        }
        if (a.fmt != KTM_FMT_F32) {
#pragma unroll
            for (int o = (T < 32 ? T : 32) / 2; o > 0; o >>= 1) {
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                my = fmaxf(my, __shfl_xor_sync(0xffffffffu, my, o));
            }
            if (T > 32) {
                if ((threadIdx.x & 31) == 0) red[set][threadIdx.x >> 5] = make_float2(mx, my);
                __syncthreads();
#pragma unroll 8
                for (int w = 0; w < T / 32; w++) {
                    const float2 o = red[set][sub * (T / 32) + w];
                    mx = fmaxf(mx, o.x);
                    my = fmaxf(my, o.y);
                }
                if constexpr (!FILTER) set ^= 1;
            }
        }
        const float sx = trace_scale(a.fmt, mx), sy = trace_scale(a.fmt, my);
        const float ix = 1.0f / sx, iy = 1.0f / sy;
        const size_t ox = (size_t)(one ? out_slot(a, k0) : 0), oy = (size_t)(two ? out_slot(a, k0 + 1) : 0);
        auto put = [&](auto* out) {
            auto *px = out + ox * a.pitch + t, *py = out + oy * a.pitch + t;
            const int px1 = one ? a.pitch - t : 0, py1 = two ? a.pitch - t : 0;
#pragma unroll
            for (int j = 0; j < E; j++) {
                if (T * j < px1) to_sample(px[T * j], z[j].x * ix);
                if (T * j < py1) to_sample(py[T * j], z[j].y * iy);
            }
            for (int n = M; n < px1; n += T) to_sample(px[n], 0.0f);       // guards past the transform
            for (int n = M; n < py1; n += T) to_sample(py[n], 0.0f);
        };
        if (a.fmt == KTM_FMT_F32) put(static_cast<float*>(a.out));
        else if (a.fmt == KTM_FMT_F16) put(static_cast<__half*>(a.out));
        else put(static_cast<__nv_bfloat16*>(a.out));
        if (t == 0) {
            if (one) a.scale[ox] = sx;
            if (two) a.scale[oy] = sy;
        }
    }
}

// Traces longer than a transform, without a filter: a CTA of 1024 threads per trace holds it in
// registers between the maximum and the store, all its loads in flight at once.  1000 traces of
// 20,000 samples to F16: 47 us (120 MB, 2.5 TB/s: one CTA an SM, its load, barrier and store in
// turn), one trace 7; a warp per trace that reads it twice took 446 and 121, a CTA per pair in
// shared memory 119 and 17.  From 8193 to 16384 samples the transform's kernel without its passes
// is the faster (2441 traces of 8193: 49 us against 74): its CTAs stay for several pairs.
constexpr int kPackThreads = 1024, kPackSamples = kMaxSmemBytes / 8;
template <class OUT>
__global__ void __launch_bounds__(kPackThreads) pack_kernel(PrepArgs a)
{
    constexpr int E = (kPackSamples + kPackThreads - 1) / kPackThreads;
    __shared__ float red[kPackThreads / 32];
    const int t = threadIdx.x, k = blockIdx.x;
    const float* x = a.in + (size_t)k * a.inStride;
    float z[E];
    if (a.ibm) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(x);
        bool other = false;
#pragma unroll
        for (int j = 0; j < E; j++) {
            const int n = t + kPackThreads * j;
            z[j] = dev::ibm32_usual(n < a.nt ? w[n] : 0u, other);
        }
        if (other) {
#pragma unroll
            for (int j = 0; j < E; j++) {
                const int n = t + kPackThreads * j;
                if (n < a.nt) z[j] = dev::ibm32_any(w[n]);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < E; j++) {
            const int n = t + kPackThreads * j;
            z[j] = n < a.nt ? x[n] : 0.0f;
        }
    }
    if (t == 0) z[0] = 0.0f;
    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < E; j++) {
        const int n = t + kPackThreads * j;
        if (a.prefold && n < a.nt) z[j] *= sqrtf((float)n * a.dt);
        m = fmaxf(m, fabsf(z[j]));
    }
    if (a.fmt != KTM_FMT_F32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((t & 31) == 0) red[t >> 5] = m;
        __syncthreads();
        m = red[t & 31];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    const float s = trace_scale(a.fmt, m), inv = 1.0f / s;
    OUT* out = static_cast<OUT*>(a.out) + (size_t)out_slot(a, k) * a.pitch;
#pragma unroll
    for (int j = 0; j < E; j++) {
        const int n = t + kPackThreads * j;
        if (n < a.pitch) to_sample(out[n], z[j] * inv);
    }
    for (int n = t + kPackThreads * E; n < a.pitch; n += kPackThreads) to_sample(out[n], 0.0f);
    if (t == 0) a.scale[out_slot(a, k)] = s;
}

template <int LOGM, bool FILTER>
int launch_filter(const PrepArgs& a, cudaStream_t s)
{
    using S = FftShape<LOGM, FILTER>;
    auto kern = prep_kernel<LOGM, FILTER>;
    KTM_CUDA_TRY(allow_smem(kern, S::kSmem, S::kSmem));
    int dev = 0, sm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
    const int room = (int)std::min<size_t>(S::kCtasPerSm, (size_t)(224 * 1024) / (S::kSmem + 1536));
    const int units = ((a.ntr + 1) / 2 + S::kPairs - 1) / S::kPairs, slots = sm * std::max(1, room);
    // as many rounds as the resident CTAs need, evenly filled
    const int rounds = (units + slots - 1) / slots, grid = (units + rounds - 1) / rounds;
    kern<<<grid, S::kThreads, S::kSmem, s>>>(a);
    KTM_CUDA_TRY(cudaGetLastError());
    return KTM_OK;
}

template <int LOGM>
int launch_prep(const PrepArgs& a, cudaStream_t s)
{
    return a.rho != KTM_RHO_NONE ? launch_filter<LOGM, true>(a, s) : launch_filter<LOGM, false>(a, s);
}

__global__ void widen_kernel(const void* __restrict__ in, int fmt, const float* __restrict__ scale,
                             int ntr, int nt, int stride, float* __restrict__ out)
{
    const size_t n = (size_t)ntr * nt;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t k = i / nt, j = i % nt;
        const size_t src = k * stride + j;
        float v = fmt == KTM_FMT_F16 ? __half2float(static_cast<const __half*>(in)[src])
                                     : __bfloat162float(static_cast<const __nv_bfloat16*>(in)[src]);
        if (scale) v *= scale[k];
        out[i] = v;
    }
}

}  // namespace

int widen_traces(const void* in, int fmt, const float* scale, int ntr, int nt, int stride,
                 void** out, cudaStream_t s)
{
    *out = nullptr;
    const size_t n = (size_t)ntr * nt;
    if (n == 0) return KTM_OK;
    KTM_CUDA_TRY(pool_malloc(out, n * sizeof(float), s));
    const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 65535 * 8);
    widen_kernel<<<blocks, 256, 0, s>>>(in, fmt, scale, ntr, nt, stride, static_cast<float*>(*out));
    KTM_CUDA_TRY(cudaGetLastError());
    return KTM_OK;
}

int packed_pitch(int nt, int fmt)
{
    const int esize = fmt == KTM_FMT_F32 ? 4 : 2;
    const int per16 = 16 / esize;
    return ((nt + 2 + per16 - 1) / per16) * per16;
}

int prepare_traces(const ktm_prep* p)
{
    if (!p) return set_error(KTM_ERR_ARG, "NULL prep");
    if (p->traceNo < 0 || p->tracePts < 0) return set_error(KTM_ERR_ARG, "negative sizes");
    if (p->outFormat < KTM_FMT_F32 || p->outFormat > KTM_FMT_BF16)
        return set_error(KTM_ERR_ARG, "bad outFormat %d", p->outFormat);
    if (p->rho < KTM_RHO_NONE || p->rho > KTM_RHO_3D) return set_error(KTM_ERR_ARG, "bad rho %d", p->rho);
    if (p->inFormat != KTM_FMT_F32 && p->inFormat != KTM_FMT_IBM32)
        return set_error(KTM_ERR_ARG, "bad inFormat %d (F32 or IBM32)", p->inFormat);
    if (!(p->sampleRate > 0.0f)) return set_error(KTM_ERR_ARG, "sampleRate must be > 0");
    if (p->traceNo == 0) return KTM_OK;
    if (!p->in || !p->out || !p->outScale) return set_error(KTM_ERR_ARG, "NULL buffer");
    PrepArgs a;
    a.ntr = p->traceNo; a.nt = p->tracePts;
    a.inStride = p->inStride > 0 ? p->inStride : p->tracePts;
    if (a.inStride < a.nt) return set_error(KTM_ERR_ARG, "inStride < tracePts");
    a.pitch = p->outPitch > 0 ? p->outPitch : packed_pitch(p->tracePts, p->outFormat);
    const int esize = p->outFormat == KTM_FMT_F32 ? 4 : 2;
    if (a.pitch < a.nt + 2 || (a.pitch * esize) % 16 != 0)
        return set_error(KTM_ERR_ARG, "outPitch must be >= tracePts + 2 and a multiple of 16 bytes");
    if (reinterpret_cast<uintptr_t>(p->out) % 16 != 0)
        return set_error(KTM_ERR_ARG, "out must be 16-byte aligned");
    a.dt = p->sampleRate; a.in = p->in; a.ibm = p->inFormat == KTM_FMT_IBM32; a.rho = p->rho; a.scriptOrder = p->rhoScriptOrder;
    a.prefold = p->prefold; a.out = p->out; a.scale = p->outScale; a.fmt = p->outFormat;
    const double w = (a.rho == KTM_RHO_25D ? 1.0 : 2.0) * 3.14159265358979323846 / (double)a.dt;
    a.wHi = (float)w;
    a.wLo = (float)(w - (double)a.wHi);
    cudaStream_t s = static_cast<cudaStream_t>(p->stream);
    if (a.rho != KTM_RHO_NONE && a.nt > kMaxFft) return set_error(KTM_ERR_LIMIT, "rho filter: tracePts > %d", kMaxFft);
    if ((size_t)a.nt * sizeof(float2) > (size_t)kMaxSmemBytes)
        return set_error(KTM_ERR_LIMIT, "prepare: tracePts > %d", kMaxSmemBytes / 8);
    if (a.nt > kMaxFft) {
        const unsigned grid = (unsigned)a.ntr;
        if (a.fmt == KTM_FMT_F32) pack_kernel<float><<<grid, kPackThreads, 0, s>>>(a);
        else if (a.fmt == KTM_FMT_F16) pack_kernel<__half><<<grid, kPackThreads, 0, s>>>(a);
        else pack_kernel<__nv_bfloat16><<<grid, kPackThreads, 0, s>>>(a);
        KTM_CUDA_TRY(cudaGetLastError());
        return KTM_OK;
    }
    int logM = 0;
    while ((1 << logM) < a.nt) logM++;
    switch (logM) {
        case 0: return launch_prep<0>(a, s);
        case 1: return launch_prep<1>(a, s);
        case 2: return launch_prep<2>(a, s);
        case 3: return launch_prep<3>(a, s);
        case 4: return launch_prep<4>(a, s);
        case 5: return launch_prep<5>(a, s);
        case 6: return launch_prep<6>(a, s);
        case 7: return launch_prep<7>(a, s);
        case 8: return launch_prep<8>(a, s);
        case 9: return launch_prep<9>(a, s);
        case 10: return launch_prep<10>(a, s);
        case 11: return launch_prep<11>(a, s);
        case 12: return launch_prep<12>(a, s);
        case 13: return launch_prep<13>(a, s);
        default: return launch_prep<14>(a, s);
    }
}

}  // namespace ktm

extern "C" {

int ktmPackedPitch(int tracePts, int format) { return ktm::packed_pitch(tracePts, format); }

int ktmPrepareTraces(const ktm_prep* prep)
{
    int rc = ktm::prepare_traces(prep);
    return rc ? rc : ktm::set_ok();
}

}  // extern "C"
