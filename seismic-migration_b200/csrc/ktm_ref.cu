// ktm_ref.cu -- reference-mode PSTM kernel: the arithmetic of psktmCPU.c:13-101
// on sm_100a, bit-identical to the reference run with one thread.
//
// How bit-identity is kept
//   * every float operation rounds as the C source's does (SSE sqrtss / divss in the
//     gcc -O3 x86-64 build of psktmCPU.c): sums and products are single explicitly
//     rounded instructions that nothing contracts into an FMA, square roots and
//     quotients are correctly rounded (below);
//   * the operand order follows the C source (:46-49, :65-72, :78-85);
//   * each image sample is owned by one lane, which adds the traces in increasing
//     k, the order of the reference's outer loop (:56-59).
//
// Correct rounding without the library sequences (ref_packs; the enumerations below were made once,
// the tests compare whole migrations bit for bit): two traces go through
// each packed f32x2 instruction, and inside the operand ranges below no special case
// is left to test for.
//   sqrt(a): y = rsqrt.approx(a), g = a y, s = g + (a - g^2) (y / 2), the residual and
//     the last step one FMA each (Markstein, IBM J. Res. Dev. 34, 1990).  Checked
//     against __fsqrt_rn on all 2^24 operands of two neighbouring binades, in five
//     ranges of exponents: no difference.
//   a / b: r = rcp.approx(b) with one Newton step is the correctly rounded reciprocal
//     (all 2^23 significands checked against __frcp_rn); q = q0 + (a - b q0) r with
//     q0 = a r rounds correctly wherever a / b lies further than n / (b 2^k) from a
//     rounding boundary, n <= 3 (Markstein's bound); the at most 8 significands a per b
//     that lie nearer are enumerated over all 2^23 b and agree with __fdiv_rn.
//   t / dt: the same with r = RN(1 / dt) from the host.
// Operand ranges: dt in [2^-20, 2^10]; tau^2 zero or in [2^-60, 2^30]; 1 / v^2 zero or
// in [2^-40, 2^10]; squared distances zero or in [2^-30, 2^44].  Then no intermediate
// overflows, no residual underflows and every value is finite.  tau = 0 would put zeros
// under the square roots; 2^-96 stands in for tau^2 = 0: it vanishes from every t that
// can reach a sample (t >= dt), and the sample's sum, all of whose terms the reference
// multiplies by sqrt(0 / t) = 0, is multiplied by zero at the end (which also gives the
// reference's NaN where a picked sample is infinite or NaN).  A chunk of traces or a
// run of tau samples outside the ranges takes slow_pair, the plain intrinsics.
//
// Work decomposition (B200: 148 SMs, 32-wide warps)
//   warp = one image column x a run of 32*R consecutive tau samples; lane L owns
//          tau = run0 + L + 32*r, r < R, so a warp reads a narrow, monotone
//          window of each trace (few shared-memory bank conflicts).
//   CTA  = neighbouring columns of one run, one per warp.
//   Traces stream in chunks through shared memory (double-buffered 16-byte cp.async).
//   Per chunk, lane c of each warp evaluates trace c's squared distances and drops the
//   traces whose first sample time over the run lies past the trace end (rounding is
//   monotone, and the test keeps a margin), so every dropped pair is one the reference
//   skips (:82); the kept ones go in order into a warp-private table, two to an entry.
//   Samples 0 and tracePts of the staged rows are zeroed: a pair outside
//   0 < it < tracePts (:82) adds zero, which leaves the sum's bits as they are.
// What bounds it: four special-function results per pair (32 cycles of a scheduler's 4
// lanes) beside 58 packed FP32 lane-operations (29 cycles) and about 31 issue slots; the
// loop alone runs at 39 cycles a pair, with staging, geometry and barriers at about 50.
// 256 x 1001 image, 16,384 traces of 1001 samples: 6.59 ms; with the library square roots
// and divisions (78.5 instructions a pair, 4-byte staging) 27.98.  437 x 401, 3001 traces of
// 451 samples: 0.836 ms against 3.23.
#include "ktm_pair.cuh"

#include <algorithm>
#include <type_traits>

namespace ktm {
namespace {

using namespace dev;

constexpr int kRefMaxChunk = 32;                 // lane c evaluates trace c of a chunk
constexpr int kRefSmem = 224 * 1024;             // of all CTAs of an SM

// Samples per lane (R), table entries of two traces in flight (U), warps per SM: 4 x 2
// packs need 124 registers (16 warps), the others fit 64 (32 warps).
template <int R>
struct RefShape {
    static constexpr int U = R == 1 ? 4 : 2;
    static constexpr int kWarpsPerSm = R == 4 ? 16 : 32;
};
constexpr float kTinyTau2 = 1.262177448353619e-29f;   // 2^-96, in place of tau^2 = 0

struct RefArgs {
    Geometry g;
    const float *midX, *midY, *offX, *offY, *traces, *vel;
    float* image;
    int accumulate;
    int chunk;            // traces per shared-memory stage
    int colGroups;        // CTAs per run
    int fastDt;           // dt within the range of the packed quotient
    float rdt;            // RN(1 / dt)
    float nzero;          // -0
    float tend;           // a first sample time above this is past every sample
};

// Shared memory of one CTA: two row buffers, two of coordinates, then per warp the kept
// traces' table (an entry: {tA0, tA1, tB0, tB1} and the two row addresses).
struct RefSmem {
    size_t rowBytes, crdOff, tabOff, total;
};
// table entries of a warp: an even number, so that every warp's entries are 16-byte aligned
__host__ __device__ __forceinline__ int ref_entries(int chunk) { return (chunk + 3) / 4 * 2; }
__host__ __device__ __forceinline__ RefSmem ref_smem(int chunk, int stride, int nt, int warps)
{
    RefSmem s;
    // a chunk starts up to 12 bytes into its buffer (the source's alignment); the last
    // row's guard may lie one float past the rows
    s.rowBytes = (((size_t)(chunk - 1) * stride + nt + 1) * 4 + 12 + 15) / 16 * 16;
    s.crdOff = 2 * s.rowBytes;
    s.tabOff = s.crdOff + 2 * 4 * (size_t)chunk * 4;
    s.total = s.tabOff + (size_t)warps * ref_entries(chunk) * 24;
    return s;
}

__device__ __forceinline__ void cp_async16(unsigned smem, const void* gmem)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem), "l"(gmem));
}

// The calling warp's share of n floats from src to the shared address dst, dst = src (mod
// 16): 16-byte pieces between the first and the last boundary, `seg` of them to a warp
// (a multiple of 32), 4-byte pieces outside them (the last warp).
__device__ __forceinline__ void stage_rows(unsigned dst, const float* src, int n, int seg, int warp, int warps,
                                           int lane)
{
    const int head = min(n, (int)((16u - (unsigned)(reinterpret_cast<uintptr_t>(src) & 15u)) & 15u) / 4);
    const int body = (n - head) / 4, tail = n - head - 4 * body;
    if (warp == warps - 1) {
        const int i = lane < head ? lane : lane >= 8 && lane < 8 + tail ? head + 4 * body + lane - 8 : -1;
        if (i >= 0)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst + 4u * i), "l"(src + i));
    }
    const int end = min(body, (warp + 1) * seg);
    int i = warp * seg + lane;
    unsigned d = dst + 4u * head + 16u * i;
    const float* p = src + head + 4 * (size_t)i;
    for (; i + 96 < end; i += 128, d += 2048, p += 512) {
        cp_async16(d, p);
        cp_async16(d + 512, p + 128);
        cp_async16(d + 1024, p + 256);
        cp_async16(d + 1536, p + 384);
    }
    for (; i < end; i += 32, d += 512, p += 128) cp_async16(d, p);
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct RefConst {
    f2 nrdt, dt, half, one, magic, nzero;
    float umax;
};

// RN(a b) of both halves as an FMA onto -0.  The compiler contracts a packed product
// whose only use is a packed sum, explicit .rn or not; -0 is a kernel argument, so that
// it cannot see this one as a product.
__device__ __forceinline__ f2 product2(f2 a, f2 b, const RefConst& k) { return fma2(a, b, k.nzero); }

// -RN(sqrt(a)) of N packs na = -a, in lock step: N independent chains in flight.
template <int N>
__device__ __forceinline__ void neg_sqrt2(const f2 (&na)[N], f2 (&ns)[N], f2 half)
{
    f2 y[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
        float a0, a1;
        upk(na[i], a0, a1);
        y[i] = pk(rsqrt_approx(-a0), rsqrt_approx(-a1));
    }
#pragma unroll
    for (int i = 0; i < N; i++) ns[i] = mul2(na[i], y[i]);
#pragma unroll
    for (int i = 0; i < N; i++) y[i] = mul2(y[i], half);
    f2 d[N];
#pragma unroll
    for (int i = 0; i < N; i++) d[i] = fma2(ns[i], ns[i], na[i]);
#pragma unroll
    for (int i = 0; i < N; i++) ns[i] = fma2(d[i], y[i], ns[i]);
}

// N image samples (nTQ = -tau^2, nSL = -1/v^2) and two traces: the values the reference
// adds (:78-85), zero where it adds none.  Signs are carried negated so that every
// residual is a plain FMA.
template <int N>
__device__ __forceinline__ void ref_packs(f2 TA, f2 TB, const f2 (&nSL)[N], const f2 (&nTQ)[N], const RefConst& k,
                                          unsigned row0, unsigned row1, f2 (&v)[N])
{
    f2 x[N], y[N], nt[N];
#pragma unroll
    for (int i = 0; i < N; i++) x[i] = add2(nTQ[i], product2(TA, nSL[i], k));
    neg_sqrt2(x, nt, k.half);
#pragma unroll
    for (int i = 0; i < N; i++) y[i] = add2(nTQ[i], product2(TB, nSL[i], k));
    neg_sqrt2(y, x, k.half);
#pragma unroll
    for (int i = 0; i < N; i++) nt[i] = add2(nt[i], x[i]);                       // -t
    f2 r[N], tr[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
        float n0, n1;
        upk(nt[i], n0, n1);
        r[i] = pk(rcp_approx(-n0), rcp_approx(-n1));
    }
    // q = RN(t / dt), then floor(min(q, tracePts)) in the low bits of q + 1.5 2^23
    f2 q[N], e[N];
#pragma unroll
    for (int i = 0; i < N; i++) q[i] = mul2(nt[i], k.nrdt);
#pragma unroll
    for (int i = 0; i < N; i++) e[i] = fma2(k.dt, q[i], nt[i]);
#pragma unroll
    for (int i = 0; i < N; i++) q[i] = fma2(e[i], k.nrdt, q[i]);
#pragma unroll
    for (int i = 0; i < N; i++) {
        float u0, u1, f0, f1;
        upk(q[i], u0, u1);
        upk(add2_rm(pk(fminf(u0, k.umax), fminf(u1, k.umax)), k.magic), f0, f1);
        tr[i] = pk(Lds<KTM_FMT_F32>::one(row0 + __float_as_uint(f0) * 4u),
                   Lds<KTM_FMT_F32>::one(row1 + __float_as_uint(f1) * 4u));
    }
    // -RN(tau^2 / t)
#pragma unroll
    for (int i = 0; i < N; i++) e[i] = fma2(nt[i], r[i], k.one);
#pragma unroll
    for (int i = 0; i < N; i++) r[i] = fma2(r[i], e[i], r[i]);
#pragma unroll
    for (int i = 0; i < N; i++) q[i] = mul2(nTQ[i], r[i]);
#pragma unroll
    for (int i = 0; i < N; i++) e[i] = fma2(nt[i], q[i], nTQ[i]);
#pragma unroll
    for (int i = 0; i < N; i++) q[i] = fma2(e[i], r[i], q[i]);
    neg_sqrt2(q, x, k.half);
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = product2(mul2(tr[i], nt[i]), x[i], k);
}

// The same pair by the plain intrinsics: any operands.
__device__ __noinline__ float slow_pair(float acc, float tA, float tB, float tauS, float slow, float dt,
                                        int nt, const float* tr)
{
    float t = __fsqrt_rn(__fadd_rn(tauS, __fmul_rn(tA, slow)));                  // :78-79
    t = __fadd_rn(t, __fsqrt_rn(__fadd_rn(tauS, __fmul_rn(tB, slow))));
    const int it = __float2int_rz(__fdiv_rn(t, dt));                             // :80
    if (it < nt && it > 0)                                                       // :82-85
        acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(tr[it], t), __fsqrt_rn(__fdiv_rn(tauS, t))));
    return acc;
}

__device__ __forceinline__ bool in_range(float x, float lo, float hi) { return x == 0.0f || (x >= lo && x <= hi); }

template <int R>
__global__ void __launch_bounds__(RefShape<R>::kWarpsPerSm * 32, 1) reference_kernel(RefArgs a)
{
    constexpr int U = RefShape<R>::U;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Geometry& g = a.g;
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const RefSmem L = ref_smem(a.chunk, g.stride, g.nt, warps);
    const unsigned smem0 = smem_u32(smem_raw);
    float* crdBase = reinterpret_cast<float*>(smem_raw + L.crdOff);
    const int entries = ref_entries(a.chunk);
    float* tab = reinterpret_cast<float*>(smem_raw + L.tabOff + (size_t)warp * entries * 24);
    unsigned* tabRow = reinterpret_cast<unsigned*>(tab + 4 * entries);

    const int col = (blockIdx.x % a.colGroups) * warps + warp;
    const bool colValid = col < g.nx * g.ny;
    const int ci = colValid ? col / g.ny : 0, cj = colValid ? col % g.ny : 0;
    const int run0 = (int)(blockIdx.x / a.colGroups) * (32 * R);

    // psktmFunctions.c:26-30: axis values in float
    const float xx = __fadd_rn(g.x0, __fmul_rn(__int2float_rn(ci), g.dx));
    const float yy = __fadd_rn(g.y0, __fmul_rn(__int2float_rn(cj), g.dy));

    f2 nTQ[R], nSL[R];
    float acc[R];
    float tmin = 3.0e38f, smin = 3.0e38f;
    bool okTables = a.fastDt != 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int l = run0 + lane + 32 * r, lc = l < g.nz ? l : g.nz - 1;
        const float zz = __fadd_rn(g.z0, __fmul_rn(__int2float_rn(lc), g.dz));
        const float tq = __fmul_rn(zz, zz);                                      // :47
        const float v = a.vel[lc];
        const float sl = __fdiv_rn(1.0f, __fmul_rn(v, v));                       // :48
        okTables = okTables && in_range(tq, 8.673617e-19f, 1.0737418e9f) && in_range(sl, 9.094947e-13f, 1024.0f);
        tmin = fminf(tmin, tq);
        smin = fminf(smin, sl);
        const float tt = tq == 0.0f ? kTinyTau2 : tq;
        nTQ[r] = pk(-tt, -tt);
        nSL[r] = pk(-sl, -sl);
        acc[r] = 0.0f;
    }
    okTables = __all_sync(0xffffffffu, okTables);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tmin = fminf(tmin, __shfl_xor_sync(0xffffffffu, tmin, o));
        smin = fminf(smin, __shfl_xor_sync(0xffffffffu, smin, o));
    }
    RefConst k;
    k.nrdt = pk(-a.rdt, -a.rdt); k.dt = pk(g.dt, g.dt); k.half = pk(0.5f, 0.5f); k.one = pk(1.0f, 1.0f);
    k.magic = pk(kMagic, kMagic); k.nzero = pk(a.nzero, a.nzero); k.umax = (float)g.nt;

    // a chunk's rows are one contiguous range that starts at the source's own offset from
    // a 16-byte boundary
    auto first_of = [&](int ch) { return a.traces + (size_t)ch * a.chunk * g.stride; };
    auto rows_of = [&](int ch) {      // byte offset of row 0 in shared memory
        return (unsigned)(ch & 1) * (unsigned)L.rowBytes + (unsigned)(reinterpret_cast<uintptr_t>(first_of(ch)) & 15u);
    };
    // 16-byte pieces of a full chunk per warp
    const int floats = (a.chunk - 1) * g.stride + g.nt;
    const int seg = ((floats / 4 + warps - 1) / warps + 31) & ~31;
    auto issue = [&](int ch) {
        const int k0 = ch * a.chunk, n = min(a.chunk, g.ntr - k0);
        stage_rows(smem0 + rows_of(ch), first_of(ch), (n - 1) * g.stride + g.nt, seg, warp, warps, lane);
        float* crd = crdBase + (ch & 1) * 4 * a.chunk;
        for (int arr = warp; arr < 4; arr += warps)
            if (lane < n)
                cp_async4(crd + arr * a.chunk + lane,
                          (arr == 0 ? a.midX : arr == 1 ? a.midY : arr == 2 ? a.offX : a.offY) + k0 + lane);
        cp_async_commit();
    };
    // zeroes samples 0 and tracePts of the rows (the next row's sample 0 where the rows are
    // dense), each by the warp that staged it, once its own copies have landed
    auto guard = [&](int ch, int n) {
        __syncwarp();
        const int head = (int)((16u - (unsigned)(reinterpret_cast<uintptr_t>(first_of(ch)) & 15u)) & 15u) / 4;
        const int total = (n - 1) * g.stride + g.nt, body = (total - head) / 4;
        if (lane < n) {
            float* rows = reinterpret_cast<float*>(smem_raw + rows_of(ch));
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int f = lane * g.stride + e * g.nt;
                const int piece = (f - head) >> 2;              // negative: the head
                const bool edge = piece < 0 || piece >= body;
                if (edge ? warp == warps - 1 : piece >= warp * seg && piece < (warp + 1) * seg) rows[f] = 0.0f;
            }
        }
    };

    const int nchunks = (g.ntr + a.chunk - 1) / a.chunk;
    issue(0);
    for (int ch = 0; ch < nchunks; ch++) {
        const int n = min(a.chunk, g.ntr - ch * a.chunk);
        cp_async_wait_all();
        guard(ch, n);
        __syncthreads();                     // chunk ch landed; chunk ch-1 fully consumed
        const unsigned rows = rows_of(ch);
        if (ch + 1 < nchunks) issue(ch + 1);
        // lane c: trace c's squared distances (:65-72, operand order of the C source)
        const float* crd = crdBase + (ch & 1) * 4 * a.chunk;
        float tA = 0.0f, tB = 0.0f;
        bool keep = false, ok = true;
        if (lane < n) {
            const float dxm = __fsub_rn(crd[lane], xx), ox = crd[2 * a.chunk + lane];
            const float dym = __fsub_rn(crd[a.chunk + lane], yy), oy = crd[3 * a.chunk + lane];
            const float cs = __fsub_rn(dxm, ox), cr = __fadd_rn(dxm, ox);
            const float ds = __fsub_rn(dym, oy), dr = __fadd_rn(dym, oy);
            tA = __fadd_rn(__fmul_rn(cs, cs), __fmul_rn(ds, ds));
            tB = __fadd_rn(__fmul_rn(cr, cr), __fmul_rn(dr, dr));
            const float first = sqrt_approx(fmaf(tA, smin, tmin)) + sqrt_approx(fmaf(tB, smin, tmin));
            keep = !(first > a.tend);
            ok = in_range(tA, 9.313226e-10f, 1.7592186e13f) && in_range(tB, 9.313226e-10f, 1.7592186e13f);
        }
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        const bool fast = okTables && __all_sync(0xffffffffu, ok || !keep);
        if (fast && keep) {
            const int p = __popc(kept & ((1u << lane) - 1u));
            tab[4 * (p >> 1) + (p & 1)] = tA;
            tab[4 * (p >> 1) + 2 + (p & 1)] = tB;
            // bits(floor) = kMagicBits + it: the row address carries the offset (mod 2^32)
            tabRow[p] = smem0 + rows + (unsigned)(lane * g.stride) * 4u - (unsigned)kMagicBits * 4u;
        }
        __syncwarp();                        // the table is written
        if (!colValid) continue;
        if (fast) {
            const int cnt = __popc(kept), full = cnt >> 1;
            auto step = [&](int e, auto nu) {
                constexpr int N = decltype(nu)::value;
                f2 TA[N], TB[N], v[N][R];
                unsigned r0[N], r1[N];
#pragma unroll
                for (int u = 0; u < N; u++) {
                    const float4 t4 = reinterpret_cast<const float4*>(tab)[e + u];
                    const uint2 rr = reinterpret_cast<const uint2*>(tabRow)[e + u];
                    TA[u] = pk(t4.x, t4.y);
                    TB[u] = pk(t4.z, t4.w);
                    r0[u] = rr.x;
                    r1[u] = rr.y;
                }
#pragma unroll
                for (int u = 0; u < N; u++) ref_packs<R>(TA[u], TB[u], nSL, nTQ, k, r0[u], r1[u], v[u]);
#pragma unroll
                for (int u = 0; u < N; u++)
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        float v0, v1;
                        upk(v[u][r], v0, v1);
                        acc[r] = __fadd_rn(__fadd_rn(acc[r], v0), v1);
                    }
            };
            int e = 0;
            for (; e + U <= full; e += U) step(e, std::integral_constant<int, U>());
            if constexpr (U > 1)
                for (; e < full; e++) step(e, std::integral_constant<int, 1>());
            if (cnt & 1) {                   // a last trace by itself: its second half is dropped
                const float tA1 = tab[4 * full], tB1 = tab[4 * full + 2];
                const unsigned r0 = tabRow[cnt - 1];
                f2 v[R];
                ref_packs<R>(pk(tA1, tA1), pk(tB1, tB1), nSL, nTQ, k, r0, r0, v);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    float v0, v1;
                    upk(v[r], v0, v1);
                    acc[r] = __fadd_rn(acc[r], v0);
                }
            }
        } else {
            for (unsigned m = kept; m; m &= m - 1u) {
                const int c = __ffs(m) - 1;
                const float sA = __shfl_sync(0xffffffffu, tA, c), sB = __shfl_sync(0xffffffffu, tB, c);
                const float* tr = reinterpret_cast<const float*>(smem_raw + rows) + (size_t)c * g.stride;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const int l = run0 + lane + 32 * r, lc = l < g.nz ? l : g.nz - 1;
                    const float zz = __fadd_rn(g.z0, __fmul_rn(__int2float_rn(lc), g.dz));
                    float nsl, unused;
                    upk(nSL[r], nsl, unused);
                    acc[r] = slow_pair(acc[r], sA, sB, __fmul_rn(zz, zz), -nsl, g.dt, g.nt, tr);
                }
            }
        }
    }

    if (colValid) {
        float* out = a.image + (size_t)col * g.nz;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int l = run0 + lane + 32 * r;
            const float zz = __fadd_rn(g.z0, __fmul_rn(__int2float_rn(l < g.nz ? l : g.nz - 1), g.dz));
            // tau = 0: every term is multiplied by zero (+0 or NaN)
            if (__fmul_rn(zz, zz) == 0.0f) acc[r] = __fadd_rn(__fmul_rn(acc[r], 0.0f), 0.0f);
            if (l < g.nz) out[l] = a.accumulate ? __fadd_rn(out[l], acc[r]) : acc[r];
        }
    }
}

// traces per stage: as many as fit `perSm` CTAs of `warps` warps into an SM (at least one):
// ref_smem rounded up and solved for the chunk
int ref_chunk(const Geometry& g, int warps, int perSm)
{
    const long long room = kRefSmem / perSm - 1024 - 62 - 36 * warps;
    return (int)std::max(1LL, std::min<long long>(kRefMaxChunk, room / (8LL * g.stride + 32 + 12 * warps)));
}

// Work split of a launch: samples per lane, warps (columns) per CTA, CTAs per SM.
struct RefSplit {
    int R, warps, perSm;
    float cost;
};

// Every image sample keeps its traces in reference order, so the traces cannot be split
// across CTAs: the image alone fills the GPU, and each SM works through the CTAs that fall
// to it.  The split with the least estimated time of the busiest SM is taken, in cycles a
// trace of one scheduler: s = the warps it holds; a trace takes 50 cycles per warp and sample
// of a lane (60 at one sample, 54 at two: table loads and loop), at least 110 for the
// latency of one warp's chain, and a chunk about 70 s + 200 for its geometry and barrier.
// 256 x 1001 image, 16,384 traces of 1001 samples: R = 4 in 15 warps 7.2 ms (4 waves of
// warps on the busiest scheduler), R = 2 in 29 7.0, in 24 10.7 (a second round for 12 SMs),
// R = 1 in 28 10.1 (three rounds).  437 x 401, 3001 traces: R = 4 in 12 warps 0.88 ms,
// R = 2 in 11 0.94, R = 1 in 14 1.00.
RefSplit ref_split(const Geometry& g, int R, int sm)
{
    const long long cols = (long long)g.nx * g.ny;
    RefSplit best = {4, 1, 1, 3.0e38f};
    for (int r : {4, 2, 1}) {
        if (R != 0 && r != R) continue;
        const int cap = r == 4 ? RefShape<4>::kWarpsPerSm : RefShape<1>::kWarpsPerSm;
        const long long runs = (g.nz + 32LL * r - 1) / (32 * r);
        for (int w = 1; w <= cap && w <= cols; w++) {
            // two stages of one trace and the warps' tables must fit a CTA (one warp's always do)
            if (w > 1 && ref_smem(1, g.stride, g.nt, w).total > (size_t)kMaxSmemBytes) break;
            const long long ctas = (cols + w - 1) / w * runs, load = (ctas + sm - 1) / sm;
            // CTAs of an SM at a time, by registers and by two stages of a trace each
            int perSm = (int)std::min<long long>(cap / w, load);
            while (perSm > 1 && (ref_smem(1, g.stride, g.nt, w).total + 1024) * perSm > (size_t)kRefSmem) perSm--;
            const int chunk = ref_chunk(g, w, perSm);
            auto round = [&](int n) {
                const float s = (float)((n * w + 3) / 4);
                const float c = r == 1 ? 60.0f : r == 2 ? 54.0f : 50.0f;
                return r * std::max(c * s, 110.0f) + (70.0f * s + 200.0f) / chunk;
            };
            const float cost = (float)(load / perSm) * round(perSm) +
                               (load % perSm ? round((int)(load % perSm)) : 0.0f);
            if (cost <= best.cost) best = RefSplit{r, w, perSm, cost};
        }
    }
    return best;
}

template <int R>
int launch_r(RefArgs a, const RefSplit& sp, cudaStream_t stream)
{
    const Geometry& g = a.g;
    a.chunk = ref_chunk(g, sp.warps, sp.perSm);
    const size_t smem = ref_smem(a.chunk, g.stride, g.nt, sp.warps).total;
    auto kern = reference_kernel<R>;
    KTM_CUDA_TRY(allow_smem(kern, smem));
    const long long cols = (long long)g.nx * g.ny;
    const long long groups = (cols + sp.warps - 1) / sp.warps;
    const long long grid = groups * ((g.nz + 32LL * R - 1) / (32 * R));
    if (grid > 0x7fffffffLL)
        return set_error(KTM_ERR_LIMIT, "reference kernel: Nz=%d too large", g.nz);
    a.colGroups = (int)groups;
    kern<<<(unsigned)grid, sp.warps * 32, smem, stream>>>(a);
    KTM_CUDA_TRY(cudaGetLastError());
    return KTM_OK;
}

}  // namespace

int launch_reference(const Geometry& g, const float* midX, const float* midY, const float* offX,
                     const float* offY, const float* traces, const float* vel, float* image,
                     int accumulate, int tileRun, cudaStream_t stream)
{
    if ((long long)g.nx * g.ny * g.nz == 0) return KTM_OK;
    if (g.ntr == 0) {
        if (!accumulate)
            KTM_CUDA_TRY(cudaMemsetAsync(image, 0,
                                         sizeof(float) * (size_t)g.nx * g.ny * g.nz, stream));
        return KTM_OK;
    }
    // two stages of at least one trace
    if ((kMaxSmemBytes - 1024) / (2 * ((size_t)g.nt * sizeof(float) + sizeof(float4))) < 1)
        return set_error(KTM_ERR_LIMIT,
                         "reference kernel: tracePts=%d exceeds the shared-memory stage "
                         "limit (%d samples)", g.nt, (int)((kMaxSmemBytes - 1024) / 8 - 4));
    const int run = tileRun > 0 ? tileRun / 32 : 0;
    if (run != 0 && run != 1 && run != 2 && run != 4 && run != 8 && run != 16)
        return set_error(KTM_ERR_ARG, "reference kernel: tileRun must be 32, 64, 128, 256 or 512");
    int dev = 0, sm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
    // runs of more than 128 samples take 128
    const RefSplit sp = ref_split(g, std::min(run, 4), sm);
    RefArgs a;
    a.g = g; a.midX = midX; a.midY = midY; a.offX = offX; a.offY = offY;
    a.traces = traces; a.vel = vel; a.image = image; a.accumulate = accumulate;
    a.chunk = a.colGroups = 0;
    a.fastDt = g.dt >= 9.5367431640625e-07f && g.dt <= 1024.0f;
    a.rdt = 1.0f / g.dt;
    a.nzero = -0.0f;
    a.tend = (float)g.nt * g.dt * 1.00001f;
    switch (sp.R) {
        case 1: return launch_r<1>(a, sp, stream);
        case 2: return launch_r<2>(a, sp, stream);
        default: return launch_r<4>(a, sp, stream);
    }
}

}  // namespace ktm
