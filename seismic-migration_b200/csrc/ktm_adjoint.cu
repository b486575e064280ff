// ktm_adjoint.cu -- Kirchhoff demigration: the exact transpose of the fast
// migration operator (ktm_fast.cu) for its linear and truncating picks and
// its table / sqrt weights.  The reference has no adjoint; this operator is
// what least-squares migration (ktm_lsm.cu) and the dot-product test need.
//
// Migration (linear pick):  I[p] = |tau_p| sum_k s_k W_pk (q_k[i0] + f (q_k[i0+1] - q_k[i0]))
// Demigration:              D_k[i0]   += W_pk |tau_p| m[p] (1 - f)
//                           D_k[i0+1] += W_pk |tau_p| m[p] f          (0 < j < tracePts only)
// With the prefolded weight the migration reads q_k[j] sqrt(j dt) and W_pk = 1, so the
// demigration scatters without a weight and multiplies D_k[j] by sqrt(j dt) once per
// sample as it writes the chunk out.
// Every pair's (u, f, i0, W) comes from the same code as the migration's
// (ktm_pair.cuh), so the two operators are transposes pair by pair.
//
// Work decomposition: a CTA owns a chunk of traces, accumulates their samples
// in shared memory (padded rows, red.shared.add) while its warps sweep the image columns of
// its column block, and writes the chunk out once (plain stores when one block
// covers all columns, red.global.add otherwise).  A warp covers one column x a
// run of 32*R tau samples at a time; the model samples, the tau tables and the
// velocity of the run stay in registers for all the chunk's traces.  FP32
// shared atomics run at ~7 per clock per SM on distinct addresses and serialise
// on equal ones, so each lane merges its own contributions before issuing them
// (demigrate_merge_kernel).
#include "ktm_pair.cuh"

#include <algorithm>
#include <cstring>

namespace ktm {
namespace {

using namespace dev;

// One CTA of 32 warps per SM, 8 tau samples per lane: each FP32 shared reduction
// is a load / compare-and-swap loop, so more warps hide more of its latency; 8
// samples a lane keep the tau tables small enough for 64 registers.  The chunk's
// accumulators get 220 KB (up to 32 traces, the lane-parallel geometry's limit).
// On the 512 x 1001 line of 32,768 traces, prefolded / table weight, padded rows:
// 32 x 1, R = 8, a padding word per 4 samples 14.8 / 18.6 ms, per 8 samples 14.9 /
// 18.9; 16 x 2 15.6 / 19.6; 24 x 1, R = 16 (80 registers) 17.3 / 21.9.  Unpadded
// rows with the lanes' visiting order rotated against bank conflicts: 32 x 1, R = 8
// 19.9 / 23.6; R = 16 (spilling) 19.6 / 25.1; 20 x 2 19.8 / 24.5; 24 x 1, R = 16
// 21.7 / 26.0; 8 x 3 (72 KB) 23.6 / 27.7.
constexpr int kAdjWarps = 32;
constexpr int kAdjThreads = kAdjWarps * 32;
constexpr int kAdjR = 8;                 // tau samples per lane per run
constexpr int kAdjMinBlocks = 1;
constexpr int kPadShift = 2;             // one padding word per 4 samples
constexpr size_t kAdjSmemBudget = 220 * 1024;
static_assert(kAdjMinBlocks * (kAdjSmemBudget + 1024) <= 228 * 1024,
              "the CTAs must fit the SM's 228 KB of shared memory");

// Accumulator rows and the weight table hold sample j at word j + (j >> kPadShift).
// At one step of the scatter the lanes of a warp sit R = 8 tau samples apart, so
// their target samples lie about 8 u' apart (u' = d(t/dt)/dtau in samples per tau
// sample, 1 at zero offset and less with offset): without padding, multiples of 4 or 8
// words that share a few banks.  The padding word per 4 samples spreads them.  A row
// of n holds every j <= n + 1; rounded up to 4 words so that the arrays after the rows
// stay 16-byte aligned.
__host__ __device__ __forceinline__ int padded_pitch(int n) { return (n + (n >> kPadShift) + 2 + 3) & ~3; }

struct AdjArgs {
    Geometry g;
    const float *midX, *midY, *offX, *offY;
    const float* vel; int velCube;
    const float* image;      // model m [nx*ny][nz]
    float* data;             // [ntr][pitch] F32
    int pitch;
    int pick, weightMethod;
    float aperture;
    int chunk;               // traces per CTA
    int colsPerBlock;        // image columns per CTA (gridDim.y blocks)
    int atomicOut;           // 1: red.global.add into data (several column blocks)
};

// Volatile, so the scatter stays between the barriers around the sweep; no
// "memory" clobber, so the arithmetic around it still schedules freely.
__device__ __forceinline__ void red_shared(unsigned addr, float v)
{
    asm volatile("red.shared.add.f32 [%0], %1;" ::"r"(addr), "f"(v));
}
// The same, issued only where `on` holds: a predicated instruction, no branch.
__device__ __forceinline__ void red_shared_if(bool on, unsigned addr, float v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.shared.add.f32 [%0], %1;\n\t}"
                 ::"r"(addr), "f"(v), "r"((unsigned)on));
}

// Lane-private merge of the scatter: lane L owns the R = kAdjR CONSECUTIVE tau
// samples run0 + R L + i of a run and visits them in increasing tau, so for one
// trace the target sample floor(u) mostly advances by 0 or 1.  The lane walks them
// keeping a running (sample, value, value of the next sample) and issues an atomic
// only when it leaves a sample: one red.shared per pair where u advances by a sample,
// fewer where it stalls (shallow, far offsets), two where it jumps by two or more or
// steps back (a steep Vrms increase at large offsets).  (Visiting the samples in a
// lane-rotated order instead, against bank conflicts on unpadded rows, made every
// lane jump once per run and took a third more time: 19.9 against 14.8 ms.)
// WT: 0 sqrt(j dt) table interpolated per pair, 1 sqrt.approx per pair,
//     2 prefolded (sqrt(j dt) per output sample at the write-out).
template <int PICK, int WT>
__global__ void __launch_bounds__(kAdjThreads, kAdjMinBlocks)
demigrate_merge_kernel(AdjArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Geometry& g = a.g;
    const int pitchP = padded_pitch(a.pitch);
    float* acc = reinterpret_cast<float*>(smem_raw);                    // [chunk][pitchP]
    float* crd = acc + (size_t)a.chunk * pitchP;                        // [4][chunk]
    float2* wtab = reinterpret_cast<float2*>(crd + 4 * a.chunk + ((4 * a.chunk) & 1));  // padded [nt+1]

    const int k0 = blockIdx.x * a.chunk;
    const int n = min(a.chunk, g.ntr - k0);
    for (int i = threadIdx.x; i < a.chunk * pitchP; i += kAdjThreads) acc[i] = 0.0f;
    for (int i = threadIdx.x; i < n; i += kAdjThreads) {
        crd[i] = a.midX[k0 + i];
        crd[a.chunk + i] = a.midY[k0 + i];
        crd[2 * a.chunk + i] = a.offX[k0 + i];
        crd[3 * a.chunk + i] = a.offY[k0 + i];
    }
    if (WT == 0) {
        for (int j = threadIdx.x; j <= g.nt; j += kAdjThreads) {
            const float w0 = sqrtf((float)j * g.dt), w1 = sqrtf((float)(j + 1) * g.dt);
            wtab[j + (j >> kPadShift)] = make_float2(w0, w1 - w0);
        }
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ncols = g.nx * g.ny;
    const int cb0 = blockIdx.y * a.colsPerBlock;
    const int cb1 = min(ncols, cb0 + a.colsPerBlock);
    const float invdt = 1.0f / g.dt;
    const float umax = (float)g.nt;
    const float ap2 = a.aperture > 0.0f ? a.aperture * a.aperture : -1.0f;
    const f2 M2 = pk(kMagic, kMagic);
    // bits(fl) = K + i0, K = kMagicBits a multiple of 4: the padded word of sample i0 is
    // q + (q >> kPadShift) - kPad, kPad = K + (K >> kPadShift); the row bases carry -kPad
    const unsigned kPad = (unsigned)kMagicBits + ((unsigned)kMagicBits >> kPadShift);
    const unsigned accS = smem_u32(acc) - kPad * 4u;
    const unsigned wS = smem_u32(wtab) - kPad * 8u;
    const int nruns = (g.nz + 32 * kAdjR - 1) / (32 * kAdjR);

    for (int col = cb0 + warp; col < cb1; col += kAdjWarps) {
        const int ci = col / g.ny, cj = col % g.ny;
        const float cx = g.x0 + (float)ci * g.dx, cy = g.y0 + (float)cj * g.dy;
        for (int run = 0; run < nruns; run++) {
            const int base = run * 32 * kAdjR + kAdjR * lane;      // the lane's first sample
            f2 T2[kAdjR / 2], S2[kAdjR / 2], MT[kAdjR / 2];
            float t2min = 3.0e38f, smin = 3.0e38f;
            bool any = false;
#pragma unroll
            for (int h = 0; h < kAdjR / 2; h++) {
                float tv[2], sv[2], mv[2];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int l = base + 2 * h + e;
                    const bool ok = l < g.nz;
                    const int lc = ok ? l : g.nz - 1;
                    const float tau = g.z0 + (float)lc * g.dz;
                    const float tq = tau * invdt;
                    const float v = a.velCube ? a.vel[(size_t)col * g.nz + lc] : a.vel[lc];
                    const float vd = v * g.dt;
                    tv[e] = tq * tq;
                    sv[e] = 1.0f / (vd * vd);
                    mv[e] = ok ? fabsf(tau) * a.image[(size_t)col * g.nz + l] : 0.0f;
                    if (ok) { t2min = fminf(t2min, tv[e]); smin = fminf(smin, sv[e]); }
                    any |= (mv[e] != 0.0f);
                }
                T2[h] = pk(tv[0], tv[1]);
                S2[h] = pk(sv[0], sv[1]);
                MT[h] = pk(mv[0], mv[1]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                t2min = fminf(t2min, __shfl_xor_sync(0xffffffffu, t2min, o));
                smin = fminf(smin, __shfl_xor_sync(0xffffffffu, smin, o));
            }
            if (!__any_sync(0xffffffffu, any)) continue;        // zero model in this run
            // lane c evaluates trace c's geometry for this column and run (chunk <= 32):
            // squared source / receiver distances and the keep flag (aperture, and a
            // lower bound of u over the run below the trace end); the warp then walks
            // the kept traces in increasing c, taking their distances by shuffle
            float lds_ = 0.0f, ldr_ = 0.0f;
            bool keep = false;
            if (lane < n) {
                const float mx = crd[lane], my = crd[a.chunk + lane], ox = crd[2 * a.chunk + lane],
                            oy = crd[3 * a.chunk + lane];
                const float dmx = mx - cx, dmy = my - cy;
                keep = !(ap2 >= 0.0f && dmx * dmx + dmy * dmy > ap2);
                const float sx = dmx - ox, sy = dmy - oy, rx = dmx + ox, ry = dmy + oy;
                lds_ = sx * sx + sy * sy;
                ldr_ = rx * rx + ry * ry;
                if (keep) {
                    const float ulb = sqrt_approx(fmaf(lds_, smin, t2min)) +
                                      sqrt_approx(fmaf(ldr_, smin, t2min));
                    keep = ulb < umax * 1.0001f + 1.0f;          // not past the trace end
                }
            }
            for (unsigned kept = __ballot_sync(0xffffffffu, keep); kept; kept &= kept - 1u) {
                const int c = __ffs(kept) - 1;
                const float ds = __shfl_sync(0xffffffffu, lds_, c);
                const float dr = __shfl_sync(0xffffffffu, ldr_, c);
                const unsigned rowS = accS + (unsigned)(c * pitchP) * 4u;
                const f2 DS = pk(ds, ds), DR = pk(dr, dr);
                unsigned qc = 0u, pc = 0u;
                float va = 0.0f, vb = 0.0f;
#pragma unroll
                for (int h = 0; h < kAdjR / 2; h++) {
                    const PairKin kk = pair_kin(DS, DR, S2[h], T2[h], umax, M2);
                    const unsigned pp0 = kk.q0 + (kk.q0 >> kPadShift), pp1 = kk.q1 + (kk.q1 >> kPadShift);
                    f2 VAL;
                    if (WT == 0) {
                        const float2 w0 = lds_f2(wS + pp0 * 8u), w1 = lds_f2(wS + pp1 * 8u);
                        VAL = mul2(fma2(kk.F, pk(w0.y, w1.y), pk(w0.x, w1.x)), MT[h]);
                    } else if (WT == 1) {
                        VAL = mul2(mul2(pk(sqrt_approx(kk.u0), sqrt_approx(kk.u1)),
                                        pk(sqrtf(g.dt), sqrtf(g.dt))),
                                   MT[h]);
                    } else {
                        VAL = MT[h];
                    }
                    float ca[2], cb[2];
                    if (PICK == KTM_PICK_LINEAR) {
                        const f2 B = mul2(VAL, kk.F);          // f * val       -> sample i0 + 1
                        const f2 A = sub2(VAL, B);             // (1 - f) * val -> sample i0
                        upk(A, ca[0], ca[1]);
                        upk(B, cb[0], cb[1]);
                    } else {
                        upk(VAL, ca[0], ca[1]);
                        cb[0] = cb[1] = 0.0f;
                    }
                    const unsigned qs[2] = {kk.q0, kk.q1}, ps[2] = {pp0, pp1};
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const unsigned q = qs[e];
                        if (h == 0 && e == 0) {
                            qc = q; pc = ps[0]; va = ca[0]; vb = cb[0];
                            continue;
                        }
                        const bool same = q == qc;
                        const bool next = q == qc + 1u;
                        red_shared_if(!same, rowS + pc * 4u, va);
                        if (PICK == KTM_PICK_LINEAR) {
                            // sample qc + 1 is flushed here only where u jumped by two or more
                            const unsigned qn = qc + 1u;
                            red_shared_if(!same && !next, rowS + (qn + (qn >> kPadShift)) * 4u, vb);
                        }
                        va = same ? va + ca[e] : (next ? vb + ca[e] : ca[e]);
                        vb = same ? vb + cb[e] : cb[e];
                        qc = q;
                        pc = ps[e];
                    }
                }
                red_shared(rowS + pc * 4u, va);
                if (PICK == KTM_PICK_LINEAR) {
                    const unsigned qn = qc + 1u;
                    red_shared(rowS + (qn + (qn >> kPadShift)) * 4u, vb);
                }
            }
        }
    }
    asm volatile("" ::: "memory");     // the scatter wrote acc: no load below reuses older values
    __syncthreads();
    for (int i = threadIdx.x; i < n * a.pitch; i += kAdjThreads) {
        const int c = i / a.pitch, j = i % a.pitch;
        float v = (j > 0 && j < g.nt) ? acc[(size_t)c * pitchP + j + (j >> kPadShift)] : 0.0f;
        if (WT == 2) v *= sqrtf((float)j * g.dt);        // the fold's factor (ktm_prep.cu, ktm_lsm.cu)
        float* dst = a.data + (size_t)(k0 + c) * a.pitch + j;
        if (a.atomicOut) {
            if (v != 0.0f) atomicAdd(dst, v);
        } else {
            *dst += v;
        }
    }
}

// ---------------------------------------------------------------------------
// Demigration with a row per warp: linear pick, 1-D velocity, traces short enough that
// sixteen rows fit an SM.
//
// A warp owns one trace (of the column block blockIdx.y): it accumulates the trace into a
// row of its own in shared memory while it sweeps runs of 256 tau samples and, for each run,
// the columns, lane c evaluating 32 columns' geometry at a time.  T2', S' of the run stay in
// registers over all columns (1-D velocity); |tau| m comes from a copy that a first kernel
// laid out so that a lane's 8 samples are two 16-byte loads (zero runs are flagged there).
//
// No other warp writes the row, so where two lanes cannot meet either, a flush is a plain
// load, add and store instead of a compare-and-swap loop.  Lane L owns samples 8 L .. 8 L + 7
// of the run and flushes sample floor(u) when u leaves it.  With all 8 indices at hand the
// warp looks whether in every lane floor(u) stays or goes on by one from each sample to the
// next, and whether the next lane is ahead at every step (past the trace end they may meet:
// those words are dropped).  If so each step's flushes hit different words, and one
// comparison a sample does the merge.  Elsewhere (shallow runs, where 8 samples may share a
// trace sample; steep steps) it takes the merge of demigrate_merge_kernel with shared
// reductions.
// 512 x 1001 image, 32,768 traces of 1001 samples, prefolded / table / sqrt weight:
// 11.4 / 18.0 / 12.5 ms, against 14.7 / 18.5 / 15.4 with rows shared by the CTA; 100 columns,
// 2000 traces 0.32 / 0.44 against 0.56 / 0.60.  Bound by issue (35 instructions a pair, three
// quarters of the slots) and by the shared-memory pipe.  At 64 registers it spills (36 / 60 / 20
// bytes stored, 92 / 124 / 76 loaded).
constexpr int kRowR = 8;
constexpr int kRowRun = 32 * kRowR;
// Warps per CTA, up to 32 warps per SM: small CTAs end at their own pace (512 x 1001 image,
// 32,768 traces, prefolded: 11.3 ms in CTAs of 8 warps, 12.2 in CTAs of 32); with the weight
// table, of which every CTA holds a copy, 16 (18.7 ms in CTAs of 8, 18.0 in CTAs of 16).
template <int WT>
constexpr int kRowWarps = WT == 0 ? 16 : 8;

struct RowArgs {
    AdjArgs a;
    const float* mt;              // |tau| m, [ncols][nruns][2][32][4]
    const unsigned char* live;    // [ncols][nruns]: a sample of the run is not zero
    int nruns, accumulate;
};

__host__ __device__ __forceinline__ int row_words(int nt) { return padded_pitch(nt + 2); }

// |tau| m and the non-zero flags, one warp per (column, run)
__global__ void __launch_bounds__(256) row_model_kernel(AdjArgs a, int nruns, float* __restrict__ mt,
                                                        unsigned char* __restrict__ live)
{
    const Geometry& g = a.g;
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (w >= (long long)g.nx * g.ny * nruns) return;
    const long long col = w / nruns;
    const int run = (int)(w - col * nruns);
    bool any = false;
#pragma unroll
    for (int i = 0; i < kRowR; i++) {
        const int x = 32 * i + lane;                       // sample of the run
        const int l = run * kRowRun + x;
        const float tau = g.z0 + (float)l * g.dz;
        const float v = l < g.nz ? fabsf(tau) * a.image[col * g.nz + l] : 0.0f;
        any |= v != 0.0f;
        // lane x / 8, half (x / 4) % 2, word x % 4
        mt[w * kRowRun + ((x >> 2) & 1) * 128 + (x >> 3) * 4 + (x & 3)] = v;
    }
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) live[w] = any;
}

// T2' and S' of tau sample l: past the image T2' goes on and S' stays
__device__ __forceinline__ void row_tables(const AdjArgs& a, int l, float invdt, float& t2, float& s)
{
    const Geometry& g = a.g;
    const float tq = (g.z0 + (float)l * g.dz) * invdt;
    const float vd = a.vel[l < g.nz ? l : g.nz - 1] * g.dt;
    t2 = tq * tq;
    s = 1.0f / (vd * vd);
}

// row[addr] += v where `on` holds: predicated, so the warp stays converged
__device__ __forceinline__ void add_shared_if(bool on, unsigned addr, float v)
{
    asm volatile("{\n\t.reg .pred p;\n\t.reg .f32 t;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.f32 t, [%0];\n\t"
                 "@p add.f32 t, t, %1;\n\t@p st.shared.f32 [%0], t;\n\t}"
                 ::"r"(addr), "f"(v), "r"((unsigned)on));
}
__device__ __forceinline__ void add_shared(unsigned addr, float v)
{
    asm volatile("{\n\t.reg .f32 t;\n\tld.shared.f32 t, [%0];\n\tadd.f32 t, t, %1;\n\tst.shared.f32 [%0], t;\n\t}"
                 ::"r"(addr), "f"(v));
}

// word (in bytes) of the sample whose bits(fl) = q, relative to the row's shifted base
__device__ __forceinline__ unsigned padded_bytes(unsigned q) { return (q + (q >> kPadShift)) * 4u; }

template <int WT>
__global__ void __launch_bounds__(kRowWarps<WT> * 32, 32 / kRowWarps<WT>) demigrate_row_kernel(RowArgs ra)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const AdjArgs& a = ra.a;
    const Geometry& g = a.g;
    constexpr int warps = kRowWarps<WT>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int words = row_words(g.nt);
    // [warps] rows, [warps][32] entries, [nruns] least T2' and S', the padded weight table
    float* row = reinterpret_cast<float*>(smem_raw) + (size_t)warp * words;
    float4* tab = reinterpret_cast<float4*>(smem_raw + (size_t)warps * words * 4) + warp * 32;
    float2* least = reinterpret_cast<float2*>(smem_raw + (size_t)warps * (words * 4 + 512));
    float2* wtab = least + (ra.nruns + 1) / 2 * 2;
    const float invdt = 1.0f / g.dt;

    for (int i = lane; i < words; i += 32) row[i] = 0.0f;
    for (int run = warp; run < ra.nruns; run += warps) {
        float t2 = 3.0e38f, sl = 3.0e38f;
        for (int i = 0; i < kRowR; i++) {
            const int l = run * kRowRun + 32 * i + lane;
            float t0, s0;
            row_tables(a, l, invdt, t0, s0);
            if (l < g.nz) {
                t2 = fminf(t2, t0);
                sl = fminf(sl, s0);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            t2 = fminf(t2, __shfl_xor_sync(0xffffffffu, t2, o));
            sl = fminf(sl, __shfl_xor_sync(0xffffffffu, sl, o));
        }
        if (lane == 0) least[run] = make_float2(t2, sl);
    }
    if (WT == 0) {
        for (int j = threadIdx.x; j <= g.nt; j += blockDim.x) {
            const float w0 = sqrtf((float)j * g.dt), w1 = sqrtf((float)(j + 1) * g.dt);
            wtab[j + (j >> kPadShift)] = make_float2(w0, w1 - w0);
        }
    }
    __syncthreads();

    const int k = blockIdx.x * warps + warp;
    if (k >= g.ntr) return;
    const float mx = a.midX[k], my = a.midY[k], ox = a.offX[k], oy = a.offY[k];
    const int cb0 = blockIdx.y * a.colsPerBlock, cb1 = min(g.nx * g.ny, cb0 + a.colsPerBlock);
    const float umax = (float)g.nt, upast = umax * 1.0001f + 1.0f;
    const float ap2 = a.aperture > 0.0f ? a.aperture * a.aperture : -1.0f;
    const f2 M2 = pk(kMagic, kMagic);
    // bits(fl) = K + i0, K a multiple of 4: the bases carry -padded(K)
    const unsigned kPad = (unsigned)kMagicBits + ((unsigned)kMagicBits >> kPadShift);
    const unsigned rowS = smem_u32(row) - kPad * 4u;
    const unsigned wS = smem_u32(wtab) - kPad * 8u;
    const unsigned qEnd = (unsigned)kMagicBits + (unsigned)g.nt;
    const float rootDt = sqrtf(g.dt);

    for (int run = 0; run < ra.nruns; run++) {
        f2 T2[kRowR / 2], S2[kRowR / 2];
#pragma unroll
        for (int h = 0; h < kRowR / 2; h++) {
            float t[2], s[2];
#pragma unroll
            for (int e = 0; e < 2; e++) row_tables(a, run * kRowRun + kRowR * lane + 2 * h + e, invdt, t[e], s[e]);
            T2[h] = pk(t[0], t[1]);
            S2[h] = pk(s[0], s[1]);
        }
        for (int cb = cb0; cb < cb1; cb += 32) {
            // lane c: column cb + c
            float ds = 0.0f, dr = 0.0f;
            bool keep = false;
            const int col = cb + lane;
            if (col < cb1) {
                const int ci = col / g.ny, cj = col - ci * g.ny;
                const float dmx = mx - (g.x0 + (float)ci * g.dx), dmy = my - (g.y0 + (float)cj * g.dy);
                const float sx = dmx - ox, sy = dmy - oy, rx = dmx + ox, ry = dmy + oy;
                ds = sx * sx + sy * sy;
                dr = rx * rx + ry * ry;
                // aperture, a zero model, a first sample past the trace end
                const float2 m = least[run];
                keep = !(ap2 >= 0.0f && dmx * dmx + dmy * dmy > ap2) && ra.live[(size_t)col * ra.nruns + run] &&
                       sqrt_approx(fmaf(ds, m.y, m.x)) + sqrt_approx(fmaf(dr, m.y, m.x)) < upast;
            }
            const unsigned kept = __ballot_sync(0xffffffffu, keep);
            if (keep) tab[__popc(kept & ((1u << lane) - 1u))] = make_float4(ds, dr, __int_as_float(col), 0.0f);
            __syncwarp();
            const int cnt = __popc(kept);
            for (int e = 0; e < cnt; e++) {
                const float4 t = tab[e];
                const float4* m4 = reinterpret_cast<const float4*>(
                    ra.mt + ((size_t)__float_as_int(t.z) * ra.nruns + run) * kRowRun) + lane;
                const float4 ma = __ldg(m4), mb = __ldg(m4 + 32);
                const f2 DS = pk(t.x, t.x), DR = pk(t.y, t.y);
                const f2 MT[4] = {pk(ma.x, ma.y), pk(ma.z, ma.w), pk(mb.x, mb.y), pk(mb.z, mb.w)};
                unsigned q[kRowR];
                float ca[kRowR], cb_[kRowR];       // to samples floor(u) and floor(u) + 1
#pragma unroll
                for (int h = 0; h < kRowR / 2; h++) {
                    const PairKin kk = pair_kin(DS, DR, S2[h], T2[h], umax, M2);
                    q[2 * h] = kk.q0;
                    q[2 * h + 1] = kk.q1;
                    f2 VAL = MT[h];
                    if (WT == 0) {
                        const float2 w0 = lds_f2(wS + 2u * padded_bytes(kk.q0)), w1 = lds_f2(wS + 2u * padded_bytes(kk.q1));
                        VAL = mul2(fma2(kk.F, pk(w0.y, w1.y), pk(w0.x, w1.x)), MT[h]);
                    } else if (WT == 1) {
                        VAL = mul2(mul2(pk(sqrt_approx(kk.u0), sqrt_approx(kk.u1)), pk(rootDt, rootDt)), MT[h]);
                    }
                    const f2 B = mul2(VAL, kk.F);          // f * val       -> sample i0 + 1
                    const f2 A = sub2(VAL, B);             // (1 - f) * val -> sample i0
                    upk(A, ca[2 * h], ca[2 * h + 1]);
                    upk(B, cb_[2 * h], cb_[2 * h + 1]);
                }
                // steps of at most one sample; the next lane ahead (the last lane has none)
                bool small = true, apart = true;
#pragma unroll
                for (int i = 0; i < kRowR; i++) {
                    const unsigned n = __shfl_down_sync(0xffffffffu, q[i], 1);
                    apart = apart && (n > q[i] || n == qEnd || lane == 31);
                    if (i > 0) small = small && q[i] - q[i - 1] <= 1u;
                }
                small = __all_sync(0xffffffffu, small);
                float va = ca[0], vb = cb_[0];
                if (__all_sync(0xffffffffu, apart) && small) {
#pragma unroll
                    for (int i = 1; i < kRowR; i++) {
                        const bool on = q[i] != q[i - 1];
                        add_shared_if(on, rowS + padded_bytes(q[i - 1]), va);
                        va = (on ? vb : va) + ca[i];
                        vb = (on ? 0.0f : vb) + cb_[i];
                        __syncwarp();
                    }
                    add_shared(rowS + padded_bytes(q[kRowR - 1]), va);
                    __syncwarp();
                    add_shared(rowS + padded_bytes(q[kRowR - 1] + 1u), vb);
                    __syncwarp();
                } else if (small) {
#pragma unroll
                    for (int i = 1; i < kRowR; i++) {
                        const bool on = q[i] != q[i - 1];
                        red_shared_if(on, rowS + padded_bytes(q[i - 1]), va);
                        va = (on ? vb : va) + ca[i];
                        vb = (on ? 0.0f : vb) + cb_[i];
                    }
                    red_shared(rowS + padded_bytes(q[kRowR - 1]), va);
                    red_shared(rowS + padded_bytes(q[kRowR - 1] + 1u), vb);
                    __syncwarp();
                } else {
#pragma unroll
                    for (int i = 1; i < kRowR; i++) {
                        const unsigned qc = q[i - 1];
                        const bool same = q[i] == qc, next = q[i] == qc + 1u;
                        red_shared_if(!same, rowS + padded_bytes(qc), va);
                        red_shared_if(!same && !next, rowS + padded_bytes(qc + 1u), vb);
                        va = same ? va + ca[i] : (next ? vb + ca[i] : ca[i]);
                        vb = same ? vb + cb_[i] : cb_[i];
                    }
                    red_shared(rowS + padded_bytes(q[kRowR - 1]), va);
                    red_shared(rowS + padded_bytes(q[kRowR - 1] + 1u), vb);
                    __syncwarp();
                }
            }
        }
    }
    asm volatile("" ::: "memory");     // the scatter wrote the row: no load below reuses older values
    __syncwarp();
    float* dst = a.data + (size_t)k * a.pitch;
    for (int j = lane; j < a.pitch; j += 32) {
        float v = (j > 0 && j < g.nt) ? row[j + (j >> kPadShift)] : 0.0f;
        if (WT == 2) v *= sqrtf((float)j * g.dt);        // the fold's factor (ktm_prep.cu, ktm_lsm.cu)
        if (a.atomicOut) {
            if (v != 0.0f) atomicAdd(dst + j, v);
        } else {
            dst[j] = ra.accumulate ? dst[j] + v : v;
        }
    }
}

// Shared memory of a CTA of the row kernel, and how many fit an SM; 0: the job takes the
// shared rows.  Sixteen warps an SM are enough for it (2201 samples: 11.8 ms against 13.4)
// except with the weight table (1501 samples, 16 warps: 29.2 ms against 28.4) and with tau
// steps of more than half a sample, which make most flushes general ones (2201 samples, 16
// warps, 41.0 ms against 28.6; 1001 samples, 32 warps, 10.8 against 10.8; 500 samples 5.3
// against 7.0): those need 32, and never take it both with the table and coarse steps (16.6
// ms against 15.4).
// A few traces give too few warps at one a trace, each with a block of columns to go through in turn,
// where the shared rows bring 32 to a chunk of up to 32 traces: one trace into 100 columns 57 us
// against 28, 8 traces 117 against 73, 12 traces 64 against 84; 24 into 2500 columns, most of them
// out of reach, 117 against 58, 64 into 512 111 against 111, 500 into 50 x 50 columns within reach
// 1.03 ms against 2.02 (table weight).
int row_ctas(const Geometry& g, int wt, size_t* smem)
{
    const int nruns = (g.nz + kRowRun - 1) / kRowRun, warps = wt == 0 ? kRowWarps<0> : kRowWarps<1>;
    *smem = warps * ((size_t)row_words(g.nt) * 4 + 512) + (nruns + 1) / 2 * 16 +
            (wt == 0 ? (size_t)padded_pitch(g.nt + 1) * sizeof(float2) : 0);
    const int ctas = (int)std::min<size_t>(32 / warps, (size_t)(227 * 1024) / (*smem + 1024));
    const bool coarse = !(2.0f * fabsf(g.dz) <= 1.05f * g.dt);
    if (g.nt > 8192 || (wt == 0 && coarse)) return 0;
    if (g.ntr < ((long long)g.nx * g.ny <= 256 ? 10 : 64)) return 0;
    return ctas * warps >= (wt == 0 || coarse ? 32 : 16) ? ctas : 0;
}

template <int WT>
int launch_rows(const RowArgs& ra, dim3 grid, size_t smem, cudaStream_t s)
{
    KTM_CUDA_TRY(allow_smem(demigrate_row_kernel<WT>, smem));
    demigrate_row_kernel<WT><<<grid, kRowWarps<WT> * 32, smem, s>>>(ra);
    KTM_CUDA_TRY(cudaGetLastError());
    return KTM_OK;
}

}  // namespace

size_t demigrate_scratch(const Geometry& g, int velCube, int pick, int weightMethod)
{
    const int wt = weightMethod == KTM_WEIGHT_SQRT ? 1 : weightMethod == KTM_WEIGHT_PREFOLD ? 2 : 0;
    size_t smem;
    if (velCube || pick != KTM_PICK_LINEAR || row_ctas(g, wt, &smem) == 0) return 0;
    const size_t items = (size_t)g.nx * g.ny * ((g.nz + kRowRun - 1) / kRowRun);
    return items * kRowRun * sizeof(float) + (items + 255) / 256 * 256;
}

namespace {

// The row kernel over all traces: one CTA per kRowWarps traces and column block.
int launch_row_demigrate(const Geometry& g, const float* midX, const float* midY, const float* offX,
                         const float* offY, const float* vel, const float* image, float* data, int pitch,
                         int weightMethod, float aperture, int accumulate, void* scratch, int sm, cudaStream_t s)
{
    const int wt = weightMethod == KTM_WEIGHT_SQRT ? 1 : weightMethod == KTM_WEIGHT_PREFOLD ? 2 : 0;
    size_t smem = 0;
    row_ctas(g, wt, &smem);
    const int ncols = g.nx * g.ny, warps = wt == 0 ? kRowWarps<0> : kRowWarps<1>;
    const int groups = (g.ntr + warps - 1) / warps;
    // column blocks where the traces alone give too few CTAs, as many as the shared rows take
    // (six groups of 32 traces per SM), so that both sum the same blocks of columns
    const int chunks = (g.ntr + 31) / 32, want = 6 * sm;
    int blocks = chunks < want ? std::min((want + chunks - 1) / chunks, std::max(1, ncols / 16)) : 1;
    const int perBlock = (ncols + blocks - 1) / blocks;
    blocks = (ncols + perBlock - 1) / perBlock;
    RowArgs ra;
    std::memset(&ra, 0, sizeof(ra));
    AdjArgs& a = ra.a;
    a.g = g; a.midX = midX; a.midY = midY; a.offX = offX; a.offY = offY;
    a.vel = vel; a.image = image; a.data = data; a.pitch = pitch; a.aperture = aperture;
    a.colsPerBlock = perBlock; a.atomicOut = blocks > 1;
    ra.nruns = (g.nz + kRowRun - 1) / kRowRun;
    ra.accumulate = accumulate;
    const size_t items = (size_t)ncols * ra.nruns;
    float* mt = static_cast<float*>(scratch);
    unsigned char* live = reinterpret_cast<unsigned char*>(mt + items * kRowRun);
    ra.mt = mt; ra.live = live;
    if (blocks > 1 && !accumulate)
        KTM_CUDA_TRY(cudaMemsetAsync(data, 0, (size_t)pitch * sizeof(float) * g.ntr, s));
    row_model_kernel<<<(unsigned)((items + 7) / 8), 256, 0, s>>>(a, ra.nruns, mt, live);
    KTM_CUDA_TRY(cudaGetLastError());
    const dim3 grid((unsigned)groups, (unsigned)blocks);
    return wt == 2 ? launch_rows<2>(ra, grid, smem, s)
         : wt == 1 ? launch_rows<1>(ra, grid, smem, s) : launch_rows<0>(ra, grid, smem, s);
}

}  // namespace

int launch_demigrate(const Geometry& g, const float* midX, const float* midY, const float* offX,
                     const float* offY, const float* vel, int velCube, const float* image,
                     float* data, int pitch, int pick, int weightMethod, float aperture,
                     int accumulate, void* scratch, bool mayAllocate, cudaStream_t s)
{
    if (pitch < g.nt + 2 || pitch % 4 != 0)
        return set_error(KTM_ERR_ARG, "demigrate: dataPitch must be >= tracePts + 2 and a multiple of 4");
    const size_t pitchBytes = (size_t)pitch * sizeof(float);
    const bool empty = g.ntr == 0 || (long long)g.nx * g.ny * g.nz == 0;
    int dev = 0, sm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
    const int wt = weightMethod == KTM_WEIGHT_SQRT ? 1 : weightMethod == KTM_WEIGHT_PREFOLD ? 2 : 0;
    // the shared rows' limit is every call's: the kernel with a row per warp may not find its memory.
    // The sqrt(j dt) table only for the table weight; the coordinates' alignment pad
    const size_t fixed = (wt == 0 ? (size_t)padded_pitch(g.nt + 1) * sizeof(float2) : 0) + 64;
    const size_t perTrace = (size_t)padded_pitch(pitch) * sizeof(float) + 4 * sizeof(float);
    if (!empty && fixed + perTrace > (size_t)kMaxSmemBytes)
        return set_error(KTM_ERR_LIMIT, "demigrate: tracePts=%d exceeds the shared-memory limit", g.nt);
    const size_t need = empty ? 0 : demigrate_scratch(g, velCube, pick, weightMethod);
    void* own = nullptr;
    if (need && !scratch && mayAllocate && pool_malloc(&own, need, s) != cudaSuccess) {
        cudaGetLastError();              // no room for the copy of the model: the shared rows
        own = nullptr;
    }
    if (need && (scratch || own)) {
        const int rc = launch_row_demigrate(g, midX, midY, offX, offY, vel, image, data, pitch, weightMethod, aperture,
                                            accumulate, scratch ? scratch : own, sm, s);
        if (own) cudaFreeAsync(own, s);
        return rc;
    }
    if (!accumulate && g.ntr > 0)
        KTM_CUDA_TRY(cudaMemsetAsync(data, 0, pitchBytes * g.ntr, s));
    if (empty) return KTM_OK;
    int chunk = 32;                     // at most 32: lane c evaluates trace c's geometry
    while (chunk > 1 && fixed + chunk * perTrace > kAdjSmemBudget) chunk--;
    const size_t smem = fixed + chunk * perTrace;

    const int ncols = g.nx * g.ny;
    const int chunks = (g.ntr + chunk - 1) / chunk;
    // column blocks only when the traces alone give too few CTAs (then the
    // chunks are added into the data with global atomics)
    int blocks = 1;
    const int want = 6 * sm;
    if (chunks < want) blocks = std::min((want + chunks - 1) / chunks, std::max(1, ncols / 16));
    const int perBlock = (ncols + blocks - 1) / blocks;
    blocks = (ncols + perBlock - 1) / perBlock;

    AdjArgs a;
    a.g = g; a.midX = midX; a.midY = midY; a.offX = offX; a.offY = offY;
    a.vel = vel; a.velCube = velCube; a.image = image; a.data = data; a.pitch = pitch;
    a.pick = pick; a.weightMethod = weightMethod; a.aperture = aperture;
    a.chunk = chunk; a.colsPerBlock = perBlock; a.atomicOut = blocks > 1;
    dim3 grid((unsigned)chunks, (unsigned)blocks);
#define KTM_ADJ_LAUNCH(P, W)                                                                    \
    do {                                                                                        \
        KTM_CUDA_TRY(allow_smem(demigrate_merge_kernel<P, W>, smem));                           \
        demigrate_merge_kernel<P, W><<<grid, kAdjThreads, smem, s>>>(a);                       \
    } while (0)
    if (wt == 2 && pick != KTM_PICK_LINEAR)
        return set_error(KTM_ERR_ARG, "demigrate: the prefolded weight takes the linear pick");
    if (pick == KTM_PICK_LINEAR) {
        if (wt == 2) KTM_ADJ_LAUNCH(KTM_PICK_LINEAR, 2);
        else if (wt) KTM_ADJ_LAUNCH(KTM_PICK_LINEAR, 1);
        else KTM_ADJ_LAUNCH(KTM_PICK_LINEAR, 0);
    } else {
        if (wt) KTM_ADJ_LAUNCH(KTM_PICK_TRUNCATE, 1); else KTM_ADJ_LAUNCH(KTM_PICK_TRUNCATE, 0);
    }
#undef KTM_ADJ_LAUNCH
    KTM_CUDA_TRY(cudaGetLastError());
    return KTM_OK;
}

}  // namespace ktm
