// ktm_fast.cu -- the fast PSTM gather kernel (mixed precision) and the FP64
// device reference.
//
// Method (psktmCPU.c:56-86, extended with linear pick, aperture, a Vrms cube and
// packed FP16 / BF16 / FP32 samples with a per-trace scale):
//   image[x,tau] = |tau| * sum_k  s_k * w(t) * pick(q_k, t/dt)
//   t = sqrt(tau^2 + |s-x|^2 S) + sqrt(tau^2 + |r-x|^2 S),  S = 1/v(x,tau)^2
//   reference weight t*sqrt(tau^2/t) = |tau| sqrt(t) (:85): |tau| per image
//   sample, sqrt(t) per pair (truncating pick) or folded into the samples as
//   sqrt(j dt) by ktmPrepareTraces (linear pick);
//   pick: linear interpolation, or truncation (:80); samples outside
//   0 < j < tracePts are zero guards of the packed layout (:82);
//   pairs with |mid - x| > aperture are skipped.
//
// Input: a PACKED trace set (ktm_prep.cu): [traceNo][pitch] F32/F16/BF16 with
// zero guard samples, a per-trace FP32 scale s_k.
//
// Per (image sample, trace) pair, FP32 with two pairs per packed f32x2 op:
//   a_s = T2' + Ds*S', a_r = T2' + Dr*S'  (T2' = (tau/dt)^2, S' = S/dt^2, so
//                                          the traveltime comes out in samples)
//   u   = sqrt(a_s) + sqrt(a_r)           2 SFU ops (sqrt.approx)
//   u   = min(u, nt)   (also maps NaN to nt, a zero guard)
//   i0  = floor(u) via the round-down add of 1.5*2^23, f = u - i0
//   v   = q[i0] + f (q[i0+1] - q[i0]);  acc += s_k * v
// Work decomposition (148 SMs, 24 warps per SM at 80 registers; the CTA shape
// CtaShape below: 24 columns x one CTA per SM by default, 12 x 2 or 8 x 3):
//   warp   = one image column x a run of 32*R tau samples (lane L owns
//            tau = run0 + L + 32 r): a warp reads a narrow window of a trace;
//   CTA    = W columns (blockIdx.x) x one run (blockIdx.y) x one slice of the
//            traces (blockIdx.z); slices write partial images that a second
//            kernel sums in a fixed order (deterministic), so small images still
//            fill the GPU;
//   traces stream through shared memory in chunks of up to 32, in two or three
//   buffers: one thread moves a chunk's packed rows (one contiguous, 16-byte
//   aligned range) with a single bulk copy (cp.async.bulk) completed on the
//   buffer's mbarrier, which every warp waits on with a one-second bound.  No
//   barrier of the CTA: a warp goes on to the next chunk as soon as it is through
//   with one, and the last warp through refills the buffer.  For each chunk, lane c
//   of every warp reads trace c's coordinates and computes its squared distances,
//   scale and reach (aperture, or a lower bound of u beyond the trace end) for the
//   warp's column; the kept traces go in order into a table of the warp in shared
//   memory, one 16-byte entry each, which the warp then walks.
//   ktmAutotuneTile picks R, the shape and the chunk per job.
// What bounds it: two special-function square roots a pair take 16 cycles of a
// scheduler; the pair loop alone runs at 19 (24 warps, 13 instructions a pair), the
// kernel at 21 to 22 with the chunks' geometry (about 1800 cycles of an SM per chunk),
// the table walk and the CTA's prologue and end.  Against two CTA barriers' worth of
// waiting per chunk, shuffles and a bit search per trace: 200 x 200 x 1501 image, 2500
// FP16 traces 52.7 ms instead of 56.6; 256 x 1001, 16,384 FP16 traces 2.27 ms instead of
// 2.34; 128 x 751, 6144 FP32 traces with the table weight 0.46 ms instead of 0.52.
#include "ktm_pair.cuh"

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

namespace ktm {
namespace {

// CTA shapes of the fast kernels: warps per CTA (one image column each), CTAs per
// SM and dynamic shared memory per CTA.  Every shape runs 24 warps per SM with
// registers capped at 80 (65,536 / 768 threads); MB x (budget + up to 1 KB of
// static shared memory + the 1 KB the SM reserves) fits the SM's 228 KB.  More
// columns per CTA share each staged chunk of traces among more warps: on the
// 200 x 200 x 1501 image, 2500 FP16 traces, 24 x 1 takes 52.7 ms, 12 x 2 54.4 and
// 8 x 3 56.5 per launch.
// Full = 1: every pick / weight / gradient path is built for the shape; 0: the
// linear pick with the prefolded or table weight only (the paths the tile
// tuner searches).
template <int W, int MB, int KB, int FULL>
struct CtaShape {
    static constexpr int kWarps = W;
    static constexpr int kThreads = W * 32;
    static constexpr int kMinBlocks = MB;
    static constexpr size_t kBudget = (size_t)KB * 1024;
    static constexpr bool kFull = FULL != 0;
};
using Shape24 = CtaShape<24, 1, 226, 1>;
using Shape12 = CtaShape<12, 2, 112, 0>;
using Shape8 = CtaShape<8, 3, 74, 0>;
template <class SH>
constexpr bool shape_fits()
{
    return SH::kMinBlocks * (SH::kBudget + 2048) <= 228 * 1024;
}
static_assert(shape_fits<Shape24>() && shape_fits<Shape12>() && shape_fits<Shape8>(),
              "each shape's CTAs must fit the SM's 228 KB of shared memory");
constexpr int kMaxChunk = 32;        // lane c of a warp evaluates trace c of a chunk
constexpr int kMaxStages = 3;
using namespace dev;

// Bound of one wait for a chunk's bulk copy.  A copy of a chunk takes
// microseconds; a wait that runs out marks the tile stalled, counts it in
// g_waitStalls and ends the tile without output (ktmCheckDeviceWaits reports it).
constexpr unsigned long long kBulkWaitNs = 1000000000ull;
__device__ unsigned g_waitStalls;

// Per-CTA state of the chunk pipeline, per row buffer: the mbarrier its copies complete
// on, how many warps are through with its chunk, how many copies it was given.
struct ChunkSync {
    unsigned long long bar[kMaxStages];
    int done[kMaxStages], issued[kMaxStages];
    int stalled;
};
static_assert(sizeof(ChunkSync) + sizeof(FastArgs) + sizeof(int) <= 1024,
              "static shared memory of the fast kernels within the 1 KB allowance");
// the 227 KB of a CTA hold its static shared memory too
constexpr size_t kMaxDynamic = kMaxSmemBytes - 1024;

// Traces per row buffer and row buffers of a launch.
struct Stages {
    int chunk, stages;
};

struct ChunkSmem {
    // layout of one CTA's dynamic shared memory: row buffers, per warp the kept traces'
    // table and the bounds of the run's steps, the weight table
    size_t rawBytes, tabOff, stepOff, wtabOff, total;
};

// table: the kernel interpolates sqrt(j dt) from a per-CTA table (the table weight);
// the prefolded and sqrt.approx weights need none, and their chunks grow by its size
__host__ __device__ __forceinline__ ChunkSmem chunk_layout(Stages st, int warps, int pitch, int esize, int nt,
                                                           bool table)
{
    ChunkSmem L;
    L.rawBytes = (size_t)st.chunk * pitch * esize;           // one buffer
    L.tabOff = st.stages * L.rawBytes;                       // [warps][chunk] float4
    L.stepOff = L.tabOff + (size_t)warps * st.chunk * 16;    // [warps][8] float2
    L.wtabOff = L.stepOff + (size_t)warps * 64;
    L.total = L.wtabOff + (table ? (size_t)(nt + 1) * sizeof(float2) : 0);   // [nt+1] weight table
    return L;
}

// Weight sqrt(t) of each pair (PRE):
//   kWtTable   sqrt(j dt) and its forward difference from a per-CTA table,
//              interpolated with the pair's own fraction f: relative error
//              about 1/(32 j^2), far below FP32 interpolation noise for j > 10;
//   kWtPrefold samples prefolded with sqrt(j dt) by ktmPrepareTraces: one
//              multiply less per pair, but the interpolation of the product
//              differs from the reference weight by f(1-f) dg dd (about 6e-4
//              relative L2 on shallow band-limited data), so it is opt-in;
//   kWtSqrt    a third sqrt.approx per pair on the special-function unit.
constexpr int kWtTable = 0, kWtPrefold = 1, kWtSqrt = 2;

// Output of a tile: the image (overwrite or accumulate), one trace slice's partial
// image, or atomic adds into the image (tiles of the batched launch).
enum { kOutImage = 0, kOutPartial = 1, kOutAtomic = 2 };

// One CTA-tile of the gather: image columns [colGroup*W, colGroup*W+W) x the tau
// run runIdx x traces [kb, ke), W = SH::kWarps.  Used by the grid launch (one tile
// per CTA) and by the persistent batched launch (a queue of tiles from many jobs).
template <class SH, int R, int PICK, int FMT, int PRE, int GRAD>
__device__ __forceinline__ bool fast_tile(const FastArgs& a, Stages st, int colGroup, int runIdx,
                                          int kb, int ke, float* __restrict__ partial, int outMode,
                                          unsigned char* smem_raw, ChunkSync& cs)
{
    static_assert(R % 2 == 0, "R pairs");
    using T = typename Elem<FMT>::T;
    const Geometry& g = a.g;
    const int chunk = st.chunk;
    const ChunkSmem L = chunk_layout(st, SH::kWarps, a.pitch, sizeof(T), a.g.nt, PRE == kWtTable);
    float2* wtab = reinterpret_cast<float2*>(smem_raw + L.wtabOff);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ncols = g.nx * g.ny;
    const int col0 = colGroup * SH::kWarps, active = min(SH::kWarps, ncols - col0);   // warps with a column
    const bool colValid = warp < active;
    const int col = colValid ? col0 + warp : 0;
    const int ci = col / g.ny, cj = col % g.ny;
    const int run0 = runIdx * (32 * R);
    const float invdt = 1.0f / g.dt;

    // ---- per-thread tau tables, two tau samples per packed register pair ----
    f2 T2[R / 2], S2[R / 2], acc[R / 2];
    // Traces that end within the run are walked step by step (200 x 200 x 1501 image, 2500
    // traces: 52.3 ms against 54.7 without); the other weights and the gradient, whose second
    // copy of the loop costs more registers than it saves pairs (table weight on a 128 x 751
    // line: 541 us against 496), evaluate the run to its end, where the guards are zero.
    constexpr bool kStepwise = PRE == kWtPrefold && GRAD == 0;
    constexpr int H = R / 2;            // steps of 64 tau samples, one packed pair per lane each
    // lower bounds of T2' and S' over the run's steps h, h + 1, .. (valid samples)
    float2* steps = reinterpret_cast<float2*>(smem_raw + L.stepOff) + warp * 8;
    float2 step[H];
    int nvalid = 0;
#pragma unroll
    for (int h = 0; h < R / 2; h++) {
        float tv[2], sv[2];
        step[h] = make_float2(3.0e38f, 3.0e38f);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int l = run0 + lane + 32 * (2 * h + e);
            const bool ok = l < g.nz;
            const int lc = ok ? l : g.nz - 1;
            const float tq = (g.z0 + (float)lc * g.dz) * invdt;
            const float v = a.velCube ? a.vel[(size_t)col * g.nz + lc] : a.vel[lc];
            const float vd = v * g.dt;
            tv[e] = tq * tq;
            sv[e] = 1.0f / (vd * vd);
            if (ok) {
                step[h] = make_float2(fminf(step[h].x, tv[e]), fminf(step[h].y, sv[e]));
                nvalid++;
            }
        }
        T2[h] = pk(tv[0], tv[1]);
        S2[h] = pk(sv[0], sv[1]);
        acc[h] = pk(0.0f, 0.0f);
    }
    // minima over the warp: no value is negative or NaN, so their bits order as they do
    auto least = [](float v) { return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(v))); };
#pragma unroll
    for (int h = H - 1; h >= 0; h--) {
        if (h + 1 < H) step[h] = make_float2(fminf(step[h].x, step[h + 1].x), fminf(step[h].y, step[h + 1].y));
        if (kStepwise || h == 0) {
            step[h] = make_float2(least(step[h].x), least(step[h].y));
            if (lane == 0) steps[h] = step[h];
        }
    }
    nvalid = (int)__reduce_add_sync(0xffffffffu, (unsigned)nvalid);
    const float colX = g.x0 + (float)ci * g.dx, colY = g.y0 + (float)cj * g.dy;
    if (PRE == kWtTable) {
        for (int j = threadIdx.x; j <= g.nt; j += SH::kThreads) {
            const float w0 = sqrtf((float)j * g.dt), w1 = sqrtf((float)(j + 1) * g.dt);
            wtab[j] = make_float2(w0, w1 - w0);
        }
    }

    const int nchunks = ke > kb ? (ke - kb + chunk - 1) / chunk : 0;
    const size_t rowBytes = (size_t)a.pitch * sizeof(T);

    // one thread starts chunk ch's copy into its buffer
    auto issue = [&](int ch, int b) {
        const int k0 = kb + ch * chunk, n = min(chunk, ke - k0);
        cs.issued[b]++;
        bulk_g2s(smem_raw + b * L.rawBytes, static_cast<const unsigned char*>(a.traces) + (size_t)k0 * rowBytes,
                 (unsigned)((size_t)n * rowBytes), &cs.bar[b]);
    };

    const float umax = (float)g.nt;
    // a first sample past this has no contribution; the margin covers the bounds'
    // approximate square roots
    const float upast2 = (umax * 1.0001f + 1.0f) * (umax * 1.0001f + 1.0f);
    const float ap2 = a.aperture > 0.0f ? a.aperture * a.aperture : -1.0f;
    const f2 M2 = pk(kMagic, kMagic);
    unsigned walked = 0;            // pairs evaluated of the traces this lane looked at

    if (threadIdx.x == 0) {
        for (int b = 0; b < st.stages; b++) {
            mbar_init(&cs.bar[b], 1);
            cs.done[b] = cs.issued[b] = 0;
        }
        cs.stalled = 0;
        for (int b = 0; b < st.stages && b < nchunks; b++) issue(b, b);
    }
    __syncthreads();                           // barriers, steps and the weight table are ready
    // Every warp goes through the chunks at its own pace, up to stages - 1 chunks ahead of
    // the slowest; the last warp through with a chunk refills its buffer.
    float4* tab = reinterpret_cast<float4*>(smem_raw + L.tabOff) + warp * chunk;
    for (int ch = 0, b = 0, parity = 0; colValid && ch < nchunks; ch++) {
        const int k0 = kb + ch * chunk, n = min(chunk, ke - k0);
        // ---- lane c: trace c's distances, scale, and how many steps of the run it
        // reaches for this column; the kept traces go in order into the warp's table ----
        float ds = 0.0f, dr = 0.0f, sc = 0.0f;
        int hmax = 0;
        if (lane < n) {
            const float mx = a.midX[k0 + lane], my = a.midY[k0 + lane], ox = a.offX[k0 + lane],
                        oy = a.offY[k0 + lane];
            sc = a.scale[k0 + lane];
            const float dmx = mx - colX, dmy = my - colY;
            const float sx = dmx - ox, sy = dmy - oy, rx = dmx + ox, ry = dmy + oy;
            ds = fmaf(sx, sx, sy * sy);             // explicit fusions: the same
            dr = fmaf(rx, rx, ry * ry);             // values in every build
            // lower bound of u from step h on: steps past the last sample contribute zero
            auto reaches = [&](int h) {
                const float2 m = steps[h];      // (sqrt(as) + sqrt(ar))^2 = as + ar + 2 sqrt(as ar)
                const float as = fmaf(ds, m.y, m.x), ar = fmaf(dr, m.y, m.x);
                return fmaf(2.0f, sqrt_approx(as * ar), as + ar) < upast2;
            };
            if (!(ap2 >= 0.0f && fmaf(dmx, dmx, dmy * dmy) > ap2) && reaches(0)) {
                hmax = 1;
#pragma unroll
                for (int d = H > 4 ? 4 : 2; kStepwise && d > 0; d >>= 1)
                    if (hmax - 1 + d < H && reaches(hmax - 1 + d)) hmax += d;
                walked += (unsigned)(kStepwise ? min(64 * hmax, nvalid) : nvalid);
            }
        }
        const unsigned kept = __ballot_sync(0xffffffffu, hmax > 0);
        const int cnt = __popc(kept);
        // bits(fl) = kMagicBits + i0: fold the magic offset into the bases (mod 2^32)
        const unsigned magicT = (unsigned)kMagicBits * (unsigned)sizeof(T);
        const unsigned wS = smem_u32(smem_raw + L.wtabOff) - (unsigned)kMagicBits * 8u;
        if (hmax > 0) {
            // rows are 16-byte aligned: the steps go into the address's low bits
            const unsigned row = smem_u32(smem_raw) + (unsigned)(b * L.rawBytes) +
                                 (unsigned)(lane * a.pitch) * (unsigned)sizeof(T) - magicT;
            tab[__popc(kept & ((1u << lane) - 1u))] = make_float4(ds, dr, sc, __uint_as_float(row + (unsigned)hmax));
        }
        __syncwarp();
        // the ch/stages-th use of buffer b completes that phase of its barrier
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&cs.bar[b], (unsigned)parity, kBulkWaitNs))) {
            if (lane == 0) {
                cs.stalled = 1;
                atomicAdd(&g_waitStalls, 1u);
            }
            break;
        }
        for (int e = 0; e < cnt; e++) {
            const float4 t = tab[e];
            const unsigned rowBits = __float_as_uint(t.w);
            const int hm = (int)(rowBits & 15u);
            const unsigned rowS = rowBits & ~15u;
            const f2 DS = pk(t.x, t.x), DR = pk(t.y, t.y), SC = pk(t.z, t.z);
            // step h: two tau samples of each lane
            auto pairs = [&](int h) __attribute__((always_inline)) {
                if (GRAD) {
                    // d/dS' of |tau| s_k W(u) V(u), u = sqrt(a_s) + sqrt(a_r):
                    // (dW/du V + W dV/du) du/dS', du/dS' = Ds/(2 sqrt a_s) + Dr/(2 sqrt a_r)
                    float as0, as1, ar0, ar1;
                    upk(fma2(DS, S2[h], T2[h]), as0, as1);
                    upk(fma2(DR, S2[h], T2[h]), ar0, ar1);
                    const f2 RS = pk(fminf(rsqrt_approx(as0), 3.0e38f), fminf(rsqrt_approx(as1), 3.0e38f));
                    const f2 RR = pk(fminf(rsqrt_approx(ar0), 3.0e38f), fminf(rsqrt_approx(ar1), 3.0e38f));
                    f2 U = fma2(pk(ar0, ar1), RR, mul2(pk(as0, as1), RS));
                    float u0, u1;
                    upk(U, u0, u1);
                    u0 = fminf(u0, umax);
                    u1 = fminf(u1, umax);
                    U = pk(u0, u1);
                    const f2 FL = add2_rm(U, M2);
                    float fl0, fl1;
                    upk(FL, fl0, fl1);
                    const unsigned q0 = __float_as_uint(fl0), q1 = __float_as_uint(fl1);
                    const f2 F = sub2(U, sub2(FL, M2));
                    const f2 DUDS = mul2(pk(0.5f, 0.5f), fma2(DS, RS, mul2(DR, RR)));
                    float a0, b0, a1, b1;
                    Lds<FMT>::pair(rowS + q0 * (unsigned)sizeof(T), a0, b0);
                    Lds<FMT>::pair(rowS + q1 * (unsigned)sizeof(T), a1, b1);
                    const f2 A = pk(a0, a1);
                    const f2 DV = sub2(pk(b0, b1), A);
                    f2 TERM;
                    if (PRE == kWtPrefold) {
                        TERM = DV;
                    } else {
                        const float2 w0 = lds_f2(wS + q0 * 8u), w1 = lds_f2(wS + q1 * 8u);
                        const f2 DW = pk(w0.y, w1.y);
                        const f2 W = fma2(F, DW, pk(w0.x, w1.x));
                        const f2 V = fma2(F, DV, A);
                        TERM = fma2(DW, V, mul2(W, DV));
                    }
                    acc[h] = fma2(mul2(SC, TERM), DUDS, acc[h]);
                    return;
                }
                const PairKin kk = pair_kin(DS, DR, S2[h], T2[h], umax, M2);
                const f2 F = kk.F;
                const float u0 = kk.u0, u1 = kk.u1;
                const unsigned q0 = kk.q0, q1 = kk.q1;
                const unsigned ad0 = rowS + q0 * (unsigned)sizeof(T);
                const unsigned ad1 = rowS + q1 * (unsigned)sizeof(T);
                f2 V;
                if (PICK == KTM_PICK_LINEAR) {
                    float a0, b0, a1, b1;
                    Lds<FMT>::pair(ad0, a0, b0);
                    Lds<FMT>::pair(ad1, a1, b1);
                    const f2 A = pk(a0, a1);
                    V = fma2(F, sub2(pk(b0, b1), A), A);
                } else {
                    V = pk(Lds<FMT>::one(ad0), Lds<FMT>::one(ad1));
                }
                if (PRE == kWtPrefold) {
                    acc[h] = fma2(SC, V, acc[h]);
                } else if (PRE == kWtTable) {
                    const float2 w0 = lds_f2(wS + q0 * 8u), w1 = lds_f2(wS + q1 * 8u);
                    const f2 W = fma2(F, pk(w0.y, w1.y), pk(w0.x, w1.x));
                    acc[h] = fma2(mul2(SC, W), V, acc[h]);
                } else {
                    // u is in samples: sqrt(t) = sqrt(u) sqrt(dt), sqrt(dt) applied at the end
                    const f2 W = pk(sqrt_approx(u0), sqrt_approx(u1));
                    acc[h] = fma2(mul2(SC, W), V, acc[h]);
                }
            };
            // all steps in one block the compiler interleaves, or step by step up to the last
            // one that reaches the trace end
            if (!kStepwise || hm == H) {
#pragma unroll
                for (int h = 0; h < H; h++) pairs(h);
            } else {
#pragma unroll
                for (int h = 0; h < H; h++) {
                    if (h > 0 && h >= hm) break;
                    pairs(h);
                }
            }
        }
        // the last warp through with the chunk starts the copy of the one that follows in
        // this buffer
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            if (atomicAdd(&cs.done[b], 1) == active - 1) {
                cs.done[b] = 0;
                __threadfence_block();
                if (ch + st.stages < nchunks) issue(ch + st.stages, b);
            }
        }
        if (++b == st.stages) {
            b = 0;
            parity ^= 1;
        }
    }

    __syncthreads();
    if (threadIdx.x == 0) {
        for (int b = 0; b < st.stages; b++) {
            // a tile that gave up waits (bounded) for its copies in flight
            if (cs.stalled && cs.issued[b]) mbar_wait_bounded(&cs.bar[b], (unsigned)(cs.issued[b] - 1) & 1u, kBulkWaitNs);
            mbar_inval(&cs.bar[b]);
        }
    }
    if (cs.stalled) return false;              // CTA-uniform: no output from this tile
    if (colValid) {
        float* out = (outMode == kOutPartial ? partial : a.image) + (size_t)col * g.nz;
#pragma unroll
        for (int h = 0; h < R / 2; h++) {
            float v2[2], s2[2];
            upk(acc[h], v2[0], v2[1]);
            upk(S2[h], s2[0], s2[1]);
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int l = run0 + lane + 32 * (2 * h + e);
                if (l < g.nz) {
                    const float tau = fabsf(g.z0 + (float)l * g.dz);
                    // GRAD: dI/dv = dI/dS' dS'/dv, S' = 1/(v dt)^2, dS'/dv = -2 dt S'^(3/2)
                    const float gfac = GRAD ? -2.0f * g.dt * s2[e] * sqrtf(s2[e]) : 1.0f;
                    const float v = v2[e] * gfac * (PRE == kWtSqrt ? tau * sqrtf(g.dt) : tau);
                    if (outMode == kOutAtomic) atomicAdd(out + l, v);
                    else out[l] = (outMode == kOutImage && a.accumulate) ? out[l] + v : v;
                }
            }
        }
    }
    if (a.pairsEvaluated && colValid) {
        const unsigned lo = __reduce_add_sync(0xffffffffu, walked & 0xffffu), hi = __reduce_add_sync(0xffffffffu, walked >> 16);
        if (lane == 0 && (lo | hi)) atomicAdd(a.pairsEvaluated, ((unsigned long long)hi << 16) + lo);
    }
    return true;
}

// ---------------------------------------------------------------------------
// Persistent batched launch: one CTA per SM slot pulls (job, column group, tau
// run, trace slice) tiles from a queue sorted longest first; each tile adds its
// result into its job's image with atomics (the images start at zero).  The
// job's arguments are copied into shared memory for the tile.
// ---------------------------------------------------------------------------
struct BatchTile {
    int job, cg, run, kb, ke, pad;
};

template <class SH, int R, int PICK, int FMT, int PRE>
__global__ void __launch_bounds__(SH::kThreads, SH::kMinBlocks)
batch_kernel(const FastArgs* __restrict__ jobs, const Stages* __restrict__ chunks,
             const BatchTile* __restrict__ tiles, int ntiles, unsigned* __restrict__ counter)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ChunkSync cs;
    __shared__ FastArgs sa;
    __shared__ int st;
    static_assert(sizeof(FastArgs) % 4 == 0, "word copy");
    for (;;) {
        if (threadIdx.x == 0) st = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int t = st;
        if (t >= ntiles) break;                    // every thread read the same t
        const BatchTile tl = tiles[t];
        const int* src = reinterpret_cast<const int*>(jobs + tl.job);
        int* dst = reinterpret_cast<int*>(&sa);
        for (int i = threadIdx.x; i < (int)(sizeof(FastArgs) / 4); i += SH::kThreads) dst[i] = src[i];
        __syncthreads();
        const bool ok = fast_tile<SH, R, PICK, FMT, PRE, 0>(sa, chunks[tl.job], tl.cg, tl.run, tl.kb, tl.ke,
                                                        nullptr, kOutAtomic, smem_raw, cs);
        __syncthreads();                           // shared memory is reused by the next tile
        if (!ok) break;                            // CTA-uniform
    }
}

template <class SH, int R, int PICK, int FMT, int PRE, int GRAD>
__global__ void __launch_bounds__(SH::kThreads, SH::kMinBlocks)
fast_kernel(FastArgs a, Stages st, int perSlice, float* __restrict__ partial)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ChunkSync cs;
    const int kb = blockIdx.z * perSlice;
    const int ke = min(a.g.ntr, kb + perSlice);
    const size_t nimg = (size_t)a.g.nx * a.g.ny * a.g.nz;
    fast_tile<SH, R, PICK, FMT, PRE, GRAD>(a, st, blockIdx.x, blockIdx.y, kb, ke,
                                       partial ? partial + blockIdx.z * nimg : nullptr,
                                       partial ? kOutPartial : kOutImage, smem_raw, cs);
}

// out[i] = (accumulate ? out[i] : 0) + sum_z partial[z][i], z in increasing order
__global__ void reduce_slices(float* __restrict__ out, const float* __restrict__ partial,
                              size_t nimg, int nslices, int accumulate)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nimg;
         i += (size_t)gridDim.x * blockDim.x) {
        float s = accumulate ? out[i] : 0.0f;
        for (int z = 0; z < nslices; z++) s += partial[(size_t)z * nimg + i];
        out[i] = s;
    }
}

// Traces per row buffer and buffers: as many traces as the shape's shared-memory budget
// holds (at most kMaxChunk per buffer, or fewer when the caller caps them: chunkCap > 0),
// in three buffers where each still gets 16 traces, else in two: the third lets the warps
// drift further apart, fewer traces per buffer cost more of the per-chunk geometry.  No more than
// the launch's traces need, which leaves the L1 cache its room (60 million samples, 8 F32 traces:
// 318 us, 391 with all buffers).  chunk 0
// for traces beyond the limit: two of them, with the weight table, exceed the largest
// allocation a CTA can have.
template <class SH>
Stages fast_stages(const FastArgs& a, int esize, bool table)
{
    const int cap = std::min(a.chunkCap > 0 ? std::min(kMaxChunk, a.chunkCap) : kMaxChunk, std::max(1, a.g.ntr));
    auto fit = [&](int stages) {
        Stages s = {cap, stages};
        while (s.chunk > 1 && chunk_layout(s, SH::kWarps, a.pitch, esize, a.g.nt, table).total > SH::kBudget)
            s.chunk--;
        return s;
    };
    // two buffers of one trace and its 48 bytes of coordinates beside the table
    if (2 * (size_t)a.pitch * esize + 48 + (table ? (a.g.nt + 1) * sizeof(float2) : 0) > (size_t)kMaxSmemBytes)
        return Stages{0, 0};
    Stages s = fit(3);
    if (s.chunk < std::min(cap, 16)) s = fit(2);
    s.stages = std::max(1, std::min(s.stages, (a.g.ntr + s.chunk - 1) / s.chunk));     // no buffer without a copy
    // the longest traces: two buffers leave no room for the warps' tables
    if (chunk_layout(s, SH::kWarps, a.pitch, esize, a.g.nt, table).total > kMaxDynamic) s.stages = 1;
    return s;
}

// Partial images of a launch at most: an image of more than half of this is written in place.
constexpr size_t kPartialBytes = 256u << 20;

// Trace slices of a launch of `base` CTAs per slice on `slots` resident CTAs: the number
// with the least estimated time, in traces of a CTA: a CTA takes its traces, times the share of the
// image that an aperture covers, + 8 for its prologue, and the last ones end half a CTA past the
// mean (columns keep uneven numbers of traces, and a line sorted by offset has slices without any:
// 88 x 225 line, 4488 traces of 226 samples, 47 us in the 37 slices that fit at once, 34 in 64;
// 1000 x 1001, 200 traces, aperture 700 m, 53 us without the share, 39 in one slice); plus the
// partial images (a trace takes about 1 us at R = 16, 6.5 MB of partial images the same).
// Estimates fitted to random surveys (prologue by R, whole rounds) gained 5 % there and lost up to
// 40 % on sorted lines.
int choose_slices(const FastArgs& a, long long base, int slots, int R)
{
    const Geometry& g = a.g;
    const int ntr = g.ntr;
    const size_t nimg = (size_t)g.nx * g.ny * g.nz;
    auto covered = [&](float extent) { return std::min(1.0f, 2.0f * a.aperture / std::max(fabsf(extent), 1e-30f)); };
    const float share = a.aperture > 0.0f ? std::max(0.1f, covered((float)g.nx * g.dx) * covered((float)g.ny * g.dy)) : 1.0f;
    const int most = (int)std::min<size_t>(std::max(1, std::min(64, ntr / 8)),
                                           std::max<size_t>(1, kPartialBytes / (nimg * sizeof(float))));
    int best = 1;
    float least = 3.0e38f;
    for (int s = 1; s <= most; s++) {
        const float per = (float)((ntr + s - 1) / s) * share + 8.0f;
        const float rounds = std::max(1.0f, (float)(base * s) / (float)slots) + 0.5f;
        const float copies = s > 1 ? (float)s * (float)nimg * (8.0f / 6.5e6f) * 16.0f / (float)R : 0.0f;
        const float cost = rounds * per + copies;
        if (cost < least) {
            least = cost;
            best = s;
        }
    }
    return best;
}

// One grid launch over all of a's traces.
template <class SH, int R, int PICK, int FMT, int PRE, int GRAD>
int launch_block(const FastArgs& a, cudaStream_t stream, int smCount)
{
    const Geometry& g = a.g;
    const int esize = FMT == KTM_FMT_F32 ? 4 : 2;
    constexpr bool kTable = PRE == kWtTable;
    const Stages st = fast_stages<SH>(a, esize, kTable);
    const int chunk = st.chunk;
    if (chunk == 0)
        return set_error(KTM_ERR_LIMIT, "fast kernel: packed pitch %d exceeds the shared-memory "
                                        "stage limit", a.pitch);
    const size_t smem = chunk_layout(st, SH::kWarps, a.pitch, esize, g.nt, kTable).total;
    auto kern = fast_kernel<SH, R, PICK, FMT, PRE, GRAD>;
    KTM_CUDA_TRY(allow_smem(kern, smem, kMaxDynamic));

    const long long cols = (long long)g.nx * g.ny;
    const unsigned gx = (unsigned)((cols + SH::kWarps - 1) / SH::kWarps);
    const unsigned gy = (unsigned)((g.nz + 32 * R - 1) / (32 * R));
    if (gy > 65535) return set_error(KTM_ERR_LIMIT, "fast kernel: Nz too large");
    const size_t nimg = (size_t)cols * g.nz;
    int slices = a.slices > 0 ? min(a.slices, max(1, g.ntr))
                              : choose_slices(a, (long long)gx * gy, SH::kMinBlocks * smCount, R);
    int perSlice = (g.ntr + slices - 1) / slices;
    slices = (g.ntr + perSlice - 1) / perSlice;

    float* partial = nullptr;
    if (slices > 1) {
        if (a.scratch && a.scratchBytes >= (size_t)slices * nimg * sizeof(float)) {
            partial = static_cast<float*>(a.scratch);
        } else {
            const cudaError_t m = pool_malloc(reinterpret_cast<void**>(&partial),
                                              (size_t)slices * nimg * sizeof(float), stream);
            if (m != cudaSuccess && a.slices > 0) KTM_CUDA_TRY(m);
            if (m != cudaSuccess) {
                cudaGetLastError();            // no room for partial images: one slice, in place
                partial = nullptr;
                slices = 1;
                perSlice = g.ntr;
            }
        }
    }
    dim3 grid(gx, gy, (unsigned)slices);
    kern<<<grid, SH::kThreads, smem, stream>>>(a, st, perSlice, partial);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && partial) {
        const int th = 256;
        const size_t want = (nimg + th - 1) / th, cap = (size_t)smCount * 8;
        const unsigned blocks = (unsigned)(want < cap ? want : cap);
        reduce_slices<<<blocks, th, 0, stream>>>(a.image, partial, nimg, slices, a.accumulate);
        e = cudaGetLastError();
    }
    if (partial && partial != a.scratch) cudaFreeAsync(partial, stream);
    if (e != cudaSuccess) return set_error(KTM_ERR_CUDA, "fast kernel launch: %s", cudaGetErrorString(e));
    return KTM_OK;
}

// Packed trace bytes per launch.  Every CTA streams all traces of its launch
// and CTAs start at different times, so the traces of one launch should stay
// resident in L2 (126 MB) while they are read: a trace set larger than this
// goes in blocks, one launch each, the later ones accumulating.
constexpr size_t kTraceBlockBytes = 40u << 20;

template <class SH, int R, int PICK, int FMT, int PRE, int GRAD>
int launch_t(const FastArgs& a, cudaStream_t stream, int smCount)
{
    const int esize = FMT == KTM_FMT_F32 ? 4 : 2;
    const size_t rowBytes = (size_t)a.pitch * esize;
    const int block = (int)std::max<size_t>(1024, kTraceBlockBytes / rowBytes);
    if (a.g.ntr <= block) return launch_block<SH, R, PICK, FMT, PRE, GRAD>(a, stream, smCount);
    // balanced blocks of at most `block` traces
    const int nblk = (a.g.ntr + block - 1) / block;
    const int per = (a.g.ntr + nblk - 1) / nblk;
    for (int kb = 0; kb < a.g.ntr; kb += per) {
        FastArgs b = a;
        b.g.ntr = std::min(per, a.g.ntr - kb);
        b.midX = a.midX + kb; b.midY = a.midY + kb; b.offX = a.offX + kb; b.offY = a.offY + kb;
        b.traces = static_cast<const unsigned char*>(a.traces) + (size_t)kb * rowBytes;
        b.scale = a.scale ? a.scale + kb : nullptr;
        b.accumulate = a.accumulate || kb > 0;
        const int rc = launch_block<SH, R, PICK, FMT, PRE, GRAD>(b, stream, smCount);
        if (rc) return rc;
    }
    return KTM_OK;
}

template <class SH, int R, int PICK, int PRE, int GRAD = 0>
int launch_fmt(const FastArgs& a, cudaStream_t s, int sm)
{
    switch (a.fmt) {
        case KTM_FMT_F32: return launch_t<SH, R, PICK, KTM_FMT_F32, PRE, GRAD>(a, s, sm);
        case KTM_FMT_F16: return launch_t<SH, R, PICK, KTM_FMT_F16, PRE, GRAD>(a, s, sm);
        default: return launch_t<SH, R, PICK, KTM_FMT_BF16, PRE, GRAD>(a, s, sm);
    }
}

// The paths a reduced shape is built for: linear pick, prefolded samples or the
// table weight, no gradient.
bool tunable_path(const FastArgs& a)
{
    return !a.grad && a.pick == KTM_PICK_LINEAR &&
           (a.weightMode == 2 || a.weightMethod == KTM_WEIGHT_TABLE);
}

template <class SH, int R>
int launch_pick(const FastArgs& a, cudaStream_t s, int sm)
{
    if constexpr (!SH::kFull) {
        if (!tunable_path(a))
            return set_error(KTM_ERR_ARG, "fast kernel: tileCols %d is built for the linear pick "
                                          "with the prefolded or table weight only (0 or 24 "
                                          "takes every path)", SH::kWarps);
        return a.weightMode == 2 ? launch_fmt<SH, R, KTM_PICK_LINEAR, kWtPrefold>(a, s, sm)
                                 : launch_fmt<SH, R, KTM_PICK_LINEAR, kWtTable>(a, s, sm);
    } else {
        if (a.grad) {
            // velocity gradient: linear pick; table weight or prefolded samples
            if (a.pick != KTM_PICK_LINEAR || (a.weightMode != 2 && a.weightMethod != KTM_WEIGHT_TABLE))
                return set_error(KTM_ERR_ARG, "ktmVrmsGradient takes the linear pick with the table "
                                              "weight or prefolded samples");
            return a.weightMode == 2 ? launch_fmt<SH, R, KTM_PICK_LINEAR, kWtPrefold, 1>(a, s, sm)
                                     : launch_fmt<SH, R, KTM_PICK_LINEAR, kWtTable, 1>(a, s, sm);
        }
        // a.weightMode: 2 samples prefolded; otherwise a.weightMethod picks table / sqrt
        if (a.weightMode == 2) {
            if (a.pick != KTM_PICK_LINEAR)
                return set_error(KTM_ERR_ARG, "truncating pick takes traces without the sqrt(t) fold");
            return launch_fmt<SH, R, KTM_PICK_LINEAR, kWtPrefold>(a, s, sm);
        }
        const bool sq = a.weightMethod == KTM_WEIGHT_SQRT;
        if (a.pick == KTM_PICK_LINEAR)
            return sq ? launch_fmt<SH, R, KTM_PICK_LINEAR, kWtSqrt>(a, s, sm)
                      : launch_fmt<SH, R, KTM_PICK_LINEAR, kWtTable>(a, s, sm);
        return sq ? launch_fmt<SH, R, KTM_PICK_TRUNCATE, kWtSqrt>(a, s, sm)
                  : launch_fmt<SH, R, KTM_PICK_TRUNCATE, kWtTable>(a, s, sm);
    }
}

template <class SH>
int launch_run(const FastArgs& a, int R, cudaStream_t s, int sm)
{
    switch (R) {
        case 8: return launch_pick<SH, 8>(a, s, sm);
        case 12: return launch_pick<SH, 12>(a, s, sm);
        case 16: return launch_pick<SH, 16>(a, s, sm);
        default: return set_error(KTM_ERR_ARG, "fast kernel: tileRun must be 256, 384 or 512");
    }
}

// tau samples per lane: from tileRun, or the run of 512 / 384 / 256 wasting the
// fewest samples at the end of Nz
int choose_run(int tileRun, int nz)
{
    if (tileRun > 0) return tileRun / 32;
    int best = 16, bestWaste = 1 << 30;
    for (int r : {16, 12, 8}) {
        const int run = 32 * r, waste = ((nz + run - 1) / run) * run - nz;
        if (waste < bestWaste) { bestWaste = waste; best = r; }
    }
    return best;
}

// ---------------------------------------------------------------------------
// FP64 device reference: one thread per image sample, traces straight from
// global memory.  Slow; used to measure the error of the fast path on
// configurations too large for the CPU oracle.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double load_any(const void* p, int fmt, size_t idx)
{
    if (fmt == KTM_FMT_F64) return static_cast<const double*>(p)[idx];
    if (fmt == KTM_FMT_F32) return (double)static_cast<const float*>(p)[idx];
    if (fmt == KTM_FMT_F16) return (double)__half2float(static_cast<const __half*>(p)[idx]);
    return (double)__bfloat162float(static_cast<const __nv_bfloat16*>(p)[idx]);
}

__global__ void f64_kernel(FastArgs a, const int* __restrict__ cols, int ncols,
                           double* __restrict__ out)
{
    const Geometry& g = a.g;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)ncols * g.nz) return;
    const int q = (int)(idx / g.nz), l = (int)(idx % g.nz);
    const int col = cols ? cols[q] : q;
    if (col < 0 || col >= g.nx * g.ny) {      // column outside the image: NaN, no reads
        out[(size_t)q * g.nz + l] = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    const int ci = col / g.ny, cj = col % g.ny;
    const double x = (double)g.x0 + (double)ci * (double)g.dx;
    const double y = (double)g.y0 + (double)cj * (double)g.dy;
    const double tau = (double)g.z0 + (double)l * (double)g.dz;
    const double v = a.velCube ? (double)a.vel[(size_t)col * g.nz + l] : (double)a.vel[l];
    const double S = 1.0 / (v * v), tau2 = tau * tau, dt = (double)g.dt;
    const double ap2 = a.aperture > 0.0f ? (double)a.aperture * (double)a.aperture : -1.0;
    const int stride = a.pitch;
    double acc = 0.0;
    for (int k = 0; k < g.ntr; k++) {
        const double mx = a.midX[k], my = a.midY[k], ox = a.offX[k], oy = a.offY[k];
        const double dmx = mx - x, dmy = my - y;
        if (ap2 >= 0.0 && dmx * dmx + dmy * dmy > ap2) continue;
        const double sx = dmx - ox, sy = dmy - oy, rx = dmx + ox, ry = dmy + oy;
        const double t = sqrt(tau2 + (sx * sx + sy * sy) * S) + sqrt(tau2 + (rx * rx + ry * ry) * S);
        const double u = t / dt;
        if (!(u < (double)g.nt)) continue;
        const double sc = a.scale ? (double)a.scale[k] : 1.0;
        const size_t base = (size_t)k * stride;
        double val;
        if (a.pick == KTM_PICK_LINEAR) {
            const double fl = floor(u);
            const int i0 = (int)fl;
            const double f = u - fl;
            double d0 = (i0 > 0 && i0 < g.nt) ? load_any(a.traces, a.fmt, base + i0) : 0.0;
            double d1 = (i0 + 1 > 0 && i0 + 1 < g.nt) ? load_any(a.traces, a.fmt, base + i0 + 1) : 0.0;
            if (a.weightMode == 1) {
                d0 *= sqrt((double)i0 * dt);
                d1 *= sqrt((double)(i0 + 1) * dt);
            }
            val = (1.0 - f) * d0 + f * d1;
        } else {
            const int it = (int)u;
            val = (it > 0 && it < g.nt) ? load_any(a.traces, a.fmt, base + it) : 0.0;
            if (a.weightMode == 1) val *= sqrt((double)it * dt);
        }
        const double w = a.weightMode ? fabs(tau) : (t > 0.0 ? t * sqrt(tau2 / t) : 0.0);
        acc += w * sc * val;
    }
    out[(size_t)q * g.nz + l] = acc;
}

}  // namespace

int launch_fast(const FastArgs& a, cudaStream_t stream)
{
    const Geometry& g = a.g;
    if ((long long)g.nx * g.ny * g.nz == 0) return KTM_OK;
    if (g.nt >= (1 << 22)) return set_error(KTM_ERR_LIMIT, "fast kernel: tracePts must be < 4194304");
    if (g.ntr == 0) {
        if (!a.accumulate)
            KTM_CUDA_TRY(cudaMemsetAsync(a.image, 0, sizeof(float) * (size_t)g.nx * g.ny * g.nz, stream));
        return KTM_OK;
    }
    const int esize = a.fmt == KTM_FMT_F32 ? 4 : 2;
    if (a.pitch < g.nt + 2 || ((size_t)a.pitch * esize) % 16 != 0 ||
        reinterpret_cast<uintptr_t>(a.traces) % 16 != 0)
        return set_error(KTM_ERR_ARG, "fast kernel: traces must be a packed set (pitch >= tracePts+2, "
                                      "16-byte rows, 16-byte aligned)");
    int dev = 0, sm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
    const int R = choose_run(a.tileRun, g.nz);
    switch (a.tileCols) {
        case 0:
        case 24: return launch_run<Shape24>(a, R, stream, sm);
        case 12: return launch_run<Shape12>(a, R, stream, sm);
        case 8: return launch_run<Shape8>(a, R, stream, sm);
        default: return set_error(KTM_ERR_ARG, "fast kernel: tileCols must be 0, 8, 12 or 24");
    }
}

int launch_f64_columns(const FastArgs& a, const int* cols, int ncols, double* out, cudaStream_t stream)
{
    const long long n = (long long)ncols * a.g.nz;
    if (n == 0) return KTM_OK;
    const int th = 128;
    f64_kernel<<<(unsigned)((n + th - 1) / th), th, 0, stream>>>(a, cols, ncols, out);
    KTM_CUDA_TRY(cudaGetLastError());
    return KTM_OK;
}

}  // namespace ktm

namespace ktm {
namespace {

// Zeroes every job's image in one launch (a memset each took 4 us: 50 of the 1475 us of twelve
// targets of 192 x 501 samples); gridDim.x CTAs an image (zero_ctas).
__global__ void __launch_bounds__(256) zero_images(const FastArgs* __restrict__ jobs, int njobs)
{
    for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
        float* __restrict__ image = jobs[j].image;
        const size_t n = (size_t)jobs[j].g.nx * jobs[j].g.ny * jobs[j].g.nz;
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
            image[i] = 0.0f;
    }
}

// CTAs per image: one per 4096 samples of the largest, at most eight per SM over all images.  A call of
// one job, 60 million samples and 8 BF16 traces: 317 us, 632 with 16 CTAs an image whatever its size.
int zero_ctas(const FastArgs* jobs, int njobs, int sm)
{
    size_t most = 1;
    for (int j = 0; j < njobs; j++) most = std::max(most, (size_t)jobs[j].g.nx * jobs[j].g.ny * jobs[j].g.nz);
    return (int)std::min<size_t>((most + 4095) / 4096, std::max(16, 8 * sm / njobs));
}

template <class SH, int R, int PICK, int FMT, int PRE>
int launch_batch_t(const FastArgs* jobs, int njobs, cudaStream_t s)
{
    const int esize = FMT == KTM_FMT_F32 ? 4 : 2;
    int dev = 0, sm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
    const int ctas = SH::kMinBlocks * sm;
    std::vector<Stages> chunks(njobs);
    size_t smem = 0;
    double totalPairs = 0.0;
    for (int j = 0; j < njobs; j++) {
        const Geometry& g = jobs[j].g;
        const Stages c = fast_stages<SH>(jobs[j], esize, PRE == kWtTable);
        if (c.chunk == 0)
            return set_error(KTM_ERR_LIMIT, "batch: job %d packed pitch %d exceeds shared memory", j,
                             jobs[j].pitch);
        const size_t need = chunk_layout(c, SH::kWarps, jobs[j].pitch, esize, g.nt, PRE == kWtTable).total;
        chunks[j] = c;
        smem = std::max(smem, need);
        totalPairs += (double)g.nx * g.ny * g.nz * g.ntr;
    }
    // tiles: every job's column groups x tau runs, traces sliced so that no tile
    // exceeds ~1/16 of a CTA's share of the whole batch
    const double perTile = std::max(1.0, totalPairs / (ctas * 16.0));
    std::vector<BatchTile> tiles;
    std::vector<double> cost;
    for (int j = 0; j < njobs; j++) {
        const Geometry& g = jobs[j].g;
        const long long cols = (long long)g.nx * g.ny;
        if (cols * g.nz == 0 || g.ntr == 0) continue;
        const int cgs = (int)((cols + SH::kWarps - 1) / SH::kWarps);
        const int runs = (g.nz + 32 * R - 1) / (32 * R);
        const double tilePairsPerTrace = (double)SH::kWarps * 32 * R;
        int per = (int)std::min<double>(g.ntr, std::max<double>(4.0 * chunks[j].chunk, perTile / tilePairsPerTrace));
        per = std::max(per, 1);
        for (int cg = 0; cg < cgs; cg++)
            for (int r = 0; r < runs; r++)
                for (int kb = 0; kb < g.ntr; kb += per) {
                    const int ke = std::min(g.ntr, kb + per);
                    tiles.push_back(BatchTile{j, cg, r, kb, ke, 0});
                    cost.push_back(tilePairsPerTrace * (ke - kb));
                }
    }
    // without tiles there is nothing to add to the zeroed images
    if (tiles.empty()) {
        for (int j = 0; j < njobs; j++) {
            const size_t nimg = (size_t)jobs[j].g.nx * jobs[j].g.ny * jobs[j].g.nz;
            if (nimg) KTM_CUDA_TRY(cudaMemsetAsync(jobs[j].image, 0, nimg * sizeof(float), s));
        }
        return KTM_OK;
    }
    // longest first, so that the queue's tail is made of short tiles
    std::vector<int> order(tiles.size());
    for (size_t i = 0; i < order.size(); i++) order[i] = (int)i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost[x] > cost[y]; });
    std::vector<BatchTile> sorted(tiles.size());
    for (size_t i = 0; i < order.size(); i++) sorted[i] = tiles[order[i]];

    const size_t bJobs = sizeof(FastArgs) * njobs, bChunks = sizeof(Stages) * njobs;
    const size_t bTiles = sizeof(BatchTile) * sorted.size();
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    // jobs, row buffers, tiles and the queue's counter in one copy
    const size_t oChunks = up(bJobs), oTiles = oChunks + up(bChunks), oCounter = oTiles + up(bTiles);
    std::vector<unsigned char> host(oCounter + sizeof(unsigned), 0);
    std::memcpy(host.data(), jobs, bJobs);
    std::memcpy(host.data() + oChunks, chunks.data(), bChunks);
    std::memcpy(host.data() + oTiles, sorted.data(), bTiles);
    unsigned char* buf = nullptr;
    KTM_CUDA_TRY(pool_malloc(reinterpret_cast<void**>(&buf), host.size(), s));
    FastArgs* dJobs = reinterpret_cast<FastArgs*>(buf);
    Stages* dChunks = reinterpret_cast<Stages*>(buf + oChunks);
    BatchTile* dTiles = reinterpret_cast<BatchTile*>(buf + oTiles);
    unsigned* dCounter = reinterpret_cast<unsigned*>(buf + oCounter);
    cudaError_t e = cudaMemcpyAsync(buf, host.data(), host.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        zero_images<<<dim3((unsigned)zero_ctas(jobs, njobs, sm), (unsigned)std::min(njobs, 65535)), 256, 0, s>>>(dJobs, njobs);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = allow_smem(batch_kernel<SH, R, PICK, FMT, PRE>, smem, kMaxDynamic);
    if (e == cudaSuccess) {
        const int grid = (int)std::min<size_t>((size_t)ctas, sorted.size());
        batch_kernel<SH, R, PICK, FMT, PRE><<<grid, SH::kThreads, smem, s>>>(dJobs, dChunks, dTiles,
                                                                      (int)sorted.size(), dCounter);
        e = cudaGetLastError();
    }
    // the host vector above is pageable: its copy was staged before the call returned
    cudaFreeAsync(buf, s);
    if (e != cudaSuccess) return set_error(KTM_ERR_CUDA, "batch launch: %s", cudaGetErrorString(e));
    return KTM_OK;
}

template <class SH, int R, int PICK, int PRE>
int launch_batch_fmt(const FastArgs* jobs, int n, cudaStream_t s)
{
    switch (jobs[0].fmt) {
        case KTM_FMT_F32: return launch_batch_t<SH, R, PICK, KTM_FMT_F32, PRE>(jobs, n, s);
        case KTM_FMT_F16: return launch_batch_t<SH, R, PICK, KTM_FMT_F16, PRE>(jobs, n, s);
        default: return launch_batch_t<SH, R, PICK, KTM_FMT_BF16, PRE>(jobs, n, s);
    }
}

template <class SH, int R>
int launch_batch_r(const FastArgs* jobs, int n, cudaStream_t s)
{
    const FastArgs& a = jobs[0];
    if constexpr (!SH::kFull) {
        if (!tunable_path(a))
            return set_error(KTM_ERR_ARG, "batch: tileCols %d is built for the linear pick with the "
                                          "prefolded or table weight only", SH::kWarps);
        return a.weightMode == 2 ? launch_batch_fmt<SH, R, KTM_PICK_LINEAR, kWtPrefold>(jobs, n, s)
                                 : launch_batch_fmt<SH, R, KTM_PICK_LINEAR, kWtTable>(jobs, n, s);
    } else {
        if (a.weightMode == 2) {
            if (a.pick != KTM_PICK_LINEAR)
                return set_error(KTM_ERR_ARG, "truncating pick takes traces without the sqrt(t) fold");
            return launch_batch_fmt<SH, R, KTM_PICK_LINEAR, kWtPrefold>(jobs, n, s);
        }
        const bool sq = a.weightMethod == KTM_WEIGHT_SQRT;
        if (a.pick == KTM_PICK_LINEAR)
            return sq ? launch_batch_fmt<SH, R, KTM_PICK_LINEAR, kWtSqrt>(jobs, n, s)
                      : launch_batch_fmt<SH, R, KTM_PICK_LINEAR, kWtTable>(jobs, n, s);
        return sq ? launch_batch_fmt<SH, R, KTM_PICK_TRUNCATE, kWtSqrt>(jobs, n, s)
                  : launch_batch_fmt<SH, R, KTM_PICK_TRUNCATE, kWtTable>(jobs, n, s);
    }
}

template <class SH>
int launch_batch_shape(const FastArgs* jobs, int n, int R, cudaStream_t s)
{
    switch (R) {
        case 8: return launch_batch_r<SH, 8>(jobs, n, s);
        case 12: return launch_batch_r<SH, 12>(jobs, n, s);
        case 16: return launch_batch_r<SH, 16>(jobs, n, s);
        default: return set_error(KTM_ERR_ARG, "batch: tileRun must be 256, 384 or 512");
    }
}

}  // namespace

int launch_batch(const FastArgs* jobs, int njobs, cudaStream_t s)
{
    if (njobs <= 0) return KTM_OK;
    const FastArgs& a = jobs[0];
    for (int j = 0; j < njobs; j++) {
        const FastArgs& b = jobs[j];
        if (b.fmt != a.fmt || b.pick != a.pick || b.weightMode != a.weightMode ||
            b.weightMethod != a.weightMethod)
            return set_error(KTM_ERR_ARG, "batch: every job needs the same trace format, pick and weight");
        const int esize = b.fmt == KTM_FMT_F32 ? 4 : 2;
        if (b.g.ntr > 0 && (b.pitch < b.g.nt + 2 || ((size_t)b.pitch * esize) % 16 != 0 ||
                            reinterpret_cast<uintptr_t>(b.traces) % 16 != 0))
            return set_error(KTM_ERR_ARG, "batch: job %d traces are not a packed set", j);
        if (b.g.nt >= (1 << 22)) return set_error(KTM_ERR_LIMIT, "batch: tracePts too large");
    }
    int R = a.tileRun > 0 ? a.tileRun / 32 : 0;
    if (R == 0) {
        int best = 16, bestWaste = 1 << 30;
        for (int r : {16, 12, 8}) {
            long long waste = 0;
            for (int j = 0; j < njobs; j++) {
                const int run = 32 * r, nz = jobs[j].g.nz;
                waste += (long long)(((nz + run - 1) / run) * run - nz) * jobs[j].g.nx * jobs[j].g.ny;
            }
            if (waste < bestWaste) { bestWaste = (int)std::min<long long>(waste, 1 << 30); best = r; }
        }
        R = best;
    }
    switch (a.tileCols) {
        case 0:
        case 24: return launch_batch_shape<Shape24>(jobs, njobs, R, s);
        case 12: return launch_batch_shape<Shape12>(jobs, njobs, R, s);
        case 8: return launch_batch_shape<Shape8>(jobs, njobs, R, s);
        default: return set_error(KTM_ERR_ARG, "batch: tileCols must be 0, 8, 12 or 24");
    }
}

namespace {

// One CTA bulk-copies `bytes` into shared memory and sums the landed words into
// out[0].  With stall = 1 thread 0 first waits on a second barrier that nothing
// arrives on: the wait runs out after limitNs and is counted in g_waitStalls,
// then the thread waits (bounded) for its own copy as a stalled tile does.
__global__ void wait_selftest_kernel(const unsigned* __restrict__ src, unsigned bytes, int stall,
                                     unsigned long long limitNs, unsigned* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char buf[];
    __shared__ unsigned long long bar[2];
    __shared__ int landed;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        bulk_g2s(buf, src, bytes, &bar[0]);
        if (stall && !mbar_wait_bounded(&bar[1], 0, limitNs)) atomicAdd(&g_waitStalls, 1u);
        landed = mbar_wait_bounded(&bar[0], 0, limitNs) ? 1 : 0;
        if (!landed) atomicAdd(&g_waitStalls, 1u);
        mbar_inval(&bar[0]);
        mbar_inval(&bar[1]);
    }
    __syncthreads();
    if (!landed) return;
    const unsigned* w = reinterpret_cast<const unsigned*>(buf);
    unsigned sum = 0;
    for (unsigned i = threadIdx.x; i < bytes / 4; i += blockDim.x) sum += w[i];
    atomicAdd(out, sum);
}

}  // namespace

int take_wait_stalls(cudaStream_t s, bool deviceSync, unsigned* n)
{
    unsigned v = 0;
    if (deviceSync) KTM_CUDA_TRY(cudaDeviceSynchronize());
    KTM_CUDA_TRY(cudaMemcpyFromSymbolAsync(&v, g_waitStalls, sizeof(v), 0, cudaMemcpyDeviceToHost, s));
    KTM_CUDA_TRY(cudaStreamSynchronize(s));
    if (v) {
        static const unsigned zero = 0;
        KTM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_waitStalls, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s));
        KTM_CUDA_TRY(cudaStreamSynchronize(s));
    }
    *n = v;
    return KTM_OK;
}

int copy_wait_stalls(void* dst, cudaStream_t s)
{
    KTM_CUDA_TRY(cudaMemcpyFromSymbolAsync(dst, g_waitStalls, sizeof(unsigned), 0, cudaMemcpyDeviceToDevice, s));
    return KTM_OK;
}

int wait_selftest(int stall, unsigned long long limitNs, unsigned* checksum)
{
    constexpr unsigned kBytes = 64 * 1024, kWords = kBytes / 4;
    cudaStream_t s = 0;
    void* mem = nullptr;
    KTM_CUDA_TRY(pool_malloc(&mem, kBytes + 64, s));
    unsigned* src = static_cast<unsigned*>(mem);
    unsigned* out = src + kWords;
    int rc = KTM_OK;
    cudaError_t e = cudaMemsetAsync(src, 0x01, kBytes, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(out, 0, 64, s);
    if (e == cudaSuccess) e = allow_smem(wait_selftest_kernel, kBytes, kBytes);
    if (e == cudaSuccess) {
        wait_selftest_kernel<<<1, 256, kBytes, s>>>(src, kBytes, stall, limitNs, out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(checksum, out, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) rc = set_error(KTM_ERR_CUDA, "wait self-test: %s", cudaGetErrorString(e));
    cudaFreeAsync(mem, s);
    return rc;
}

}  // namespace ktm
