// ves_fx.cu -- kernels of the fixed-point FP64 solve (ves_fx.cuh): fixed-size
// batches, with and without eigenvectors, optionally over a device list.
#include "ves_fx.cuh"
#include "ves_internal.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace ves {

namespace {

// Matrices to work on: the batch, or a list whose length lies in the launch's range.
__device__ __forceinline__ long long fx_count(const FxArgs &a)
{
    if (!a.list) return a.g.N;
    const long long c = *a.list_count;
    return c > a.list_above && c <= a.list_upto ? c : 0;
}

template <int G> struct FxShape {
    static constexpr int threads = G > 32 ? G : 32;
    static constexpr int mats = G < 32 ? 32 / G : 1;  // matrices per block
};

template <int G, bool kVec>
__global__ void __launch_bounds__(FxShape<G>::threads) fx_kernel(const FxArgs a)
{
    extern __shared__ longlong2 fxsm[];
    const FxGroup<G> gr;
    constexpr int M = FxShape<G>::mats;
    const int n = a.g.n, tc = a.g.tc;
    longlong2 *sm = fxsm + (G < 32 ? (threadIdx.x / G) * fx_slot(n, G, kVec) : 0);
    const int lda = fx_lda(n);
    const FxMat<1> H{sm, lda, n}, Z{sm + (kVec ? n * lda : 0), lda, n};
    const FxVec<1> U{sm + (kVec ? 2 : 1) * n * lda};
    VES_CHECK_SMEM(fxsm, fxsm + M * fx_slot(n, G, kVec));
    const long long Nw = fx_count(a);
    for (long long base = (long long)blockIdx.x * M; base < Nw; base += (long long)gridDim.x * M) {
        const long long w = base + (G < 32 ? threadIdx.x / G : 0);
        const bool valid = w < Nw;
        const long long m = !valid ? 0 : a.list ? (long long)a.list[w] : a.m_begin + w;
        const long long mo = (m / tc) * (long long)tc * n * n + m % tc, vo = (m / tc) * (long long)tc * n + m % tc;
        FxOut o{a.rE + vo, a.iE + vo, nullptr, nullptr, nullptr, nullptr, tc, tc};
        if (kVec) {
            o.rV = a.rV + mo;
            o.iV = a.iV + mo;
            if (a.rT) { o.rT = a.rT + mo; o.iT = a.iT + mo; }
        }
        int sweeps = 0, status = 0;
        const bool ok = fx_solve<G, kVec>(gr, n, H, Z, U, valid, a.rA + mo, a.iA + mo, tc, o, a.max_its,
                                          a.vnorm, sweeps, status);
        if (valid && gr.gl == 0) {
            if (ok) {
                if (a.status) a.status[m] = status | a.status_or;
                if (a.sweeps) a.sweeps[m] = sweeps;
            } else {
                a.out_list[atomicAdd(a.out_count, 1)] = (int)m;
            }
        }
    }
}

// One matrix per lane, or per G lanes, the warp's 32 / G matrices in lockstep,
// H, Z and U in the warp's workspace ([element][matrix]): the FP64 steps of a
// rotation serve all of them.  kShifts: with predicted shifts (G = 1), whose
// storage follows U in the slot.
constexpr int kLaneThreads = 128;
template <int G, bool kVec, bool kShifts>
__device__ __forceinline__ void fx_lanes(const FxArgs &a)
{
    constexpr int kChunk = FxChunkOf<G>::k, kSlots = FxChunkOf<G>::slots, M = 32 / G;
    __shared__ longlong2 chs[kLaneThreads * kSlots];
    __shared__ i64 chi[kLaneThreads * kChunk];
    const FxLanes<G> gr;
    const int n = a.g.n, tc = a.g.tc, lane = threadIdx.x & 31, mat = lane % M;
    const int warp0 = (threadIdx.x >> 5) * 32;
    const FxChunk ch{chs + warp0 * kSlots + lane, chi + warp0 * kChunk + lane};
    const long long slot = (long long)blockIdx.x * (kLaneThreads / 32) + (threadIdx.x >> 5);
    const long long nslots = (long long)gridDim.x * (kLaneThreads / 32);
    const long long nn = (long long)n * n, nu = (kVec ? 2 : 1) * nn;
    longlong2 *base = static_cast<longlong2 *>(a.ws) + slot * (kShifts ? shift_slot_elems(n) : nu + n) * M + mat;
    const FxMat<M> H{base, n, n}, Z{base + (kVec ? nn * M : 0), n, n};
    const FxVec<M> U{base + nu * M};
    const long long Nw = fx_count(a);
    for (long long group = slot; group * M < Nw;) {
        const long long w = group * M + mat;
        const bool valid = w < Nw;
        const long long m = !valid ? 0 : a.list ? (long long)a.list[w] : a.m_begin + w;
        const long long mo = (m / tc) * (long long)tc * n * n + m % tc, vo = (m / tc) * (long long)tc * n + m % tc;
        FxOut o{a.rE + vo, a.iE + vo, nullptr, nullptr, nullptr, nullptr, tc, tc};
        if (kVec) {
            o.rV = a.rV + mo;
            o.iV = a.iV + mo;
            if (a.rT) { o.rT = a.rT + mo; o.iT = a.iT + mo; }
        }
        int sweeps = 0, status = 0;
        bool ok;
        if constexpr (kShifts) {
            FxShifts sh;
            float2 *const region = reinterpret_cast<float2 *>(base - lane + (nu + n) * 32);
            sh.Hf = MatIlv<float>{region + lane, n};
            sh.P = VecIlv<double>{reinterpret_cast<double2 *>(base + (nu + n + (nn + 1) / 2) * 32)};
            sh.scratch = n >= 6 ? Z.p : base + (shift_slot_elems(n) - 6 * n) * 32;
            sh.polish = a.shift_polish;
            sh.newton = a.shift_newton64;
            sh.sweeps_used = a.shift_sweeps;
            sh.gate = a.shift_gate;
            for (int k = 1; k <= n; ++k)
                sh.P.st(k, valid ? mk(a.rS[vo + (long long)(k - 1) * tc], a.iS[vo + (long long)(k - 1) * tc]) : mk(0.0, 0.0));
            ok = fx_solve<1, kVec>(gr, n, H, Z, U, valid, a.rA + mo, a.iA + mo, tc, o, a.max_its, a.vnorm, sweeps,
                                   status, ch, &sh);
            if (ok && sh.sp.fallbacks) status |= ST_SHIFT_FALLBACK;
            if (ok && a.fallbacks) a.fallbacks[m] = sh.sp.fallbacks;
        } else {
            ok = fx_solve<G, kVec>(gr, n, H, Z, U, valid, a.rA + mo, a.iA + mo, tc, o, a.max_its, a.vnorm, sweeps,
                                   status, ch);
        }
        if (valid && gr.gl == 0) {
            if (ok) {
                if (a.status) a.status[m] = status | a.status_or;
                if (a.sweeps) a.sweeps[m] = sweeps;
            } else {
                a.out_list[atomicAdd(a.out_count, 1)] = (int)m;
            }
        }
        // the first group is the slot's, the next ones whichever warp is free takes
        // (fixed strides -> this: n=16 x 1,048,576 255.5 -> 247.6 ms, n=32 x 131,072
        // 200 -> 190, n=48 x 20,000 166 -> 154)
        if (nslots * M >= Nw) break;
        int next = 0;
        if (lane == 0) next = atomicAdd(a.out_count + 1, 1);
        group = nslots + __shfl_sync(FULL, next, 0);
    }
}
template <int G, bool kVec> __global__ void __launch_bounds__(kLaneThreads, 4) fx_lane_kernel(const FxArgs a)
{
    fx_lanes<G, kVec, false>(a);
}
__global__ void __launch_bounds__(kLaneThreads, 4) fx_shifts_kernel(const FxArgs a) { fx_lanes<1, true, true>(a); }

int fx_sms()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

template <int G> size_t fx_smem(int n, bool vec) { return (size_t)FxShape<G>::mats * fx_slot(n, G, vec) * sizeof(longlong2); }
constexpr size_t kMaxSmem = 227 * 1024;

// Blocks that fit an SM: 228 KB of shared memory (1 KB of it per block is the
// system's) and 64 K registers (168 a thread for one warp, at most 128 for more).
int fx_blocks_per_sm(int G, size_t smem)
{
    const int regs = G > 32 ? G * 128 : 32 * 168;
    return std::max(1, (int)std::min<size_t>(228 * 1024 / (smem + 1024), (size_t)65536 / regs));
}

template <int G, bool kVec> cudaError_t launch_fx_g(const FxArgs &a, cudaStream_t st)
{
    const size_t smem = fx_smem<G>(a.g.n, kVec);
    if (smem > kMaxSmem) return cudaErrorInvalidValue;
    const long long work = a.list ? std::min(a.g.N, a.list_upto) : a.g.N;
    const long long need = (work + FxShape<G>::mats - 1) / FxShape<G>::mats;
    const long long blocks = std::min<long long>(need, (long long)fx_sms() * fx_blocks_per_sm(G, smem));
    fx_kernel<G, kVec><<<(unsigned)std::max<long long>(blocks, 1), FxShape<G>::threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <bool kVec> cudaError_t launch_fx_v(const FxArgs &a, int G, cudaStream_t st)
{
    switch (G) {
    case 4: return launch_fx_g<4, kVec>(a, st);
    case 8: return launch_fx_g<8, kVec>(a, st);
    case 16: return launch_fx_g<16, kVec>(a, st);
    case 32: return launch_fx_g<32, kVec>(a, st);
    case 64: return launch_fx_g<64, kVec>(a, st);
    default: return launch_fx_g<128, kVec>(a, st);
    }
}

}  // namespace

// Which kernel, and how many lanes per matrix.  The lane kernel's warps hold
// 32 / G matrices in the workspace (G = 1, 2, 4, 8) and share the FP64 steps;
// the group kernel keeps a matrix in shared memory (G = 4 .. 128).  More lanes
// finish a matrix sooner; fewer waste less.  The rule takes the smallest
// estimated time, x = n / 8:
//   lanes  (0.07 + 1.05 x^2.66) ms r (1 + c w) for a wave of w * 2,432 warps, r =
//          a + (1 - a) / G, a = 1.9 / n^0.62 the share of a rotation that all
//          lanes repeat, c = 1.5, 1.2, 1.3, 0.8 for G = 1, 2, 4, 8
//   group  waves * 0.33 ms x^1.85 (1 + n / (3 G)), and for G > 32, whose
//          warps repeat the FP64 steps, 3% per warp on the SM
// Measured on GB300, ms.  Lanes G = 1, 2, 4, 8: n=16, N=96 6.35 5.35 3.86 3.02,
// N=16,384 8.05 6.97 7.21 11.8, N=65,536 14.3 20.3 33.2 49.1; n=32, N=4,096 48 36.0
// 23.6 19.3, N=16,384 59.5 48.9 40.5 59.9; n=64, N=96 292 207 123 80, N=4,096
// 360 278 174 135.  Group G = 4, 8, 16, 32: n=16, N=64 2.41 1.70 1.35 1.19,
// N=2,048 2.57 1.85 1.68 2.47, N=8,192 7.43 5.65 5.69 9.40; G = 16, 32, 64: n=32,
// N=64 6.05 4.83 4.28, N=8,192 53.8 47.7 65.2; G = 64, 128: n=64, N=512 68.2 64.1.
// Without vectors 0.9 of the group's time, and lanes (0.066 + 0.43 x^2.66) ms times
// the larger of r (a = 3 / n^0.62) and {1, 0.57, 0.2, 0.15} + 1.64 w: n=24, N=10,000
// G = 1, 2, 4, 8: 9.98 8.00 8.05 11.2; N=30,720 14.0 15.1 23.3 39.3.
struct FxChoice {
    bool lanes;
    int G;
};
// x^p of the fits, x = n / 8
double fx_pow(int n, double p) { return pow(n / 8.0, p); }
// ms of the lane kernel with G = 2^k lanes per matrix; N = 0: of a warp alone
double fx_lane_ms(int n, long long N, int k, bool vec)
{
    const double lat = vec ? 0.07 + 1.05 * fx_pow(n, 2.66) : 0.066 + 0.43 * fx_pow(n, 2.66);
    const double a = std::min(1.0, (vec ? 1.9 : 3.0) / pow(n, 0.62));
    const double c[4] = {1.5, 1.2, 1.3, 0.8}, r[4] = {1, 0.57, 0.2, 0.15};
    const int G = 1 << k;
    const double w = (double)N * G / 32 / (fx_sms() * 16.0), full = floor(w), alone = a + (1 - a) / G;
    return lat * (N == 0 ? alone
                  : vec  ? alone * (full * (1 + c[k]) + (w > full ? 1 + c[k] * (w - full) : 0))
                         : std::max(alone, r[k] + 1.64 * w));
}
// matrices of a wave of the group kernel, and ms of N matrices (G fits: fx_group_fits)
long long fx_group_wave(int n, int G, bool vec)
{
    const int mats = G < 32 ? 32 / G : 1;
    return (long long)fx_sms() * mats * fx_blocks_per_sm(G, (size_t)mats * fx_slot(n, G, vec) * sizeof(longlong2));
}
double fx_group_ms(int n, long long N, int G, bool vec)
{
    const int mats = G < 32 ? 32 / G : 1;
    const double wave = (double)fx_group_wave(n, G, vec);
    double t = ceil(N / wave) * (vec ? 0.33 : 0.30) * fx_pow(n, 1.85) * (1.0 + n / ((vec ? 3.0 : 5.0) * G));
    if (G > 32) t *= 1.0 + 0.03 * std::min(wave / (fx_sms() * mats), ceil((double)N / (fx_sms() * mats))) * G / 32;
    return t;
}
bool fx_group_fits(int n, int G, bool vec)
{
    return G <= (G > 32 ? 2 : 4) * n && (size_t)(G < 32 ? 32 / G : 1) * fx_slot(n, G, vec) * sizeof(longlong2) <= kMaxSmem;
}
int fx_best_group(int n, long long N, bool vec)
{
    int best = 0;
    for (int G = 4; G <= 128; G *= 2)
        if (fx_group_fits(n, G, vec) && (!best || fx_group_ms(n, N, G, vec) < fx_group_ms(n, N, best, vec))) best = G;
    return best;
}
bool fx_forced(FxChoice &c)
{
    if (const char *e = getenv("VES_FX_LANES")) {  // tuning: 1, 2, 4, 8 lanes ("l4"), or a group of 4 .. 128 ("g16")
        const int v = atoi(e + (*e != 0));
        if (e[0] == 'l' && (v == 1 || v == 2 || v == 4 || v == 8)) { c = {true, v}; return true; }
        if (e[0] == 'g' && v >= 4 && v <= 128 && (v & (v - 1)) == 0) { c = {false, v}; return true; }
    }
    return false;
}
FxChoice fx_choose(int n, long long N, bool vec)
{
    FxChoice best{true, 1};
    if (fx_forced(best)) return best;
    double t = 1e300;
    for (int k = 0; k < 4; ++k) {
        const double tl = fx_lane_ms(n, N, k, vec);
        if (tl < t) {
            t = tl;
            best = {true, 1 << k};
        }
    }
    const int G = fx_best_group(n, N, vec);
    if (G && fx_group_ms(n, N, G, vec) < t) best = {false, G};
    return best;
}

template <int G> static void launch_fx_lanes_g(const FxArgs &a, bool vec, cudaStream_t st)
{
    // G times the warps in the same workspace, at most the four blocks that fit an SM
    const long long per_block = kLaneThreads / G;
    long long blocks = std::min<long long>((a.g.N + per_block - 1) / per_block, (long long)a.lane_blocks * G);
    if (G > 1) blocks = std::min<long long>(blocks, std::max(a.lane_blocks, fx_sms() * 4));
    if (vec) fx_lane_kernel<G, true><<<(unsigned)blocks, kLaneThreads, 0, st>>>(a);
    else fx_lane_kernel<G, false><<<(unsigned)blocks, kLaneThreads, 0, st>>>(a);
}

cudaError_t launch_fx_lanes(const FxArgs &a, bool vec, int G, cudaStream_t st)
{
    if (G == 2) launch_fx_lanes_g<2>(a, vec, st);
    else if (G == 4) launch_fx_lanes_g<4>(a, vec, st);
    else if (G == 8) launch_fx_lanes_g<8>(a, vec, st);
    else launch_fx_lanes_g<1>(a, vec, st);
    return cudaGetLastError();
}

cudaError_t launch_fx_shifts(const FxArgs &a, cudaStream_t st)
{
    fx_shifts_kernel<<<a.lane_blocks, kLaneThreads, 0, st>>>(a);
    return cudaGetLastError();
}

static cudaError_t launch_fx_group(const FxArgs &a, bool vec, int G, cudaStream_t st)
{
    return vec ? launch_fx_v<true>(a, G, st) : launch_fx_v<false>(a, G, st);
}

// A list's length is known to the device only.  A lone warp of the lane kernel
// takes as long as a full one, so up to the length whose waves of the group kernel
// (with the G that is best for a matrix per SM) take that long, the group kernel
// has the list, else the lane kernel; the other launch returns at once.  One matrix
// that falls back from FP32+refine, the lane kernel alone -> this, ms added: n=16 x
// 524,288 6.6 -> 1.0, n=32 x 65,536 42.3 -> 4.0, n=64 x 8,192 68.5 -> 16.0; a list
// of 8,192 at n=32 51.3 -> 51.4.
cudaError_t launch_fx(const FxArgs &a, bool vec, cudaStream_t st)
{
    if (a.g.N <= 0) return cudaSuccess;
    const int n = a.g.n;
    if (!fx_order(n)) return cudaErrorInvalidValue;
    FxChoice c = fx_choose(n, a.g.N, vec);
    FxArgs f = a;
    f.list_above = 0;
    f.list_upto = a.g.N;
    if (a.list && c.lanes && !fx_forced(c)) {
        const int G = fx_best_group(n, fx_sms(), vec);
        const long long wave = G ? fx_group_wave(n, G, vec) : 0;
        const double lone = fx_lane_ms(n, 0, c.G == 1 ? 0 : c.G == 2 ? 1 : c.G == 4 ? 2 : 3, vec);
        if (wave) f.list_upto = wave * std::max(1LL, (long long)(lone / fx_group_ms(n, wave, G, vec)));
        if (wave) {
            const cudaError_t e = launch_fx_group(f, vec, G, st);
            if (e != cudaSuccess || f.list_upto >= a.g.N) return e;
            f.list_above = f.list_upto;
            f.list_upto = a.g.N;
        }
    }
    return c.lanes ? launch_fx_lanes(f, vec, c.G, st) : launch_fx_group(f, vec, c.G, st);
}

template <int G> static void load_fx_g()
{
    load_kernel(fx_kernel<G, true>);
    load_kernel(fx_kernel<G, false>);
    cudaFuncSetAttribute(fx_kernel<G, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
    cudaFuncSetAttribute(fx_kernel<G, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
}
void load_fx_kernels()
{
    load_kernel(fx_lane_kernel<1, true>);
    load_kernel(fx_lane_kernel<1, false>);
    load_kernel(fx_lane_kernel<2, true>);
    load_kernel(fx_lane_kernel<2, false>);
    load_kernel(fx_lane_kernel<4, true>);
    load_kernel(fx_lane_kernel<4, false>);
    load_kernel(fx_lane_kernel<8, true>);
    load_kernel(fx_lane_kernel<8, false>);
    load_kernel(fx_shifts_kernel);
    load_fx_g<4>(); load_fx_g<8>(); load_fx_g<16>(); load_fx_g<32>(); load_fx_g<64>();
    load_fx_g<128>();
}

}  // namespace ves
