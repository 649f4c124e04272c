// The fixed-point solve (ves_fx.cuh) on the CPU, one block at a time: the loops
// of fx_kernel (matrices in shared memory, G lanes each) and fx_lane_kernel
// (32 / G matrices in a warp's workspace).  Matrix m is column-major at m n n.
#include "cuda_runtime.h"

#include "ves_fx.cuh"

using namespace ves;

namespace {

struct Batch {
    int n, N;
    const double *rA, *iA;
    double *rE, *iE, *rV, *iV;
    int *ok, *sweeps;
};

FxOut out_of(const Batch &b, long long m, bool vec)
{
    const long long mo = m * b.n * b.n, vo = m * b.n;
    return {b.rE + vo, b.iE + vo, vec ? b.rV + mo : nullptr, vec ? b.iV + mo : nullptr, nullptr, nullptr, 1, 1};
}

template <int G, bool kVec> std::string group(const Batch &b, int order)
{
    constexpr int T = G > 32 ? G : 32, M = G < 32 ? 32 / G : 1;
    const int n = b.n, lda = fx_lda(n), slot = fx_slot(n, G, kVec);
    std::vector<longlong2> sm((size_t)M * slot, longlong2{0x7ff8000000000000ll, 0x7ff8000000000000ll});
    return host::run(T, order, threadIdx, [&] {
        const FxGroup<G> gr;
        const int t = threadIdx.x, g = G < 32 ? t / G : 0;
        longlong2 *p = sm.data() + g * slot;
        const FxMat<1> H{p, lda, n}, Z{p + (kVec ? n * lda : 0), lda, n};
        const FxVec<1> U{p + (kVec ? 2 : 1) * n * lda};
        for (long long base = 0; base < b.N; base += M) {
            host::blk->f[t].epoch = base;
            const long long w = base + g;
            const bool valid = w < b.N;
            const long long m = valid ? w : 0, mo = m * n * n;
            int sweeps = 0, status = 0;
            const bool ok = fx_solve<G, kVec>(gr, n, H, Z, U, valid, b.rA + mo, b.iA + mo, 1, out_of(b, m, kVec), 30, 2, sweeps,
                                              status);
            if (valid && gr.gl == 0) { b.ok[m] = ok ? 1 + status : 0; b.sweeps[m] = sweeps; }
        }
    });
}

template <int G, bool kVec> std::string lanes(const Batch &b, int order)
{
    constexpr int M = 32 / G, kChunk = FxChunkOf<G>::k;
    const int n = b.n;
    const long long nn = (long long)n * n, nu = (kVec ? 2 : 1) * nn;
    std::vector<longlong2> ws((nu + n) * M, longlong2{0x7ff8000000000000ll, 0x7ff8000000000000ll}), chs(32 * FxChunkOf<G>::slots);
    std::vector<i64> chi(32 * kChunk);
    return host::run(32, order, threadIdx, [&] {
        const FxLanes<G> gr;
        const int lane = threadIdx.x, mat = lane % M;
        const FxChunk ch{chs.data() + lane, chi.data() + lane};
        longlong2 *p = ws.data() + mat;
        const FxMat<M> H{p, n, n}, Z{p + (kVec ? nn * M : 0), n, n};
        const FxVec<M> U{p + nu * M};
        for (long long base = 0; base < b.N; base += M) {
            host::blk->f[lane].epoch = base;
            const long long w = base + mat;
            const bool valid = w < b.N;
            const long long m = valid ? w : 0, mo = m * nn;
            int sweeps = 0, status = 0;
            const bool ok = fx_solve<G, kVec>(gr, n, H, Z, U, valid, b.rA + mo, b.iA + mo, 1, out_of(b, m, kVec), 30, 2, sweeps,
                                              status, ch);
            if (valid && gr.gl == 0) { b.ok[m] = ok ? 1 + status : 0; b.sweeps[m] = sweeps; }
        }
    });
}

template <bool kVec> std::string any_form(const Batch &b, char kind, int G, int order)
{
    if (kind == 'l')
        return G == 1 ? lanes<1, kVec>(b, order) : G == 2 ? lanes<2, kVec>(b, order) : G == 4 ? lanes<4, kVec>(b, order)
                                                                                          : lanes<8, kVec>(b, order);
    return G == 4 ? group<4, kVec>(b, order) : G == 8 ? group<8, kVec>(b, order) : G == 16 ? group<16, kVec>(b, order) :
           G == 32 ? group<32, kVec>(b, order) : group<64, kVec>(b, order);
}

}  // namespace

// kind 'l' or 'g' with G lanes per matrix; ok[m]: 0 = left to the FP64 kernels,
// else 1 + status.  Returns 0, or 1 with what went wrong in msg (256 bytes).
extern "C" int fxh_solve(int kind, int G, int vec, int order, int n, int N, const double *rA, const double *iA, double *rE,
                         double *iE, double *rV, double *iV, int *ok, int *sweeps, char *msg)
{
    const Batch b{n, N, rA, iA, rE, iE, rV, iV, ok, sweeps};
    const std::string e = vec ? any_form<true>(b, (char)kind, G, order) : any_form<false>(b, (char)kind, G, order);
    snprintf(msg, 256, "%s", e.c_str());
    return !e.empty();
}
