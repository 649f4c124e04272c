// The pointer loops' checks of the bounds-checked build, on the CPU: a walk that
// stays in its matrix counts nothing, one that leaves it by an element is counted
// and not taken.
#define VES_BOUNDS_CHECK 1
#include "cuda_runtime.h"

static unsigned long long atomicAdd(unsigned long long *p, unsigned long long v) { *p += v; return *p - v; }
template <class T> void cudaMemcpyFromSymbol(T *d, T &s, size_t) { *d = s; }
template <class T> void cudaMemcpyToSymbol(T &d, const T *s, size_t) { d = *s; }

#include "ves_fx.cuh"

namespace ves {
void register_bounds_counter(unsigned long long (*)(), void (*)()) {}
}  // namespace ves
using namespace ves;

// what: 0 a reflector over `count` columns of an n x n matrix, its vector in column
// `extra`; 1 a chunk of ns rotations streamed over `count` rows; 2 a rotation of the
// chunk's storage at `extra`; 3 a row of the chunk at `extra` (G = 4).  Returns the
// violations; changed: whether any of the guard elements around the matrix were written.
extern "C" long long fxh_bounds(int what, int n, int count, int ns, int extra, int *changed)
{
    const longlong2 mark{0x1234567890abcdefll, 77};
    const int guard = 64 * 64;
    std::vector<longlong2> m(n * n + 2 * guard, mark), cs(64 * 32, longlong2{1ll << 61, 0});
    std::vector<i64> si(64 * 32, 0);
    for (int e = 0; e < n * n; ++e) m[guard + e] = {1ll << 40, 3};
    const FxMat<1> A{m.data() + guard, n, n};
    const FxChunk ch{cs.data(), si.data()};
    g_bounds_violations = 0;
    if (what == 0) fx_reflect_all<1, 1>(0, A, A.p, 1, n, count, A, A.p + (n - ns) + (long long)extra * n, {1, 1}, ns + 1, false);
    if (what == 1) fx_stream_all<1>(0, A, A.p, n, 1, count, ch, ns, true);
    if (what == 2) { FxRot q{}; ch.put(extra, q); ch.get(extra); }
    if (what == 3) *ch.row<4>(extra) = mark;
    *changed = 0;
    for (int k = 0; k < guard; ++k)
        for (longlong2 v : {m[k], m[guard + n * n + k]}) *changed |= v.x != mark.x || v.y != mark.y;
    return (long long)g_bounds_violations;
}
