// cuda_runtime.h for the CPU -- enough of CUDA's device language to run the solver's device
// functions on the CPU: a block's threads are fibers that switch only at
// collectives (warp votes, shuffles, barriers), so each runs alone from one
// collective to the next, in an order the caller chooses.  Code whose result
// depends on how lanes are interleaved between two collectives gives another
// result under another order; a collective that its lanes reach at different
// places (source line, matrix, or count) is reported.
#pragma once

#include <ucontext.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

using std::copysign;
using std::fabs;
using std::fma;
using std::fmax;
using std::fmin;
using std::max;
using std::min;
using std::sqrt;

#define __host__
#define __device__
#define __global__
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)

struct float2 { float x, y; };
struct double2 { double x, y; };
struct longlong2 { long long x, y; };
inline float2 make_float2(float a, float b) { return {a, b}; }
inline double2 make_double2(double a, double b) { return {a, b}; }
inline longlong2 make_longlong2(long long a, long long b) { return {a, b}; }

namespace host {

enum Kind { kSync, kAny, kBallot, kShfl, kMin, kMax, kOr, kBlock };
struct Fiber {
    ucontext_t ctx;
    std::vector<char> stack;
    bool done = false, waiting = false;
    // the collective it waits at: what the lanes that meet there must agree on
    int kind = 0, line = 0, src = 0;
    long long epoch = 0, count = 0;
    unsigned mask = 0;
    uint64_t value = 0, result = 0;
};
struct Block {
    std::vector<Fiber> f;
    ucontext_t main;
    int cur = 0;
    std::string error;
};
inline Block *blk = nullptr;
struct Dim { int x = 0, y = 0, z = 0; };

inline uint64_t meet(int kind, int line, unsigned mask, uint64_t value, int src)
{
    Fiber &f = blk->f[blk->cur];
    if (mask == 0xffffffffu || kind == kBlock) ++f.count;
    f.waiting = true;
    f.kind = kind; f.line = line; f.mask = mask; f.value = value; f.src = src;
    swapcontext(&f.ctx, &blk->main);
    return f.result;
}
// lanes [base, base + 32) whose mask is m all wait: give each its result
inline void complete(const std::vector<int> &who)
{
    const Fiber &a = blk->f[who[0]];
    uint64_t any = 0, ballot = 0;
    int mn = INT_MAX, mx = INT_MIN;
    for (int t : who) {
        const Fiber &b = blk->f[t];
        if (b.kind != a.kind || b.line != a.line || b.epoch != a.epoch || (a.mask == 0xffffffffu && b.count != a.count)) {
            char s[200];
            snprintf(s, sizeof s, "threads %d and %d meet at lines %d and %d, matrices %lld and %lld, collectives %lld and %lld",
                     who[0], t, a.line, b.line, a.epoch, b.epoch, a.count, b.count);
            blk->error = s;
            return;
        }
        any |= b.value;
        if (b.value) ballot |= 1ull << (t & 31);
        mn = std::min(mn, (int)b.value);
        mx = std::max(mx, (int)b.value);
    }
    const int kind = a.kind;
    for (int t : who) {
        Fiber &b = blk->f[t];
        b.result = kind == kAny || kind == kBlock ? any != 0 : kind == kBallot ? ballot : kind == kMin ? (uint64_t)mn :
                   kind == kMax ? (uint64_t)mx : kind == kOr ? any : kind == kShfl ? blk->f[(t & ~31) + b.src].value : 0;
    }
    for (int t : who) blk->f[t].waiting = false;
}

// Runs body() as `threads` threads of one block.  order: 0 ascending, 1
// descending, else a random order per round.  Returns what went wrong, or "".
inline std::string run(int threads, int order, Dim &tid, const std::function<void()> &body)
{
    static std::function<void()> entry;
    entry = body;
    Block b;
    blk = &b;
    b.f.resize(threads);
    for (auto &f : b.f) {
        f.stack.resize(256 * 1024);
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = f.stack.data();
        f.ctx.uc_stack.ss_size = f.stack.size();
        f.ctx.uc_link = &b.main;
        makecontext(&f.ctx, +[] { entry(); blk->f[blk->cur].done = true; }, 0);
    }
    uint64_t seed = 88172645463325252ull + order;
    std::vector<int> seq(threads);
    for (;;) {
        for (int i = 0; i < threads; ++i) seq[i] = order == 1 ? threads - 1 - i : i;
        if (order > 1)
            for (int i = threads - 1; i > 0; --i) {
                seed ^= seed << 13; seed ^= seed >> 7; seed ^= seed << 17;
                std::swap(seq[i], seq[seed % (i + 1)]);
            }
        bool ran = false, alive = false;
        for (int t : seq) {
            Fiber &f = b.f[t];
            if (f.done || f.waiting) continue;
            b.cur = t;
            tid.x = t;
            swapcontext(&b.main, &f.ctx);
            ran = true;
        }
        for (int t = 0; t < threads; ++t) {
            Fiber &f = b.f[t];
            alive |= !f.done;
            if (f.done || !f.waiting) continue;
            std::vector<int> who;
            bool all = true;
            if (f.kind == kBlock) {
                for (int u = 0; u < threads; ++u) { all &= b.f[u].waiting && b.f[u].kind == kBlock; who.push_back(u); }
            } else {
                for (int u = 0; u < 32; ++u)
                    if (f.mask >> u & 1) {
                        const Fiber &g = b.f[(t & ~31) + u];
                        all &= g.waiting && g.mask == f.mask && g.kind != kBlock;
                        who.push_back((t & ~31) + u);
                    }
            }
            if (all) complete(who);
            if (!b.error.empty()) return b.error;
        }
        if (!alive) return "";
        if (!ran) {
            bool wake = false;
            for (auto &f : b.f) wake |= !f.done && !f.waiting;
            if (!wake) {
                for (int t = 0; t < threads; ++t)
                    if (!b.f[t].done)
                        return "thread " + std::to_string(t) + " waits at line " + std::to_string(b.f[t].line) + " for lanes that never come";
            }
        }
    }
}

template <class T> uint64_t raw(T v) { uint64_t r = 0; memcpy(&r, &v, sizeof v); return r; }
template <class T> T shfl(int line, unsigned mask, T v, int src)
{
    const uint64_t r = meet(kShfl, line, mask, raw(v), src);
    T out;
    memcpy(&out, &r, sizeof out);
    return out;
}
inline unsigned mask_of(unsigned m = 0xffffffffu) { return m; }
inline int lane() { return blk->cur & 31; }

}  // namespace host

static host::Dim threadIdx, blockIdx, blockDim, gridDim;
#define __syncwarp(...) host::meet(host::kSync, __LINE__, host::mask_of(__VA_ARGS__), 0, 0)
#define __syncthreads() host::meet(host::kBlock, __LINE__, 0, 0, 0)
#define __any_sync(m, p) (bool)host::meet(host::kAny, __LINE__, m, (bool)(p), 0)
#define __ballot_sync(m, p) (unsigned)host::meet(host::kBallot, __LINE__, m, (bool)(p), 0)
#define __reduce_min_sync(m, v) (int)host::meet(host::kMin, __LINE__, m, (uint64_t)(v), 0)
#define __reduce_max_sync(m, v) (int)host::meet(host::kMax, __LINE__, m, (uint64_t)(v), 0)
#define __shfl_xor_sync_3(m, v, o) host::shfl(__LINE__, m, v, host::lane() ^ (o))
#define __shfl_xor_sync_4(m, v, o, w) host::shfl(__LINE__, m, v, host::lane() ^ (o))
#define __shfl_sync_3(m, v, s) host::shfl(__LINE__, m, v, (s) & 31)
#define __shfl_sync_4(m, v, s, w) host::shfl(__LINE__, m, v, (host::lane() & ~((w) - 1)) + ((s) & ((w) - 1)))
#define HOST_PICK(_1, _2, _3, _4, name, ...) name
#define __shfl_xor_sync(...) HOST_PICK(__VA_ARGS__, __shfl_xor_sync_4, __shfl_xor_sync_3, 0, 0)(__VA_ARGS__)
#define __shfl_sync(...) HOST_PICK(__VA_ARGS__, __shfl_sync_4, __shfl_sync_3, 0, 0)(__VA_ARGS__)

inline int __double2hiint(double d) { return (int)(host::raw(d) >> 32); }
inline int __double2loint(double d) { return (int)host::raw(d); }
inline double __longlong_as_double(long long v) { double d; memcpy(&d, &v, 8); return d; }
inline double __hiloint2double(int h, int l) { return __longlong_as_double((long long)(((uint64_t)(unsigned)h << 32) | (unsigned)l)); }
inline unsigned __float_as_uint(float f) { return (unsigned)host::raw(f); }
inline int __float_as_int(float f) { return (int)host::raw(f); }
inline float __int_as_float(int v) { float f; memcpy(&f, &v, 4); return f; }
inline long long __double2ll_rn(double d) { return llrint(d); }
inline long long __float2ll_rn(float f) { return llrintf(f); }
inline int __float2int_rn(float f) { return (int)lrintf(f); }
inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) { return (unsigned long long)(((unsigned __int128)a * b) >> 64); }
inline int __clz(int x) { return x ? __builtin_clz(x) : 32; }
inline int __clzll(long long x) { return x ? __builtin_clzll(x) : 64; }
inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) { return s & 31 ? (hi << (s & 31)) | (lo >> (32 - (s & 31))) : hi; }
inline int __ffsll(long long x) { return __builtin_ffsll(x); }
inline int __ffs(int x) { return __builtin_ffs(x); }
inline double rsqrt(double x) { return 1.0 / sqrt(x); }
inline float rsqrtf(float x) { return 1.0f / sqrtf(x); }
inline float __fdividef(float a, float b) { return a / b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsqrt_rn(float a) { return std::sqrt(a); }
inline float __frcp_rn(float a) { return 1.f / a; }
