// common.cuh -- shared device helpers for the subdivision kernels.
//
// Position arithmetic is IEEE binary32 round-to-nearest with no FMA
// contraction (explicit __f*_rn intrinsics, and the library is built with
// -fmad=false), so every float result is reproducible and equals the CPU
// restatement bit for bit.
#pragma once

#include <cstdint>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>
#include <cuda.h>
#include <cuda_runtime.h>

namespace slak {

constexpr int kBlock = 256;

// ------------------------------------------------------- dependent launches
// Programmatic dependent launch: every kernel is launched with the
// programmatic-serialization attribute and starts with griddep_enter(): it
// waits until the grid before it in the stream has completed and its memory
// is visible (griddepcontrol.wait returns at once when there is none), then
// allows the grid after it to begin launching.  So each launch overlaps the
// tail of the grid before it instead of following its end, while no thread
// touches memory before its predecessor is done.  SLAK_NO_PDL builds launch
// plainly, for comparisons.
__device__ __forceinline__ void griddep_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

#ifdef SLAK_NO_PDL
constexpr bool kUsePdl = false;
#else
constexpr bool kUsePdl = true;
#endif

template <class... KArgs, class... Args>
inline void launch_k(void (*kernel)(KArgs...), unsigned grid, unsigned block, cudaStream_t s, Args&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = kUsePdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// ---------------------------------------------------------- grouped launches
// Every kernel a plan launches is written as a body, a __device__ function of
// its block index (k_*_body); a __global__ wrapper (k_*) runs it for
// blockIdx.x, and a group functor (k_*_g) names it for grouped launches.  A
// grouped launch runs one kernel for many meshes at once: its grid is the
// meshes' grids end to end, and each block finds its mesh in a table of block
// offsets (binary search) and its arguments in an array of argument packs.
// A batch records the launches of its small meshes' plans (launch_g with
// g_record set) and replays each step of a group of plans with identical
// launch sequences as one grouped launch.

// The arguments of one launch, trivially copyable, in one block of bytes.
template <size_t I, class T> struct PackLeaf { T v; };
template <class Seq, class... A> struct PackImpl;
template <size_t... I, class... A>
struct PackImpl<std::index_sequence<I...>, A...> : PackLeaf<I, A>... {
    PackImpl() = default;
    explicit PackImpl(const A&... a) : PackLeaf<I, A>{a}... {}
};
template <class... A> using Pack = PackImpl<std::index_sequence_for<A...>, A...>;

template <class G, size_t... I, class... A>
__device__ __forceinline__ void run_pack(unsigned bx, const PackImpl<std::index_sequence<I...>, A...>& p)
{
    G{}(bx, static_cast<const PackLeaf<I, A>&>(p).v...);
}

// the mesh whose block range [bstart[m], bstart[m+1]) holds this block
__device__ __forceinline__ int group_mesh(const unsigned* __restrict__ bstart, int nm)
{
    int lo = 0, hi = nm - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(bstart + mid) <= blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// G::kBounds: the launch bounds of the kernel's own wrapper (0 none, 1 the
// block size, 2 the block size and blocks per SM), repeated here
template <class G, class P>
__global__ void k_group(const P* __restrict__ args, const unsigned* __restrict__ bstart, int nm)
{
    griddep_enter();
    const int m = group_mesh(bstart, nm);
    run_pack<G>(blockIdx.x - __ldg(bstart + m), args[m]);
}
template <class G, class P>
__global__ void __launch_bounds__(G::kMaxT) k_group_t(const P* __restrict__ args, const unsigned* __restrict__ bstart,
                                                      int nm)
{
    griddep_enter();
    const int m = group_mesh(bstart, nm);
    run_pack<G>(blockIdx.x - __ldg(bstart + m), args[m]);
}
template <class G, class P>
__global__ void __launch_bounds__(G::kMaxT, G::kMinB) k_group_b(const P* __restrict__ args,
                                                                const unsigned* __restrict__ bstart, int nm)
{
    griddep_enter();
    const int m = group_mesh(bstart, nm);
    run_pack<G>(blockIdx.x - __ldg(bstart + m), args[m]);
}

using GroupLaunchFn = void (*)(const void* args, const unsigned* bstart, int nm, unsigned grid, unsigned block,
                               cudaStream_t s);

template <class G, class P>
void group_launch(const void* args, const unsigned* bstart, int nm, unsigned grid, unsigned block, cudaStream_t s)
{
    const P* a = static_cast<const P*>(args);
    if constexpr (G::kBounds == 2) launch_k(k_group_b<G, P>, grid, block, s, a, bstart, nm);
    else if constexpr (G::kBounds == 1) launch_k(k_group_t<G, P>, grid, block, s, a, bstart, nm);
    else launch_k(k_group<G, P>, grid, block, s, a, bstart, nm);
}

// One recorded launch: the grouped launcher of its kernel and argument types
// (which identifies it), its shape and its argument pack.
struct RecLaunch {
    GroupLaunchFn fn = nullptr;
    unsigned grid = 0, block = 0;
    size_t align = 0;
    std::vector<unsigned char> pack;
};
inline thread_local std::vector<RecLaunch>* g_record = nullptr;

template <class G, class... Args>
inline void launch_g(unsigned grid, unsigned block, cudaStream_t s, Args&&... args)
{
    if (g_record) {
        using P = Pack<std::decay_t<Args>...>;
        static_assert(std::is_trivially_copyable<P>::value, "launch arguments must be trivially copyable");
        const P pk(args...);
        RecLaunch r;
        r.fn = &group_launch<G, P>;
        r.grid = grid;
        r.block = block;
        r.align = alignof(P);
        r.pack.resize(sizeof(P));
        std::memcpy(r.pack.data(), &pk, sizeof(P));
        g_record->push_back(std::move(r));
        return;
    }
    launch_k(G::kernel(), grid, block, s, std::forward<Args>(args)...);
}

// ---------------------------------------------------------------- float4 ops
__device__ __forceinline__ float4 f4_add(float4 a, float4 b)
{
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}
__device__ __forceinline__ float4 f4_mul(float4 a, float s)
{
    return make_float4(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s), __fmul_rn(a.w, s));
}
// x / s.  When s is a normal power of two the quotient is an exact scaling, so
// the product with the exact reciprocal 2^-e is the same correctly rounded
// number (also under overflow / underflow) and avoids the IEEE divide sequence.
__device__ __forceinline__ bool pow2_recip(float s, float& r)
{
    const unsigned u = __float_as_uint(s), ex = u & 0x7f800000u;
    if ((u & 0x007fffffu) != 0u || ex == 0u || ex >= 0x7f000000u) return false;
    r = __uint_as_float((0x7f000000u - ex) | (u & 0x80000000u));
    return true;
}
__device__ __forceinline__ float4 f4_div(float4 a, float s)
{
    float r;
    if (pow2_recip(s, r)) return f4_mul(a, r);
    return make_float4(__fdiv_rn(a.x, s), __fdiv_rn(a.y, s), __fdiv_rn(a.z, s), __fdiv_rn(a.w, s));
}
// x / s + 0.0f (turns -0 into +0, as an element-wise divide-then-add does)
__device__ __forceinline__ float4 f4_div_z(float4 a, float s)
{
    float4 q = f4_div(a, s);
    return make_float4(__fadd_rn(q.x, 0.0f), __fadd_rn(q.y, 0.0f), __fadd_rn(q.z, 0.0f), __fadd_rn(q.w, 0.0f));
}
__device__ __forceinline__ float4 f4_zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }

__device__ __forceinline__ float4 ldg4(const float* p, int64_t i)
{
    return __ldg(reinterpret_cast<const float4*>(p) + i);
}
__device__ __forceinline__ void st4(float* p, int64_t i, float4 v)
{
    reinterpret_cast<float4*>(p)[i] = v;
}
// streaming store for outputs that are not read again by this level
__device__ __forceinline__ void st4_cs(float* p, int64_t i, float4 v)
{
    __stcs(reinterpret_cast<float4*>(p) + i, v);
}

// TwoSum (Knuth): s + e == a + b exactly
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
    s = __fadd_rn(a, b);
    float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// (hi, lo) += x, componentwise, with TwoSum: hi + lo carries the sum to about
// twice the working precision
__device__ __forceinline__ void dd_acc1(float& hi, float& lo, float x)
{
    float s, e;
    two_sum(hi, x, s, e);
    hi = s;
    lo = __fadd_rn(lo, e);
}
__device__ __forceinline__ void dd_acc(float4& hi, float4& lo, float4 x)
{
    dd_acc1(hi.x, lo.x, x.x); dd_acc1(hi.y, lo.y, x.y);
    dd_acc1(hi.z, lo.z, x.z); dd_acc1(hi.w, lo.w, x.w);
}

// (sh + sl) / n^2 + p (n-2) / n with exact remainders (fmaf) for both quotients
// and for the product, then a TwoSum of the two quotients; rounded once.
__device__ __forceinline__ float vp_finish1(float sh, float sl, float p, int n)
{
    const float nn = (float)(n * n), fn = (float)n, k = (float)(n - 2);
    float q = __fdiv_rn(sh, nn);
    float ql = __fdiv_rn(__fadd_rn(fmaf(-q, nn, sh), sl), nn);
    float oh = __fmul_rn(p, k);
    float ol = fmaf(p, k, -oh);
    float o = __fdiv_rn(oh, fn);
    float olo = __fdiv_rn(__fadd_rn(fmaf(-o, fn, oh), ol), fn);
    float hi, lo;
    two_sum(q, o, hi, lo);
    return __fadd_rn(hi, __fadd_rn(lo, __fadd_rn(ql, olo)));
}
__device__ __forceinline__ float4 vp_finish(float4 sh, float4 sl, float4 p, int n)
{
    return make_float4(vp_finish1(sh.x, sl.x, p.x, n), vp_finish1(sh.y, sl.y, p.y, n),
                       vp_finish1(sh.z, sl.z, p.z, n), vp_finish1(sh.w, sl.w, p.w, n));
}

// ---------------------------------------------------------------- in-order sums
// add(load(k)) for k = 0..n-1, in that order, with W loads in flight: a
// long column's records come from L2, and a loop that waited for each one
// would pay the full latency per slot.
template <int W = 4, class Load, class Add>
__device__ __forceinline__ void for_each_loaded(int n, Load load, Add add)
{
    for (int k0 = 0; k0 < n; k0 += W) {
        float4 t[W];
#pragma unroll
        for (int i = 0; i < W; ++i)
            if (k0 + i < n) t[i] = load(k0 + i);
#pragma unroll
        for (int i = 0; i < W; ++i)
            if (k0 + i < n) add(k0 + i, t[i]);
    }
}

// ---------------------------------------------------------------- ordering
// Columns longer than kBigCol slots (and up to kWarpCol) are taken by their
// whole warp: ranks and loads run in parallel, and the sums run in the fixed
// order by shuffle (same bits as the single-thread paths).  Shorter columns, and
// longer ones, stay on one thread.
constexpr int kBigCol = 16;
constexpr int kWarpCol = 64;

__device__ __forceinline__ float4 shfl4(float4 v, int src)
{
    return make_float4(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                       __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src));
}

// A long column's keys in its warp: slot k is element k >> 5 of lane k & 31
// (two per lane for up to kWarpCol = 64 slots).  col1 fetches slot k (k the
// same on every lane) from its lane; column_order gives the slots in ascending
// key order, ties by slot: order[rank] = slot, in the warp's row of shared
// memory.
__device__ __forceinline__ int col1(int e0, int e1, int k) { return __shfl_sync(0xffffffffu, k < 32 ? e0 : e1, k & 31); }
__device__ __forceinline__ void column_order(int n, int key0, int key1, unsigned char* order)
{
    const int lane = threadIdx.x & 31;
    int r0 = 0, r1 = 0;
#pragma unroll 8
    for (int j = 0; j < n; ++j) {
        const int y = col1(key0, key1, j);
        r0 += (y < key0) | ((y == key0) & (j < lane));
        r1 += (y < key1) | ((y == key1) & (j < lane + 32));
    }
    if (lane < n) order[r0] = (unsigned char)lane;
    if (lane + 32 < n) order[r1] = (unsigned char)(lane + 32);
    __syncwarp();
}
// A long column's terms, one component per lane: lane l holds component l & 3
// of terms 8j + (l >> 2), j = 0..7, so a step of a sum in column order is one
// shuffle and one scalar add (as float4, two slots per lane, it was four
// shuffles and all four components' adds on every lane).  Such a column is a
// serial chain beside which the level waits: with two 64-slot poles and
// compensated sums (capped cylinder, B200), this, all of a column's loads in
// flight at once and for_each_big took k_g3 of its small levels from 18.4 to
// 14.3 us each (8 us without poles), k_c0_verts from 38 to 15 and k_c0_long from
// 19 to 12 us.
__device__ __forceinline__ int term_slot() { return (threadIdx.x & 31) >> 2; }
__device__ __forceinline__ int term_comp() { return threadIdx.x & 3; }
template <class Add>
__device__ __forceinline__ void each_term(const float (&x)[8], int n, Add add)
{
    const int c = term_comp();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (8 * j >= n) break;
        const int m = n - 8 * j < 8 ? n - 8 * j : 8;
        float t = __shfl_sync(0xffffffffu, x[j], c);
#pragma unroll 1
        for (int i = 1; i <= m; ++i) {          // the next term on its way while this one is added
            const float tn = __shfl_sync(0xffffffffu, x[j], ((4 * i) & 31) + c);
            add(t);
            t = tn;
        }
    }
}
// f(i) by a whole warp for each thread i of the block with `big` set.  SPREAD:
// over the block's warps (the two poles of a sphere are often neighbours, and
// a column's serial sum is microseconds); else by the thread's own warp, without
// a barrier.  Every thread of the block takes part, `spread` the same on all.
template <int BS, class F>
__device__ __forceinline__ void for_each_big(bool big, bool spread, F f)
{
    __shared__ unsigned short list[BS];
    __shared__ int count;
    if (!spread) {
        unsigned m = __ballot_sync(0xffffffffu, big);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            f((int)(threadIdx.x & ~31u) + src);
        }
        return;
    }
    if (!__syncthreads_or(big)) return;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    if (big) list[atomicAdd(&count, 1)] = (unsigned short)threadIdx.x;
    __syncthreads();
    for (int i = threadIdx.x >> 5; i < count; i += BS / 32) f((int)list[i]);
}
__device__ __forceinline__ float div1(float a, float s)
{
    float r;
    return pow2_recip(s, r) ? __fmul_rn(a, r) : __fdiv_rn(a, s);
}
// The vertex point of a column of n slots from its neighbours (SLAK: slot
// order; LAK: ascending id) and face points (slot order); p: component l & 3 of
// the vertex.  Every lane returns the whole point.
template <bool LAK>
__device__ __forceinline__ float4 column_point(const float (&nb)[8], const float (&fp)[8], float p, int n, bool comp)
{
    const float nn = (float)(n * n), fn = (float)n;
    float acc = 0.0f, lo = 0.0f, y;
    const auto sum = [&](float t) { acc = __fadd_rn(acc, t); };
    const auto dd = [&](float t) { dd_acc1(acc, lo, t); };
    if (comp) {
        if (LAK) { each_term(fp, n, dd); each_term(nb, n, dd); }
        else { each_term(nb, n, dd); each_term(fp, n, dd); }
        y = vp_finish1(acc, lo, p, n);
    } else if (!LAK) {
        each_term(nb, n, sum);
        y = __fadd_rn(div1(acc, nn), div1(__fmul_rn(p, (float)(n - 2)), fn));
        each_term(fp, n, [&](float t) { y = __fadd_rn(y, div1(t, nn)); });
    } else {
        each_term(fp, n, sum);
        each_term(nb, n, sum);
        const float m = __fadd_rn(div1(acc, fn), 0.0f);
        y = __fadd_rn(div1(__fadd_rn(m, __fmul_rn(p, __fadd_rn(fn, -2.0f))), fn), 0.0f);
    }
    return make_float4(__shfl_sync(0xffffffffu, y, 0), __shfl_sync(0xffffffffu, y, 1), __shfl_sync(0xffffffffu, y, 2),
                       __shfl_sync(0xffffffffu, y, 3));
}
__device__ __forceinline__ float ldg1(const float* p, int64_t i, int c) { return __ldg(p + 4 * i + c); }

// The slots k = 0..n-1 of key[b..b+n) in ascending key order (equal keys by
// slot): perm[r] = the slot of rank r.  n^2 independent compares, instead of
// n selection passes that each wait for the previous minimum; for one thread's
// columns of 5 to kBigCol slots (shorter ones are ranked in registers).
__device__ __forceinline__ void rank_order(const int* __restrict__ key, int b, int n, int* perm)
{
    for (int k = 0; k < n; ++k) {
        const int x = __ldg(key + b + k);
        int r = 0, j = 0;
        for (; j + 8 <= n; j += 8) {          // eight loads in flight before the compares
            int y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = __ldg(key + b + j + i);
#pragma unroll
            for (int i = 0; i < 8; ++i) r += (y[i] < x) | ((y[i] == x) & (j + i < k));
        }
        for (; j < n; ++j) {
            const int y = __ldg(key + b + j);
            r += (y < x) | ((y == x) & (j < k));
        }
        perm[r] = k;
    }
}

// ---------------------------------------------------------------- small sorts
__device__ __forceinline__ void key_cswap(int4& a, int4& b)
{
    const bool s = b.x < a.x;
    const int4 t = a;
    a.x = s ? b.x : a.x; a.y = s ? b.y : a.y; a.z = s ? b.z : a.z; a.w = s ? b.w : a.w;
    b.x = s ? t.x : b.x; b.y = s ? t.y : b.y; b.z = s ? t.z : b.z; b.w = s ? t.w : b.w;
}

__device__ __forceinline__ void key_cswap(int& a, int& b)
{
    const int lo = min(a, b);
    b = max(a, b);
    a = lo;
}
__device__ __forceinline__ void key_cswap(unsigned long long& a, unsigned long long& b)
{
    const unsigned long long lo = min(a, b);
    b = max(a, b);
    a = lo;
}
// sorting networks of 4 and 8 (Batcher's odd-even merge)
template <int NMAX, class T>
__device__ __forceinline__ void sort_keys(T (&r)[NMAX])
{
    key_cswap(r[0], r[1]); key_cswap(r[2], r[3]); key_cswap(r[0], r[2]); key_cswap(r[1], r[3]); key_cswap(r[1], r[2]);
    if constexpr (NMAX == 8) {
        key_cswap(r[4], r[5]); key_cswap(r[6], r[7]); key_cswap(r[4], r[6]); key_cswap(r[5], r[7]); key_cswap(r[5], r[6]);
        key_cswap(r[0], r[4]); key_cswap(r[1], r[5]); key_cswap(r[2], r[6]); key_cswap(r[3], r[7]);
        key_cswap(r[2], r[4]); key_cswap(r[3], r[5]);
        key_cswap(r[1], r[2]); key_cswap(r[3], r[4]); key_cswap(r[5], r[6]);
    }
}

// ---------------------------------------------------------------- status
// Device-side status written by kernels; the host reads it after a sync.
struct DevStatus {
    int err;          // first error code (slak_status), 0 = ok
    int detail;       // kernel-specific detail (e.g. offending index)
    int nextern;      // boundary half-edges of level 0
    int nedges;       // edges of level 0
    int bcount[32];   // boundary half-edges counted per level
    int vhist[17];    // level 0: vertices of valence 0..15, and 16 or more
};

__device__ __forceinline__ void set_error(DevStatus* st, int code, int detail)
{
    if (atomicCAS(&st->err, 0, code) == 0) st->detail = detail;
}

// ---------------------------------------------------------------- faces
// Corner navigation: QUAD uses the implicit 4-corner faces of the reference's
// quad functions (`threadId / 4 * 4 + (threadId + 1) % 4`,
// CatmullClarkKernels.cuh:155); otherwise face offsets + a corner->face map.
constexpr unsigned kNavFar = 0xffffffffu;
template <bool QUAD>
struct Faces {
    const int* __restrict__ ptr;
    const int* __restrict__ cface;
    const unsigned* __restrict__ nav = nullptr;     // corners before c in its face | after it << 16 (kNavFar: use ptr)
    __device__ __forceinline__ int face(int c) const { return QUAD ? (c >> 2) : __ldg(cface + c); }
    // next and previous corner, with `nav`: one load instead of the face's two offsets behind its id
    __device__ __forceinline__ void around(int c, int& nc, int& pc) const
    {
        const unsigned u = QUAD || nav == nullptr ? kNavFar : __ldg(nav + c);
        if (u != kNavFar) {
            const int before = (int)(u & 0xffffu), after = (int)(u >> 16);
            nc = after ? c + 1 : c - before;
            pc = before ? c - 1 : c + after;
        } else {
            nc = next(c);
            pc = prev(c);
        }
    }
    __device__ __forceinline__ int next(int c) const
    {
        if (QUAD) return (c & ~3) | ((c + 1) & 3);
        int f = __ldg(cface + c);
        return c + 1 < __ldg(ptr + f + 1) ? c + 1 : __ldg(ptr + f);
    }
    __device__ __forceinline__ int prev(int c) const
    {
        if (QUAD) return (c & ~3) | ((c + 3) & 3);
        int f = __ldg(cface + c);
        int b = __ldg(ptr + f);
        return c > b ? c - 1 : __ldg(ptr + f + 1) - 1;
    }
};

inline unsigned grid_for(int64_t n, int block = kBlock)
{
    int64_t g = (n + block - 1) / block;
    return (unsigned)(g < 1 ? 1 : g);
}

}  // namespace slak
