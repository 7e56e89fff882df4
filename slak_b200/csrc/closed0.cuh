// closed0.cuh -- level 0 of a closed mesh in four passes.
//
// general.cuh rebuilds an arbitrary mesh's adjacency in a dozen dependent
// launches.  When the mesh is closed (the plan's level-0 probe counted no
// boundary half-edge), every edge has two half-edges, so a vertex's number of
// owned edges is known from its corners alone (SLAK: the next vertex is larger;
// LAK: it is smaller), before any twin is looked up:
//
//   k_c0_faces   per face: corner -> face, face point, and per corner one 64-bit
//                atomic that counts the vertex's corners (low half) and owned
//                edges (high half) at once; CAP: the corner's record into its
//                vertex's bucket of 8, else its arrival rank
//   k_c0_sums, k_c0_offsets   both counts' offsets: columns (sptr), edge ids (eptr)
//   k_c0_bucket  (not CAP) the corners' records into their columns
//   k_c0_verts   per vertex: its column sorted by corner, twins, edge ids of its
//                owned edges, corner -> slot / twin, its vertex point
//   k_c0_long    (columns of more than 8 slots, where the probe saw any) edge ids
//                and vertex points
//   k_c0_quads   per corner: refined quad, t, and (owner) the edge's point
//
// CAP (no vertex above valence 8, the probe's histogram) saves the bucket pass.
// A record is {corner, next vertex (top bit: first corner of its face), previous
// vertex, face}: a column's whole adjacency without further gathers.  Numbering,
// float formulas and their order are general.cuh's.
//
// Why: these passes move little (about 100 MB at 1 M corners) and are bound by
// the latency of dependent launches and gathers, so fewer passes is what
// counts.  Measured on B200, launch by launch: 243,905 polygons (1 M corners)
// 163 -> 98 us, 400,000 triangles in scattered order (LAK) 250 -> 115 us; whole
// plans of one level: the scattered triangles 200 -> 107 us, 128x128 torus 28 -> 17
// us.  CAP needs 128 bytes per vertex, so it stays with valences up to 8; above
// that the compact records of the bucket pass serve every valence.  One level with
// CAP and, for the same meshes, without: 32x32 torus 12.8 and 14.9 us, 512x512
// torus 44.2 and 49.6, 512x512 mixed torus 63.9 and 65.9 (SLAK; LAK 67.4 and 68.2).
#pragma once

#include "general.cuh"
#include "scan.cuh"

namespace slak {

constexpr int kC0Cap = 8;
constexpr unsigned kFirst = 0x80000000u;

template <bool LAK>
__device__ __forceinline__ unsigned long long c0_count(int v, int w)
{
    return 1ull | ((unsigned long long)(LAK ? w < v : v < w) << 32);
}

// Corner c of face f (vertex v, next vertex w, previous u): its vertex's counts, its
// record (CAP) or arrival rank.
template <bool LAK, bool CAP>
__device__ __forceinline__ void c0_corner(int c, int f, int v, int w, int u, bool first, int V,
                                          unsigned long long* __restrict__ cnt, int* __restrict__ rank,
                                          int4* __restrict__ rec, DevStatus* st)
{
    if ((unsigned)v >= (unsigned)V) { set_error(st, 4, c); return; }
    if ((unsigned)w >= (unsigned)V) w = v;      // (that corner reports its id)
    if ((unsigned)u >= (unsigned)V) u = v;
    const int r = (int)(unsigned)atomicAdd(cnt + v, c0_count<LAK>(v, w));
    if (CAP) {
        if (r < kC0Cap) rec[(int64_t)v * kC0Cap + r] = make_int4(c, first ? (int)((unsigned)w | kFirst) : w, u, f);
        else set_error(st, 4, c);               // a larger valence than the plan was made for
    } else {
        rank[c] = r;
    }
}

// A face of n > kBigCol corners from b on by its warp: corners over the lanes,
// the sum of its positions in corner order, one component per lane.  One thread
// waits for each corner's atomic in turn (its result is the corner's place).
// Level 0 of a prism on B200, by its caps' corners: 17 25 -> 19 us, 33 33 -> 19,
// 64 46 -> 19, 256 153 -> 36, 1000 468 -> 109 (the general level 30, 32, 36, 68 and
// 188); 2,000 prisms of 24 40 -> 33.  16 corners in turn take 21 us.
template <bool LAK, bool CAP>
__device__ __forceinline__ void c0_long_face(const int* __restrict__ ids, int f, int b, int n, int V,
                                          const float* __restrict__ P, float* __restrict__ FP, int* __restrict__ cface,
                                          unsigned* __restrict__ nav, unsigned long long* __restrict__ cnt,
                                          int* __restrict__ rank, int4* __restrict__ rec, DevStatus* st)
{
    const int lane = threadIdx.x & 31, c4 = term_comp();
    for (int k = lane; k < n; k += 32) {
        const int c = b + k;
        const int v = __ldg(ids + c), w = __ldg(ids + (k + 1 < n ? c + 1 : b)), u = __ldg(ids + (k ? c - 1 : b + n - 1));
        cface[c] = f;
        if (nav != nullptr) nav[c] = n <= 0xffff ? (unsigned)k | ((unsigned)(n - 1 - k) << 16) : kNavFar;
        c0_corner<LAK, CAP>(c, f, v, w, u, k == 0, V, cnt, rank, rec, st);
    }
    float acc = 0.0f;
    for (int k0 = 0; k0 < n; k0 += 64) {
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = k0 + 8 * j + term_slot();
            x[j] = 0.0f;
            if (k < n) {
                const int v = __ldg(ids + b + k);
                x[j] = ldg1(P, (unsigned)v < (unsigned)V ? v : 0, c4);
            }
        }
        each_term(x, n - k0, [&](float t) { acc = __fadd_rn(acc, t); });
    }
    const float y = LAK ? __fadd_rn(div1(acc, (float)n), 0.0f) : __fmul_rn(acc, __fdiv_rn(1.0f, (float)n));
    if (lane < 4) FP[4 * (int64_t)f + lane] = y;
}

template <bool QUAD, bool LAK, bool CAP>
__device__ __forceinline__ void k_c0_faces_body(const unsigned bx_, const int* __restrict__ ptr,
                                                const int* __restrict__ ids, int F, int N, int V,
                                                const float* __restrict__ P, float* __restrict__ FP,
                                                int* __restrict__ cface, unsigned* __restrict__ nav,
                                                unsigned long long* __restrict__ cnt,
                                                int* __restrict__ rank, int4* __restrict__ rec, DevStatus* st)
{
    const int f = bx_ * kBlock + threadIdx.x;
    const auto pos = [&](int v) { return ldg4(P, (unsigned)v < (unsigned)V ? v : 0); };
    if constexpr (QUAD) {
        if (f >= F) return;
        const int4 q = __ldg(reinterpret_cast<const int4*>(ids) + f);
        const float4 a = pos(q.x), b = pos(q.y), c = pos(q.z), e = pos(q.w);
        c0_corner<LAK, CAP>(4 * f + 0, f, q.x, q.y, q.w, true, V, cnt, rank, rec, st);
        c0_corner<LAK, CAP>(4 * f + 1, f, q.y, q.z, q.x, false, V, cnt, rank, rec, st);
        c0_corner<LAK, CAP>(4 * f + 2, f, q.z, q.w, q.y, false, V, cnt, rank, rec, st);
        c0_corner<LAK, CAP>(4 * f + 3, f, q.w, q.x, q.z, false, V, cnt, rank, rec, st);
        if (!LAK) st4(FP, f, f4_mul(f4_add(f4_add(a, c), f4_add(b, e)), 0.25f));
        else st4(FP, f, f4_div_z(f4_add(f4_add(f4_add(f4_add(f4_zero(), a), b), c), e), 4.0f));
    } else {
        if (f == 0 && (ptr[0] != 0 || ptr[F] != N)) set_error(st, 4, -1);
        int b = 0, e = 0;
        if (f < F) { b = ptr[f]; e = ptr[f + 1]; }
        const int n = e - b;
        const bool ok = b >= 0 && e <= N && n >= 3;
        if (f < F && !ok) set_error(st, 4, f);
        float4 acc = f4_zero();
        if (ok && n <= 8) {                   // every id and position in flight at once
            int v[8];
            float4 p[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = k < n ? __ldg(ids + b + k) : 0;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < n) p[k] = pos(v[k]);
            int last = v[0];
#pragma unroll
            for (int k = 1; k < 8; ++k)
                if (k < n) last = v[k];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < n) {
                    const int w = k + 1 < n ? v[(k + 1) & 7] : v[0], u = k ? v[(k + 7) & 7] : last;
                    cface[b + k] = f;
                    if (nav != nullptr) nav[b + k] = (unsigned)k | ((unsigned)(n - 1 - k) << 16);
                    c0_corner<LAK, CAP>(b + k, f, v[k], w, u, k == 0, V, cnt, rank, rec, st);
                }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < n) acc = f4_add(acc, p[k]);
        } else if (ok && n <= kBigCol) {
            int u = __ldg(ids + e - 1), v = __ldg(ids + b);
            for (int c = b; c < e; ++c) {
                const int w = __ldg(ids + (c + 1 < e ? c + 1 : b));
                cface[c] = f;
                if (nav != nullptr) nav[c] = n <= 0xffff ? (unsigned)(c - b) | ((unsigned)(e - 1 - c) << 16) : kNavFar;
                c0_corner<LAK, CAP>(c, f, v, w, u, c == b, V, cnt, rank, rec, st);
                acc = f4_add(acc, pos(v));
                u = v;
                v = w;
            }
        }
        if (ok && n <= kBigCol) st4(FP, f, LAK ? f4_div_z(acc, (float)n) : f4_mul(acc, __fdiv_rn(1.0f, (float)n)));
        // a long face by its warp: one thread would wait for each corner's atomic in turn
        for_each_big<kBlock>(ok && n > kBigCol, false, [&](int i) {
            const int g = bx_ * kBlock + i, gb = ptr[g];
            c0_long_face<LAK, CAP>(ids, g, gb, ptr[g + 1] - gb, V, P, FP, cface, nav, cnt, rank, rec, st);
        });
    }
}
template <bool QUAD, bool LAK, bool CAP>
__global__ void __launch_bounds__(kBlock) k_c0_faces(const int* __restrict__ ptr, const int* __restrict__ ids, int F,
                                                     int N, int V, const float* __restrict__ P, float* __restrict__ FP,
                                                     int* __restrict__ cface, unsigned* __restrict__ nav,
                                                     unsigned long long* __restrict__ cnt,
                                                     int* __restrict__ rank, int4* __restrict__ rec, DevStatus* st)
{
    griddep_enter();
    k_c0_faces_body<QUAD, LAK, CAP>(blockIdx.x, ptr, ids, F, N, V, P, FP, cface, nav, cnt, rank, rec, st);
}
template <bool QUAD, bool LAK, bool CAP>
struct k_c0_faces_g {
    static constexpr int kBounds = 1, kMaxT = kBlock, kMinB = 0;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const
    {
        k_c0_faces_body<QUAD, LAK, CAP>(bx, a...);
    }
    static constexpr auto kernel() { return &k_c0_faces<QUAD, LAK, CAP>; }
};

// ------------------------------------------------------------------ the scan of both counts
using u64 = unsigned long long;

__device__ __forceinline__ u64 block_excl_scan2(u64 x, u64* total)
{
    __shared__ u64 warp_tot[kBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    u64 before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < kBlock / 32; ++k) {
        const u64 t = warp_tot[k];
        if (k < warp) before += t;
        all += t;
    }
    __syncthreads();
    *total = all;
    return before + incl - x;
}

__device__ __forceinline__ void k_c0_sums_body(const unsigned bx_, const u64* __restrict__ cnt, int n, u64* __restrict__ tsum)
{
    u64 s = 0, tot;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const int k = bx_ * kScanTile + i * kBlock + threadIdx.x;
        if (k < n) s += cnt[k];
    }
    block_excl_scan2(s, &tot);
    if (threadIdx.x == 0) tsum[bx_] = tot;
}
template <int = 0>
__global__ void __launch_bounds__(kBlock) k_c0_sums(const u64* __restrict__ cnt, int n, u64* __restrict__ tsum)
{
    griddep_enter();
    k_c0_sums_body(blockIdx.x, cnt, n, tsum);
}
struct k_c0_sums_g {
    static constexpr int kBounds = 1, kMaxT = kBlock, kMinB = 0;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const { k_c0_sums_body(bx, a...); }
    static constexpr auto kernel() { return &k_c0_sums<>; }
};

// Each block adds up the tiles before its own (DIRECT, up to kC0Direct tiles:
// from the counts themselves, one launch instead of two), then scans its tile.
// Block 0 also checks the totals against the plan's corners and edges.  One level
// of a torus, by its tiles, with and without the counts themselves: 2 tiles 14.8
// and 16.6 us, 4 16.9 and 16.7 (SLAK; with their state 18.1 and 16.8), 16 23.0 and
// 16.9.
constexpr int kC0Direct = 4;
template <bool DIRECT>
__device__ __forceinline__ void k_c0_offsets_body(const unsigned bx_, const u64* __restrict__ cnt, int n,
                                                  const u64* __restrict__ tsum, int nt, int* __restrict__ sptr,
                                                  int* __restrict__ eptr, int N, int E, DevStatus* st)
{
    __shared__ u64 tile[kScanTile];
    u64 before = 0, all = 0, carry, total;
    if (DIRECT) {
        for (int k = threadIdx.x; k < n; k += kBlock) {
            const u64 x = cnt[k];
            all += x;
            if (k < (int)bx_ * kScanTile) before += x;
        }
    } else {
        for (int k = threadIdx.x; k < nt; k += kBlock) {
            const u64 x = tsum[k];
            all += x;
            if (k < (int)bx_) before += x;
        }
    }
    block_excl_scan2(before, &carry);
    block_excl_scan2(all, &total);
    const int base = bx_ * kScanTile;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const int j = i * kBlock + threadIdx.x;
        tile[j] = base + j < n ? cnt[base + j] : 0;
    }
    __syncthreads();
    u64 loc[kScanItems], s = 0, tt;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) { loc[i] = s; s += tile[threadIdx.x * kScanItems + i]; }
    const u64 e = block_excl_scan2(s, &tt) + carry;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) tile[threadIdx.x * kScanItems + i] = e + loc[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const int j = i * kBlock + threadIdx.x;
        if (base + j < n) {
            const u64 x = tile[j];
            sptr[base + j] = (int)(unsigned)x;
            eptr[base + j] = (int)(x >> 32);
        }
    }
    if (bx_ == 0 && threadIdx.x == 0) {
        sptr[n] = (int)(unsigned)total;
        eptr[n] = (int)(total >> 32);
        if ((int)(unsigned)total != N || (int)(total >> 32) != E) set_error(st, 4, 1000);
    }
}
template <bool DIRECT>
__global__ void __launch_bounds__(kBlock) k_c0_offsets(const u64* __restrict__ cnt, int n, const u64* __restrict__ tsum,
                                                       int nt, int* __restrict__ sptr, int* __restrict__ eptr, int N,
                                                       int E, DevStatus* st)
{
    griddep_enter();
    k_c0_offsets_body<DIRECT>(blockIdx.x, cnt, n, tsum, nt, sptr, eptr, N, E, st);
}
template <bool DIRECT>
struct k_c0_offsets_g {
    static constexpr int kBounds = 1, kMaxT = kBlock, kMinB = 0;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const
    {
        k_c0_offsets_body<DIRECT>(bx, a...);
    }
    static constexpr auto kernel() { return &k_c0_offsets<DIRECT>; }
};

// ------------------------------------------------------------------ records into columns (valences above 8)
// face, next and previous corner of c
template <bool QUAD>
__device__ __forceinline__ void c0_nav(const Faces<QUAD>& fc, int c, int N, int F, int& f, int& nc, int& p)
{
    if constexpr (QUAD) {
        f = c >> 2; nc = fc.next(c); p = fc.prev(c);
    } else {
        f = __ldg(fc.cface + c);
        if ((unsigned)f >= (unsigned)F) f = 0;
        fc.around(c, nc, p);
        if ((unsigned)nc >= (unsigned)N) nc = c;
        if ((unsigned)p >= (unsigned)N) p = c;
    }
}

template <bool QUAD>
__device__ __forceinline__ void k_c0_bucket_body(const unsigned bx_, Faces<QUAD> fc, const int* __restrict__ ids, int N,
                                                 int F, int V, const int* __restrict__ sptr, const int* __restrict__ rank,
                                                 int4* __restrict__ rec)
{
    const int c = bx_ * kBlock + threadIdx.x;
    if (c >= N) return;
    const int v = __ldg(ids + c);
    if ((unsigned)v >= (unsigned)V) return;
    // (a plan's mesh keeps its topology; where the caller changed it all the same,
    // a corner of a face the first pass rejected has neither face nor rank of this
    // run, and overlapping faces count more than N corners: what is read and written
    // here stays in range)
    int f, nc, p;
    c0_nav<QUAD>(fc, c, N, F, f, nc, p);
    int w = __ldg(ids + nc), u = __ldg(ids + p);
    if ((unsigned)w >= (unsigned)V) w = v;
    if ((unsigned)u >= (unsigned)V) u = v;
    const int b = __ldg(sptr + v), r = __ldg(rank + c);
    if ((unsigned)r < (unsigned)(__ldg(sptr + v + 1) - b) && (unsigned)(b + r) < (unsigned)N)
        rec[b + r] = make_int4(c, p > c ? (int)((unsigned)w | kFirst) : w, u, f);
}
template <bool QUAD>
__global__ void __launch_bounds__(kBlock) k_c0_bucket(Faces<QUAD> fc, const int* __restrict__ ids, int N, int F, int V,
                                                      const int* __restrict__ sptr, const int* __restrict__ rank,
                                                      int4* __restrict__ rec)
{
    griddep_enter();
    k_c0_bucket_body<QUAD>(blockIdx.x, fc, ids, N, F, V, sptr, rank, rec);
}
template <bool QUAD>
struct k_c0_bucket_g {
    static constexpr int kBounds = 1, kMaxT = kBlock, kMinB = 0;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const
    {
        k_c0_bucket_body<QUAD>(bx, a...);
    }
    static constexpr auto kernel() { return &k_c0_bucket<QUAD>; }
};

// ------------------------------------------------------------------ vertices
// What a vertex pass writes: corner -> slot / twin / edge id; the slot-ordered
// column (sc, snext, sprev, sprevc) of long columns, and of all with creases.
struct C0Out {
    int *xslot, *xtw, *xnt, *eid;        // (xnt: next(twin), where another level follows a polygon mesh)
    int *sc, *snext, *sprev, *sprevc, *sflag;
    int all;                // every column's slots are wanted (creases)
};

template <bool QUAD>
__device__ __forceinline__ int rec_prev(const int* __restrict__ ptr, int4 r)
{
    if (QUAD) return (r.x & ~3) | ((r.x + 3) & 3);
    return r.y < 0 ? __ldg(ptr + r.w + 1) - 1 : r.x - 1;
}
// One vertex of n <= NMAX corners (records rec, unsorted) on its own thread.
template <bool QUAD, bool LAK, int NMAX>
__device__ __forceinline__ void c0_vertex(const int* __restrict__ ptr, const int4* __restrict__ rec, int v, int b,
                                          int n, int id0, int E, const C0Out& o, const float* __restrict__ P,
                                          const float* __restrict__ FP, float* __restrict__ R, int compensated,
                                          DevStatus* st)
{
    const float4 Pv = ldg4(P, v);
    int4 r[NMAX];
#pragma unroll
    for (int k = 0; k < NMAX; ++k) r[k] = k < n ? __ldg(rec + k) : make_int4(INT32_MAX, 0, 0, 0);
    sort_keys<NMAX>(r);
    int nx[NMAX], pc[NMAX], nb[NMAX];
    float4 pn[NMAX], pf[NMAX];              // face point of each slot; SLAK the next vertex of each slot,
#pragma unroll                              // LAK the previous vertices in ascending id
    for (int k = 0; k < NMAX; ++k) {
        nx[k] = r[k].y & 0x7fffffff;
        nb[k] = LAK ? (k < n ? r[k].z : INT32_MAX) : nx[k];
    }
    if constexpr (LAK) sort_keys<NMAX>(nb);
#pragma unroll
    for (int k = 0; k < NMAX; ++k)
        if (k < n) {
            pn[k] = ldg4(P, nb[k]);
            pf[k] = ldg4(FP, r[k].w);
            pc[k] = rec_prev<QUAD>(ptr, r[k]);
        }
    int bad = 0, own = 0;
#pragma unroll
    for (int k = 0; k < NMAX; ++k) {
        if (k >= n) continue;
        const int w = nx[k], c = r[k].x;
        int tw = -1, nt = c, less = 0;
#pragma unroll
        for (int t = 0; t < NMAX; ++t) {
            if (t >= n) continue;
            if (r[t].z == w) { if (tw < 0) { tw = pc[t]; nt = r[t].x; } else bad = 1; }
            if (t < k && nx[t] == w) bad = 1;
            less += nx[t] < w;
        }
        if (w == v || r[k].z == v || tw < 0) bad = 1;
        const int twc = tw < 0 ? c : tw;
        o.xslot[c] = b + k;
        o.xtw[c] = twc;
        if (!QUAD && o.xnt != nullptr) o.xnt[c] = nt;
        if (LAK ? w < v : v < w) {
            int id = id0 + (LAK ? less : own);
            if ((unsigned)id >= (unsigned)E) { bad = 1; id = 0; }
            o.eid[c] = id;
            o.eid[twc] = id;
            ++own;
        }
        if (o.all) {
            o.sc[b + k] = c;
            o.snext[b + k] = w;
            o.sprev[b + k] = r[k].z;
            o.sprevc[b + k] = pc[k];
            o.sflag[b + k] = 0;
        }
    }
    if (bad) set_error(st, 4, v);
    const float nn = (float)(n * n);
    float4 y;
    const bool comp = compensated && n > 4;
    if (!LAK) {
        if (!comp) {
            float4 acc = f4_zero();
#pragma unroll
            for (int k = 0; k < NMAX; ++k)
                if (k < n) acc = f4_add(acc, pn[k]);
            y = f4_add(f4_div(acc, nn), f4_div(f4_mul(Pv, (float)(n - 2)), (float)n));
#pragma unroll
            for (int k = 0; k < NMAX; ++k)
                if (k < n) y = f4_add(y, f4_div(pf[k], nn));
        } else {
            float4 sh = f4_zero(), sl = f4_zero();
#pragma unroll
            for (int k = 0; k < NMAX; ++k)
                if (k < n) dd_acc(sh, sl, pn[k]);
#pragma unroll
            for (int k = 0; k < NMAX; ++k)
                if (k < n) dd_acc(sh, sl, pf[k]);
            y = vp_finish(sh, sl, Pv, n);
        }
    } else {
        float4 acc = f4_zero(), sh = f4_zero(), sl = f4_zero();
#pragma unroll
        for (int k = 0; k < NMAX; ++k)
            if (k < n) { if (comp) dd_acc(sh, sl, pf[k]); else acc = f4_add(acc, pf[k]); }
#pragma unroll
        for (int k = 0; k < NMAX; ++k)
            if (k < n) { if (comp) dd_acc(sh, sl, pn[k]); else acc = f4_add(acc, pn[k]); }
        if (comp) y = vp_finish(sh, sl, Pv, n);
        else y = f4_div_z(f4_add(f4_div_z(acc, (float)n), f4_mul(Pv, __fadd_rn((float)n, -2.0f))), (float)n);
    }
    st4(R, v, y);
}

template <bool QUAD, bool LAK, bool CAP>
__device__ __forceinline__ void k_c0_verts_body(const unsigned bx_, const int* __restrict__ ptr, int V, int E,
                                                const int* __restrict__ sptr, const int* __restrict__ eptr,
                                                const int4* __restrict__ rec, C0Out o, const float* __restrict__ P,
                                                const float* __restrict__ FP, float* __restrict__ R, int compensated,
                                                DevStatus* st)
{
    const int v = bx_ * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int b = 0, n = 0, id0 = 0;
    if (v < V) { b = __ldg(sptr + v); n = __ldg(sptr + v + 1) - b; id0 = __ldg(eptr + v); }
    const int4* rv = rec + (CAP ? (int64_t)v * kC0Cap : (int64_t)b);
    // one path per warp: its lanes wait for the same loads once
    const bool wide = __any_sync(0xffffffffu, v < V && n > 4);
    if (v < V && n <= 8) {
        if (!wide) c0_vertex<QUAD, LAK, 4>(ptr, rv, v, b, n, id0, E, o, P, FP, R, compensated, st);
        else c0_vertex<QUAD, LAK, 8>(ptr, rv, v, b, n, id0, E, o, P, FP, R, compensated, st);
    }
    if constexpr (!CAP) {
        // longer columns by their warp: slots by rank, twins by search; k_c0_long does the rest
        for_each_big<128>(v < V && n > 8, true, [&](int i) {
            const int bv = bx_ * blockDim.x + i, bb = __ldg(sptr + bv), bn = __ldg(sptr + bv + 1) - bb;
            int bad = 0;
            for (int k = lane; k < bn; k += 32) {
                const int4 me = __ldg(rec + bb + k);
                const int w = me.y & 0x7fffffff;
                int4 hit = make_int4(-1, 0, 0, 0);       // the record entered from w
                int rk = 0;
#pragma unroll 8
                for (int t = 0; t < bn; ++t) {
                    const int4 x = __ldg(rec + bb + t);
                    rk += x.x < me.x;
                    if (x.z == w) {
                        if (hit.x < 0) hit = x;
                        else bad = 1;
                    }
                    if (t < k && (x.y & 0x7fffffff) == w) bad = 1;
                }
                const int tw = hit.x < 0 ? -1 : rec_prev<QUAD>(ptr, hit);
                if (w == bv || me.z == bv || tw < 0) bad = 1;
                const int s = bb + rk;
                o.xslot[me.x] = s;
                o.xtw[me.x] = tw < 0 ? me.x : tw;
                if (!QUAD && o.xnt != nullptr) o.xnt[me.x] = hit.x < 0 ? me.x : hit.x;
                o.sc[s] = me.x;
                o.snext[s] = w;
                o.sprev[s] = me.z;
                o.sprevc[s] = rec_prev<QUAD>(ptr, me);
                o.sflag[s] = 0;
            }
            if (bad) set_error(st, 4, bv);
        });
    }
}
template <bool QUAD, bool LAK, bool CAP>
__global__ void __launch_bounds__(128) k_c0_verts(const int* __restrict__ ptr, int V, int E,
                                                  const int* __restrict__ sptr, const int* __restrict__ eptr,
                                                  const int4* __restrict__ rec, C0Out o, const float* __restrict__ P,
                                                  const float* __restrict__ FP, float* __restrict__ R, int compensated,
                                                  DevStatus* st)
{
    griddep_enter();
    k_c0_verts_body<QUAD, LAK, CAP>(blockIdx.x, ptr, V, E, sptr, eptr, rec, o, P, FP, R, compensated, st);
}
template <bool QUAD, bool LAK, bool CAP>
struct k_c0_verts_g {
    static constexpr int kBounds = 1, kMaxT = 128, kMinB = 0;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const
    {
        k_c0_verts_body<QUAD, LAK, CAP>(bx, a...);
    }
    static constexpr auto kernel() { return &k_c0_verts<QUAD, LAK, CAP>; }
};

// Columns of more than 8 slots, from the slot-ordered arrays k_c0_verts wrote:
// edge ids of the owned edges and the vertex point, a warp per column (LAK ids
// and vertex points of columns above kWarpCol: one thread, as in general.cuh).
template <bool QUAD, bool LAK>
__device__ __forceinline__ void k_c0_long_body(const unsigned bx_, Faces<QUAD> fc, int V, int E,
                                               const int* __restrict__ sptr, const int* __restrict__ eptr,
                                               const int* __restrict__ sc, const int* __restrict__ snext,
                                               const int* __restrict__ sprev, const int* __restrict__ sprevc,
                                               const int* __restrict__ xtw, int* __restrict__ eid,
                                               const float* __restrict__ P, const float* __restrict__ FP,
                                               float* __restrict__ R, int compensated, DevStatus* st)
{
    const int v = bx_ * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int b = 0, n = 0;
    if (v < V) { b = __ldg(sptr + v); n = __ldg(sptr + v + 1) - b; }
    for_each_big<kBlock>(v < V && n > 8, true, [&](int i) {
        const int bv = bx_ * blockDim.x + i, bb = __ldg(sptr + bv), bn = __ldg(sptr + bv + 1) - bb;
        const int bid = __ldg(eptr + bv);
        int before = 0, bad = 0;
        for (int k0 = 0; k0 < bn; k0 += 32) {
            const int k = k0 + lane;
            const int w = k < bn ? __ldg(snext + bb + k) : bv;
            const bool own = k < bn && (LAK ? w < bv : bv < w);
            int rk;
            if (LAK) {
                rk = 0;
                if (own) {
#pragma unroll 8
                    for (int t = 0; t < bn; ++t) rk += __ldg(snext + bb + t) < w;
                }
            } else {
                const unsigned g = __ballot_sync(0xffffffffu, own);
                rk = before + __popc(g & ((1u << lane) - 1));
                before += __popc(g);
            }
            if (own) {
                int id = bid + rk;
                if ((unsigned)id >= (unsigned)E) { bad = 1; id = 0; }
                const int c = __ldg(sc + bb + k);
                eid[c] = id;
                eid[__ldg(xtw + c)] = id;
            }
        }
        if (bad) set_error(st, 4, bv);
        if (bn > kBigCol && bn <= kWarpCol) {
            if constexpr (LAK)
                vp_lak_warp<QUAD>(fc, sc, snext, sprev, sprevc, nullptr, eid, 0, P, FP, R, compensated, bv, bb, bn);
            else
                vp_slak_warp<QUAD>(fc, sc, snext, sprev, nullptr, 0, P, FP, R, compensated, bv, bb, bn);
        }
    });
    if (v < V && n > 8 && (n <= kBigCol || n > kWarpCol)) {
        if constexpr (LAK)
            vp_lak_vertex<QUAD>(fc, sc, snext, sprev, sprevc, nullptr, eid, 0, P, FP, R, compensated, v, b, n);
        else
            vp_slak_vertex<QUAD>(fc, sc, snext, sprev, nullptr, 0, P, FP, R, compensated, v, b, n);
    }
}
template <bool QUAD, bool LAK>
__global__ void __launch_bounds__(kBlock) k_c0_long(Faces<QUAD> fc, int V, int E, const int* __restrict__ sptr,
                                                    const int* __restrict__ eptr, const int* __restrict__ sc,
                                                    const int* __restrict__ snext, const int* __restrict__ sprev,
                                                    const int* __restrict__ sprevc, const int* __restrict__ xtw,
                                                    int* __restrict__ eid, const float* __restrict__ P,
                                                    const float* __restrict__ FP, float* __restrict__ R,
                                                    int compensated, DevStatus* st)
{
    griddep_enter();
    k_c0_long_body<QUAD, LAK>(blockIdx.x, fc, V, E, sptr, eptr, sc, snext, sprev, sprevc, xtw, eid, P, FP, R,
                              compensated, st);
}
template <bool QUAD, bool LAK>
struct k_c0_long_g {
    static constexpr int kBounds = 1, kMaxT = kBlock, kMinB = 0;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const
    {
        k_c0_long_body<QUAD, LAK>(bx, a...);
    }
    static constexpr auto kernel() { return &k_c0_long<QUAD, LAK>; }
};

// ------------------------------------------------------------------ refined quads, t and edge points
// Thread c: refined quad of corner c, t[c] = slot[twin(prev c)] (`xt`), and, on
// the min -> max half-edge, the edge point of its edge.
template <bool QUAD, bool LAK>
__device__ __forceinline__ void k_c0_quads_body(const unsigned bx_, Faces<QUAD> fc, const int* __restrict__ ids,
                                                const int* __restrict__ eid, const int* __restrict__ xslot,
                                                const int* __restrict__ xtw, int* __restrict__ xt, int N, int V, int F,
                                                int E, int4* __restrict__ out_ids, int* __restrict__ out_ptr,
                                                int4* __restrict__ out_vals, const float* __restrict__ P,
                                                const float* __restrict__ FP, float* __restrict__ EP)
{
    const int c = bx_ * kBlock + threadIdx.x;
    if (c >= N) return;
    int f, nc, p;
    c0_nav<QUAD>(fc, c, N, F, f, nc, p);
    const int v = __ldg(ids + c), w = __ldg(ids + nc);
    const int VF = V + F;
    const auto edge = [&](int x) { const int e = __ldg(eid + x); return (unsigned)e < (unsigned)E ? e : 0; };
    const auto twin = [&](int x) { const int t = __ldg(xtw + x); return (unsigned)t < (unsigned)N ? t : x; };
    const auto face = [&](int x) { const int g = fc.face(x); return (unsigned)g < (unsigned)F ? g : 0; };
    const int e0 = edge(c);
    __stcs(out_ids + c, make_int4(v, VF + e0, V + f, VF + edge(p)));
    if (xt) xt[c] = __ldg(xslot + twin(p));
    if (v < w && v >= 0 && w < V) {
        const float4 a = ldg4(P, v), b = ldg4(P, w), fa = ldg4(FP, f), fb = ldg4(FP, face(twin(c)));
        float4 r;
        if (!LAK)
            r = f4_add(f4_add(f4_zero(), f4_mul(f4_add(a, fa), 0.25f)), f4_mul(f4_add(b, fb), 0.25f));
        else
            r = f4_mul(f4_add(f4_add(f4_add(a, b), fa), fb), 0.25f);
        st4(EP, e0, r);
    }
    if (LAK && out_vals != nullptr) {          // only the final level stores ptr / vals
        __stcs(out_vals + c, make_int4(1, 2, 3, 4));
        out_ptr[c] = 4 * c;
        if (c == N - 1) out_ptr[N] = 4 * N;
    }
}
template <bool QUAD, bool LAK>
__global__ void __launch_bounds__(kBlock) k_c0_quads(Faces<QUAD> fc, const int* __restrict__ ids,
                                                     const int* __restrict__ eid, const int* __restrict__ xslot,
                                                     const int* __restrict__ xtw, int* __restrict__ xt, int N, int V,
                                                     int F, int E, int4* __restrict__ out_ids,
                                                     int* __restrict__ out_ptr, int4* __restrict__ out_vals,
                                                     const float* __restrict__ P, const float* __restrict__ FP,
                                                     float* __restrict__ EP)
{
    griddep_enter();
    k_c0_quads_body<QUAD, LAK>(blockIdx.x, fc, ids, eid, xslot, xtw, xt, N, V, F, E, out_ids, out_ptr, out_vals, P, FP,
                               EP);
}
template <bool QUAD, bool LAK>
struct k_c0_quads_g {
    static constexpr int kBounds = 1, kMaxT = kBlock, kMinB = 0;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const
    {
        k_c0_quads_body<QUAD, LAK>(bx, a...);
    }
    static constexpr auto kernel() { return &k_c0_quads<QUAD, LAK>; }
};

}  // namespace slak
