// grand.cuh -- closed-form refinement from the grandparent's adjacency state.
//
// C is the level being refined, P its parent and PP its grandparent: C =
// refine(P), P = refine(PP), PP a closed mesh (N2 corners, V2 vertices, F2
// faces, E2 edges).  P face y is PP corner y, and P corner x = 4y + k is
// corner k of the P quad {v, eo, f, ei} of y: PP's vertex v, the edge points
// eo / ei of PP's edges through y / prev(y), the face point f.  C quad 4y + k is
// then
//   k = 0  {v,  a, g, d}      a = edge point of v -eo    d = edge point of ei-v
//   k = 1  {eo, b, g, a}      b = edge point of eo-f     g = P's face point of y
//   k = 2  {f,  c, g, b}      c = edge point of f -ei
//   k = 3  {ei, d, g, c}
// so one thread holds the nine C vertices of its P face and refines its four
// quads from them.  C's ids, P's edge ids and P's columns all follow from P's
// quad y (16 bytes) and PP's twin, slot and t of y:
//   - C's own id array is not read (the level before it need not write it when
//     C is the last level refined);
//   - P's vertex columns at PP's face and edge points lie in the thread's face
//     and its neighbours across one edge, so they are summed here: only PP's
//     old vertices (a quarter of the columns) leave slot records for k_g3.
// The far side of PP's edge through y (twin corner tw, nh2 = next(tw)): P's
// faces tw and nh2, whose face points, the edge point X of the P edge eo-f(tw)
// between them and the edge point W of v -next(nh2) are gathered.
//
// Each P edge is worked by the thread of its lower id's half-edge: k = 0 (v <
// eo: the edge v-eo) and k = 2 (f < ei: the edge f-ei) always, k = 1 and 3
// never.  Numbering, float formulas and their order are fast.cuh's.
//
// Bound by HBM: the level's compulsory bytes are nearly all it moves (18 bytes
// of records per C quad at the old vertices' quarter, against 72 for every
// column).  One thread per P face has eleven gathers in flight at 126-128
// registers, 16 warps per SM; one thread per C quad (k_g1, 64 registers, 32
// warps with three or four each, and warp shuffles for what a thread here
// holds) was bound by load latency.  Measured on B200, last level of the
// 512x512 mixed torus: SLAK k_g1 + k_g3 590 + 166 us -> k_pp + k_g3 402 + 52 us
// (5.7 TB/s of algorithmic bytes, 88% of copy bandwidth), LAK 752 + 125 ->
// 634 + 50 us; this step alone took the whole call from 1.150 to 0.780 ms (SLAK)
// and 1.261 to 1.065 ms (LAK).  A cap of 96 registers (20 warps) spills 48-116
// bytes: 402 -> 472 us, LAK 634 -> 716 us.
#pragma once

#include "fast.cuh"

namespace slak {

__device__ __forceinline__ float4 quad_fp(bool lak, float4 c0, float4 c1, float4 c2, float4 c3)
{
    if (!lak) return f4_mul(f4_add(f4_add(c0, c2), f4_add(c1, c3)), 0.25f);
    return f4_div_z(f4_add(f4_add(f4_add(f4_add(f4_zero(), c0), c1), c2), c3), 4.0f);
}

// R[i..i+3] (64 contiguous bytes, 16-byte aligned): 256-bit stores where a pair
// is 32-byte aligned, which depends on i's parity alone
__device__ __forceinline__ void st8f(float* p, float4 a, float4 b)
{
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "l"(p), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}
__device__ __forceinline__ void st_pos4(float* R, int64_t i, float4 a, float4 b, float4 c, float4 e)
{
    float* p = R + 4 * i;
    if ((i & 1) == 0) {
        st8f(p, a, b);
        st8f(p + 8, c, e);
    } else {
        st4(R, i, a);
        st8f(p + 4, b, c);
        st4(R, i + 3, e);
    }
}

// The vertex point of P's edge point with position Pe from its column's two
// quads on the thread's own side (o0, o1) and on the far side (t0, t1), each
// pair in corner order; own_first: the own side's corners come first.  nb: the
// neighbour (SLAK e_out), fq: the face point.
__device__ __forceinline__ float4 vp4_slak(bool own_first, float4 Pe, float4 nbo0, float4 nbo1, float4 nbt0,
                                           float4 nbt1, float4 fo0, float4 fo1, float4 ft0, float4 ft1)
{
    const float4 n0 = own_first ? nbo0 : nbt0, n1 = own_first ? nbo1 : nbt1;
    const float4 n2 = own_first ? nbt0 : nbo0, n3 = own_first ? nbt1 : nbo1;
    const float4 g0 = own_first ? fo0 : ft0, g1 = own_first ? fo1 : ft1;
    const float4 g2 = own_first ? ft0 : fo0, g3 = own_first ? ft1 : fo1;
    const float4 acc = f4_add(f4_add(f4_add(f4_add(f4_zero(), n0), n1), n2), n3);
    float4 y = f4_add(f4_div(acc, 16.0f), f4_div(f4_mul(Pe, 2.0f), 4.0f));
    y = f4_add(y, f4_div(g0, 16.0f));
    y = f4_add(y, f4_div(g1, 16.0f));
    y = f4_add(y, f4_div(g2, 16.0f));
    return f4_add(y, f4_div(g3, 16.0f));
}
// LAK: face points in corner order, then the tails t0..t3 (already ascending)
__device__ __forceinline__ float4 vp4_lak(bool own_first, float4 Pe, float4 fo0, float4 fo1, float4 ft0, float4 ft1,
                                          float4 t0, float4 t1, float4 t2, float4 t3)
{
    float4 acc = f4_add(f4_zero(), own_first ? fo0 : ft0);
    acc = f4_add(acc, own_first ? fo1 : ft1);
    acc = f4_add(acc, own_first ? ft0 : fo0);
    acc = f4_add(acc, own_first ? ft1 : fo1);
    acc = f4_add(f4_add(f4_add(f4_add(acc, t0), t1), t2), t3);
    return f4_div_z(f4_add(f4_div_z(acc, 4.0f), f4_mul(Pe, 2.0f)), 4.0f);
}

__device__ __forceinline__ float4 ep_slak(float4 pa, float4 fa, float4 pb, float4 fb)
{
    return f4_add(f4_add(f4_zero(), f4_mul(f4_add(pa, fa), 0.25f)), f4_mul(f4_add(pb, fb), 0.25f));
}
__device__ __forceinline__ float4 ep_lak(float4 a, float4 e, float4 f0, float4 f1)
{
    return f4_mul(f4_add(f4_add(f4_add(a, e), f0), f1), 0.25f);
}

// The vertex point of PP's face point f (position Pf) of a polygon face with
// corners fb..fe-1, at most kPpFace of them: its column is the corners 4j + 2,
// ascending, each C quad {f, c(j), g(j), c(next j)}.  Formulas and order of
// g3_vertex.  Longer faces leave records for k_g3.  3 levels, B200, with the line
// at 4, 8 and 16 corners: faces of 9 (5,000 prisms) SLAK 105, 105, 109 us, LAK 125,
// 125, 137; of 12 (4,000) 112, 112, 120 and 137, 137, 154; of 6 (6,000) 82, 83, 84
// and 89, 94, 94; of 8 (5,000) 90, 88, 88 and 102, 113, 113; 512x512 mixed torus 321,
// 321, 320 and 368, 382, 383.  (SLAK is indifferent below 8; LAK, whose tails are
// selected one by one here, is better off with 4.)
constexpr int kPpFace = 8;
template <bool LAK>
__device__ __forceinline__ float4 pp_face_vertex(const FastDims& d, const int4* __restrict__ pids,
                                                 const float* __restrict__ P, const QState& pp, int fb, int fe,
                                                 float4 Pf, int compensated)
{
    const int k = fe - fb, VF1 = d.V1 + d.F1;
    const float nn = (float)(k * k);
    // C's vertex on the P edge f-eo(j), and its id
    const auto bid = [&](int j) {
        if (!LAK) return VF1 + d.N2 + (j + 1 == fe ? fb : j + 1);
        return VF1 + 4 * (__ldg(&pids[j].y) - d.V2 - d.F2) + 2 + (j > __ldg(pp.tw + j));
    };
    const bool comp = compensated && k > 4;
    float4 acc = f4_zero(), sh = f4_zero(), sl = f4_zero(), yv = f4_zero();
    const auto add = [&](float4 x) { if (comp) dd_acc(sh, sl, x); else acc = f4_add(acc, x); };
    if (!LAK) {
        for_each_loaded(k, [&](int j) { return ldg4(P, VF1 + d.N2 + fb + j); }, [&](int, float4 x) { add(x); });
        yv = f4_add(f4_div(acc, nn), f4_div(f4_mul(Pf, (float)(k - 2)), (float)k));
    }
    float4 cj = ldg4(P, bid(fe - 1));
    for (int j = fb; j < fe; ++j) {
        const float4 bj = ldg4(P, bid(j));
        const float4 q2 = quad_fp(LAK, Pf, cj, ldg4(P, d.V1 + j), bj);
        if (LAK || comp) add(q2);
        else yv = f4_add(yv, f4_div(q2, nn));
        cj = bj;
    }
    if (LAK) {                                  // tails b(j) in ascending id
        for (int last = -1;;) {
            int xm = INT32_MAX;
            for (int j = fb; j < fe; ++j) {
                const int x = bid(j);
                if (x > last && x < xm) xm = x;
            }
            if (xm == INT32_MAX) break;
            add(ldg4(P, xm));
            last = xm;
        }
        yv = f4_div_z(f4_add(f4_div_z(acc, (float)k), f4_mul(Pf, __fadd_rn((float)k, -2.0f))), (float)k);
    }
    return comp ? vp_finish(sh, sl, Pf, k) : yv;
}

// One thread per PP corner y.  PQ: PP's faces are quads (four consecutive lanes
// exchange by shuffles); else polygons (offsets and corner -> face map `pf`;
// what the neighbouring corners hold is loaded and recomputed).
// `wids`: write the refined quads (a level whose successor takes them from its
// grandparent's needs none).
template <bool LAK, bool STATE, bool PQ, int BS>
__device__ __forceinline__ void k_pp_body(const unsigned bx_, FastDims d, Faces<PQ> pf, const int4* __restrict__ pids,
                                          const float* __restrict__ P, QState pp, QState c, int wids,
                                          const CUtensorMap& otm, float* __restrict__ R, SlotScratch z,
                                          int* __restrict__ optr, int4* __restrict__ ovals, int compensated)
{
    const unsigned full = 0xffffffffu;
    const int y0 = bx_ * BS, t = threadIdx.x;
    const bool valid = y0 + t < d.N2;
    const int y = valid ? y0 + t : (PQ ? (y0 + t) & 3 : 0);      // idle lanes repeat an early corner's loads
    const int lane = t & 31;
    const int ln = (lane & ~3) | ((lane + 1) & 3), lp = (lane & ~3) | ((lane + 3) & 3);
    const int VF1 = d.V1 + d.F1, VFc = d.V + d.N1, VF2 = d.V2 + d.F2;

    // ---- P's quad, PP's state, the corner's neighbours
    const int4 q = __ldg(pids + y);
    const int tw = __ldg(pp.tw + y);
    const int s2 = __ldg(pp.slot + y);
    const int t2 = LAK ? 0 : __ldg(pp.t + y);
    int ny, py, twp, vn, vp = 0, fb = 0, fe = 0, nh2;
    int4 qp;                                                // P's quad of prev(y) (polygon PP)
    if constexpr (PQ) {
        ny = qnext(y); py = qprev(y);
        nh2 = qnext(tw);
        twp = __shfl_sync(full, tw, lp);
        vn = __shfl_sync(full, q.x, ln);
        if (LAK) vp = __shfl_sync(full, q.x, lp);
    } else {
        const unsigned u = __ldg(pf.nav + y);
        if (u != kNavFar) { fb = y - (int)(u & 0xffffu); fe = y + 1 + (int)(u >> 16); }
        else { fb = __ldg(pf.ptr + q.z - d.V2); fe = __ldg(pf.ptr + q.z - d.V2 + 1); }
        ny = y + 1 == fe ? fb : y + 1;
        py = y == fb ? fe - 1 : y - 1;
        twp = __ldg(pp.tw + py);
        vn = __ldg(&pids[ny].x);
        qp = __ldg(pids + py);
        vp = qp.x;
        nh2 = __ldg(pp.nt + y);
    }
    const int ee = q.y - VF2, ep = q.w - VF2;              // PP's edges through y and prev(y)
    // P's edges of the P face: v-eo, eo-f, f-ei, ei-v
    int E0, E1, E2, E3;
    if (!LAK) {
        E0 = s2; E1 = d.N2 + ny; E2 = d.N2 + y; E3 = t2;
    } else {
        E0 = 4 * ee + (q.x > vn); E1 = 4 * ee + 2 + (y > tw);
        E2 = 4 * ep + 2 + (y > twp); E3 = 4 * ep + (q.x > vp);
    }
    // the P edges eo-f(tw) (X) and v-next(nh2) (W) across PP's edge
    const int EX = LAK ? 4 * ee + 2 + (tw > y) : d.N2 + nh2;
    int EW;
    if (!LAK) {
        EW = __ldg(pp.slot + nh2);
    } else {
        int vnn;
        if constexpr (PQ) vnn = __ldg(&pids[qnext(nh2)].x);
        else {
            int nn2, pn2;
            pf.around(nh2, nn2, pn2);
            vnn = __ldg(&pids[nn2].x);
        }
        EW = 4 * (__ldg(&pids[nh2].y) - VF2) + (q.x > vnn);
    }
    const bool own = valid && q.x < vn;                     // sums PP's edge point eo's column

    // ---- positions
    const float4 Pv = ldg4(P, q.x), Pe = ldg4(P, q.y), Pf = ldg4(P, q.z), Pg = ldg4(P, d.V1 + y);
    const float4 Pa = ldg4(P, VF1 + E0), Pc = ldg4(P, VF1 + E2), Pd = ldg4(P, VF1 + E3);
    const float4 Gn = ldg4(P, d.V1 + nh2), PX = ldg4(P, VF1 + EX), PW = ldg4(P, VF1 + EW);
    float4 Gt = f4_zero();
    if (own) Gt = ldg4(P, d.V1 + tw);
    float4 Pi, Pb;
    if constexpr (PQ) { Pi = shfl4(Pe, lp); Pb = shfl4(Pc, ln); }
    else { Pi = ldg4(P, q.w); Pb = ldg4(P, VF1 + E1); }

    // ---- C's edges of the four quads' corners (e_out): k = 0: E of (v, a) etc.
    // e[k][0..3] as fast.cuh's e0..e3 of C quad 4y + k
    {
        int e00, e01, e02, e03, e10, e11, e12, e13, e20, e21, e22, e23, e30, e31, e32, e33;
        if (!LAK) {
            // columns of PP's edge points in P: 2 N2 + 4e + rank among {own pair, far pair}
            const int oe = y < tw ? 0 : 2, op = y < twp ? 0 : 2;
            const int be = 2 * d.N2 + 4 * ee, bp = 2 * d.N2 + 4 * ep;
            const int x4 = 4 * y;
            e00 = s2;                    e01 = d.N1 + x4 + 1; e02 = d.N1 + x4;     e03 = t2;
            e10 = be + oe + (ny < y);    e11 = d.N1 + x4 + 2; e12 = d.N1 + x4 + 1; e13 = be + (2 - oe) + (nh2 > tw);
            e20 = d.N2 + y;              e21 = d.N1 + x4 + 3; e22 = d.N1 + x4 + 2; e23 = d.N2 + ny;
            e30 = bp + op + (py < y);    e31 = d.N1 + x4;     e32 = d.N1 + x4 + 3; e33 = bp + op + (py > y);
        } else {
            e00 = 4 * E0;     e01 = 4 * E0 + 2 + (y > nh2); e02 = 4 * E3 + 2 + (y > twp); e03 = 4 * E3;
            e10 = 4 * E1 + 1; e11 = 4 * E1 + 2 + (y > ny);  e12 = e01;                    e13 = 4 * E0 + 1;
            e20 = 4 * E2;     e21 = 4 * E2 + 2 + (y > py);  e22 = e11;                    e23 = 4 * E1;
            e30 = 4 * E3 + 1; e31 = e02;                    e32 = e21;                    e33 = 4 * E2 + 1;
        }
        // refined quads {corner k', V + F + e_k', face point, V + F + e_(k'-1)}: the
        // thread's 256 bytes as two 128-byte halves, staged in the tensor map's
        // 128-byte swizzle (16-byte chunk j of row t at j ^ (t mod 8): free of
        // bank conflicts), one TMA tensor store per half; rows past N2 are clipped
        __shared__ __align__(1024) int4 sq[2 * 8 * BS];
        const int sw = t & 7, fp0 = d.V + 4 * y;
        const int ai = VF1 + E0, bi = VF1 + E1, ci = VF1 + E2, di = VF1 + E3, gi = d.V1 + y;
        int4* h0 = sq + 8 * t;
        int4* h1 = sq + 8 * BS + 8 * t;
        const auto put = [&](int4* h, int j, int c0, int c1, int c2, int c3, int e0, int e1, int e2, int e3, int fp) {
            h[(j + 0) ^ sw] = make_int4(c0, VFc + e0, fp, VFc + e3);
            h[(j + 1) ^ sw] = make_int4(c1, VFc + e1, fp, VFc + e0);
            h[(j + 2) ^ sw] = make_int4(c2, VFc + e2, fp, VFc + e1);
            h[(j + 3) ^ sw] = make_int4(c3, VFc + e3, fp, VFc + e2);
        };
        if (wids) {
        put(h0, 0, q.x, ai, gi, di, e00, e01, e02, e03, fp0);
        put(h0, 4, q.y, bi, gi, ai, e10, e11, e12, e13, fp0 + 1);
        put(h1, 0, q.z, ci, gi, bi, e20, e21, e22, e23, fp0 + 2);
        put(h1, 4, q.w, di, gi, ci, e30, e31, e32, e33, fp0 + 3);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (t < 2) {
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
                         :: "l"(reinterpret_cast<uint64_t>(&otm)), "r"(0), "r"(t), "r"(y0),
                            "r"((uint32_t)__cvta_generic_to_shared(sq + 8 * BS * t))
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        }
        if (STATE && valid) {
            // C's state for its corners 4x + k, x = 4y + k (write_state's formulas on P's
            // twin, slot and t, which are e_k0 and e_k3 for SLAK)
            const int x4 = 4 * y;
            const int twx[4] = {4 * nh2 + 3, 4 * ny + 2, 4 * py + 1, 4 * twp};
            int sl[4], tt[4];
            if (!LAK) {
                sl[0] = e00; sl[1] = e10; sl[2] = e20; sl[3] = e30;
                tt[0] = e03; tt[1] = e13; tt[2] = e23; tt[3] = e33;
            } else {
                const int oe = y < tw ? 0 : 2, op = y < twp ? 0 : 2;
                sl[0] = s2;
                sl[1] = 2 * d.N2 + 4 * ee + oe + (ny < y);
                sl[2] = d.N2 + y;
                sl[3] = 2 * d.N2 + 4 * ep + op + (py < y);
                tt[0] = tt[1] = tt[2] = tt[3] = 0;
            }
            const int eP[4] = {E0, E1, E2, E3};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = x4 + k, kp = (k + 3) & 3;
                write_state<LAK>(d, c, x, x4 + ((k + 1) & 3), x4 + kp, twx[k], twx[kp], qnext(twx[k]), qnext(twx[kp]),
                                 sl[k], tt[k], eP[k], eP[kp]);
            }
            c.sptr[d.V1 + y] = d.N1 + 4 * y;
            c.sptr[VF1 + E0] = 2 * d.N1 + 4 * E0;
            c.sptr[VF1 + E2] = 2 * d.N1 + 4 * E2;
            if (PQ ? (y & 3) == 0 : y == fb) c.sptr[q.z] = d.N2 + y;
            if (own) c.sptr[q.y] = 2 * d.N2 + 4 * ee;
        }
    }

    // ---- face points of the four quads
    const float4 q0 = quad_fp(LAK, Pv, Pa, Pg, Pd), q1 = quad_fp(LAK, Pe, Pb, Pg, Pa);
    const float4 q2 = quad_fp(LAK, Pf, Pc, Pg, Pb), q3 = quad_fp(LAK, Pi, Pd, Pg, Pc);
    if (valid) {
        st_pos4(R, (int64_t)d.V + 4 * (int64_t)y, q0, q1, q2, q3);
        // records of PP's old vertex v for k_g3: SLAK the face point alone (its
        // neighbour a is C's vertex VF1 + slot, in slot order already)
        if (!LAK) {
            z.Z[s2] = q0;
            z.rot[t2] = s2;
        } else {
            st8_keep(z.Z + 2 * (int64_t)s2, q0, Pd);
            z.T[s2] = VF1 + E3;
        }
        if (!PQ && fe - fb > kPpFace) {     // a long face's column goes to k_g3 as well
            const int64_t s = d.N2 + y;
            if (!LAK) {
                z.Z[s] = q2;
                z.rot[d.N2 + ny] = d.N2 + y;
            } else {
                st8_keep(z.Z + 2 * s, q2, Pb);
                z.T[s] = VF1 + E1;
            }
        }
    }

    // ---- what the neighbouring corners of the PP face hold
    float4 g_p, q1_p, q2_p, d_n, q3_n;      // prev: face point of its P face, C face points 1, 2; next: d, C face point 3
    if constexpr (PQ) {
        g_p = shfl4(Pg, lp); q1_p = shfl4(q1, lp); q2_p = shfl4(q2, lp);
        d_n = shfl4(Pd, ln); q3_n = shfl4(q3, ln);
    } else {
        // E0 of prev(y) (v(py)-ei) and E2 of prev(y) (f-ei(py)), E3 of next(y) (eo-vn)
        int E0p, E2p, E3n;
        if (!LAK) {
            E0p = __ldg(pp.slot + py); E2p = d.N2 + py; E3n = __ldg(pp.t + ny);
        } else {
            const int ppy = py == fb ? fe - 1 : py - 1;
            E0p = 4 * ep + (vp > q.x);
            E2p = 4 * (qp.w - VF2) + 2 + (py > __ldg(pp.tw + ppy));
            E3n = 4 * ee + (vn > q.x);
        }
        g_p = ldg4(P, d.V1 + py);
        const float4 a_p = ldg4(P, VF1 + E0p), c_p = ldg4(P, VF1 + E2p), g_n = ldg4(P, d.V1 + ny);
        d_n = ldg4(P, VF1 + E3n);
        q1_p = quad_fp(LAK, Pi, Pc, g_p, a_p);
        q2_p = quad_fp(LAK, Pf, c_p, g_p, Pc);
        q3_n = quad_fp(LAK, Pe, d_n, g_n, Pb);
    }

    // ---- vertex point of g and (SLAK) the edge points of C's edges at g
    if (valid) {
        if (!LAK) {
            const float4 acc = f4_add(f4_add(f4_add(f4_add(f4_zero(), Pd), Pa), Pb), Pc);
            float4 yv = f4_add(f4_div(acc, 16.0f), f4_div(f4_mul(Pg, 2.0f), 4.0f));
            yv = f4_add(yv, f4_div(q0, 16.0f));
            yv = f4_add(yv, f4_div(q1, 16.0f));
            yv = f4_add(yv, f4_div(q2, 16.0f));
            yv = f4_add(yv, f4_div(q3, 16.0f));
            st_pos<STATE>(R, d.V1 + y, yv);
            st_pos4(R, (int64_t)VFc + d.N1 + 4 * (int64_t)y, ep_slak(Pg, q0, Pd, q3), ep_slak(Pg, q1, Pa, q0),
                    ep_slak(Pg, q2, Pb, q1), ep_slak(Pg, q3, Pc, q2));
        } else {
            float4 acc = f4_add(f4_add(f4_add(f4_add(f4_zero(), q0), q1), q2), q3);
            // tails a, b, c, d in ascending id
            const int id[4] = {E0, E1, E2, E3};
            const float4 pt[4] = {Pa, Pb, Pc, Pd};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float4 x = pt[0];
#pragma unroll
                for (int j = 1; j < 4; ++j)
                    if (rank4(id[j], id[(j + 1) & 3], id[(j + 2) & 3], id[(j + 3) & 3]) == r) x = pt[j];
                acc = f4_add(acc, x);
            }
            st_pos<STATE>(R, d.V1 + y, f4_div_z(f4_add(f4_div_z(acc, 4.0f), f4_mul(Pg, 2.0f)), 4.0f));
        }
    }

    // ---- P's edge v-eo (edge point a): own quads 0, 1; far quads 4 nh2 + 3 and 4 nh2
    const float4 fD = quad_fp(LAK, Pe, Pa, Gn, PX);       // C face point of quad 4 nh2 + 3
    const float4 fW = quad_fp(LAK, Pv, PW, Gn, Pa);       // C face point of quad 4 nh2
    if (valid) {
        const bool of = y < nh2;
        if (!LAK) {
            // corners in order: own 4(4y)+1 (nbr g), 4(4y+1)+3 (nbr eo); far 4(4 nh2)+3 (nbr v), 4(4 nh2+3)+1 (nbr Gn)
            st4_cs(R, VF1 + E0, vp4_slak(of, Pa, Pg, Pe, Pv, Gn, q0, q1, fW, fD));
        } else {
            st4_cs(R, VF1 + E0, vp4_lak(of, Pa, q0, q1, fW, fD, Pv, Pe, of ? Pg : Gn, of ? Gn : Pg));
            const int64_t b = (int64_t)VFc + 4 * (int64_t)E0;
            const float4 eg = ep_lak(Pg, Pa, q1, q0), en = ep_lak(Gn, Pa, fW, fD);
            st_pos4(R, b, ep_lak(Pv, Pa, q0, fW), ep_lak(Pe, Pa, fD, q1), of ? eg : en, of ? en : eg);
        }
    }
    // ---- P's edge f-ei (edge point c): own quads 2, 3; prev(y)'s quads 1, 2
    if (valid) {
        const bool of = y < py;
        if (!LAK) {
            // own 4(4y+2)+1 (nbr g), 4(4y+3)+3 (nbr ei); far 4(4py+1)+1 (nbr g_p), 4(4py+2)+3 (nbr f)
            st4_cs(R, VF1 + E2, vp4_slak(of, Pc, Pg, Pi, g_p, Pf, q2, q3, q1_p, q2_p));
        } else {
            st4_cs(R, VF1 + E2, vp4_lak(of, Pc, q2, q3, q1_p, q2_p, Pf, Pi, of ? Pg : g_p, of ? g_p : Pg));
            const int64_t b = (int64_t)VFc + 4 * (int64_t)E2;
            const float4 eg = ep_lak(Pg, Pc, q3, q2), en = ep_lak(g_p, Pc, q2_p, q1_p);
            st_pos4(R, b, ep_lak(Pf, Pc, q2, q2_p), ep_lak(Pi, Pc, q1_p, q3), of ? eg : en, of ? en : eg);
        }
    }

    // ---- PP's edge point eo: P corners A = 4y+1, B = 4 ny+3 (own face), C = 4 tw+1, D = 4 nh2+3 (twin's)
    if (own) {
        const float4 fC = quad_fp(LAK, Pe, PX, Gt, d_n);
        const bool of = y < tw, lo = ny < y, lt = nh2 < tw;     // lo: B before A; lt: D before C
        if (!LAK) {
            // neighbours e_out: A b, B d(ny), C X, D a
            st_pos<STATE>(R, q.y, vp4_slak(of, Pe, lo ? d_n : Pb, lo ? Pb : d_n, lt ? Pa : PX, lt ? PX : Pa,
                                           lo ? q3_n : q1, lo ? q1 : q3_n, lt ? fD : fC, lt ? fC : fD));
            const int oe = of ? 0 : 2;
            const int64_t b = (int64_t)VFc + 2 * (int64_t)d.N2 + 4 * (int64_t)ee;
            st4_cs(R, b + oe + lo, ep_slak(Pe, q1, Pb, q3_n));            // quad A with B
            st4_cs(R, b + oe + !lo, ep_slak(Pe, q3_n, d_n, fC));          // B with C
            st4_cs(R, b + (2 - oe) + lt, ep_slak(Pe, fC, PX, fD));        // C with D
            st4_cs(R, b + (2 - oe) + !lt, ep_slak(Pe, fD, Pa, q1));       // D with A
        } else {
            // tails e_in of A, B, C, D = a, b, d(ny), X, with ids 4e + {0: a, 1: d(ny), 2, 3: b and X}
            st_pos<STATE>(R, q.y, vp4_lak(of, Pe, lo ? q3_n : q1, lo ? q1 : q3_n, lt ? fD : fC, lt ? fC : fD, Pa, d_n,
                                          of ? Pb : PX, of ? PX : Pb));
        }
    }

    // ---- PP's face point f: corners 4j+2 of the face's corners j, ascending
    if (!LAK && valid && (PQ || fe - fb <= kPpFace))
        st4_cs(R, (int64_t)VFc + d.N2 + y, ep_slak(Pf, q2, Pc, q2_p));     // slot N2 + y: quad y with prev(y)
    if constexpr (PQ) {
        float4 yv;
        const int gl = lane & ~3;
        if (!LAK) {
            float4 acc = f4_zero();
#pragma unroll
            for (int j = 0; j < 4; ++j) acc = f4_add(acc, shfl4(Pc, gl | j));
            yv = f4_add(f4_div(acc, 16.0f), f4_div(f4_mul(Pf, 2.0f), 4.0f));
#pragma unroll
            for (int j = 0; j < 4; ++j) yv = f4_add(yv, f4_div(shfl4(q2, gl | j), 16.0f));
        } else {
            float4 acc = f4_zero();
#pragma unroll
            for (int j = 0; j < 4; ++j) acc = f4_add(acc, shfl4(q2, gl | j));
            int id[4];                                      // the tails' ids: b of each corner
#pragma unroll
            for (int j = 0; j < 4; ++j) id[j] = __shfl_sync(full, E1, gl | j);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                int src = 0;
#pragma unroll
                for (int j = 1; j < 4; ++j)
                    if (rank4(id[j], id[(j + 1) & 3], id[(j + 2) & 3], id[(j + 3) & 3]) == r) src = j;
                acc = f4_add(acc, shfl4(Pb, gl | src));
            }
            yv = f4_div_z(f4_add(f4_div_z(acc, 4.0f), f4_mul(Pf, 2.0f)), 4.0f);
        }
        if (valid && (y & 3) == 0) st_pos<STATE>(R, q.z, yv);
    } else if (valid && y == fb && fe - fb <= kPpFace) {
        st_pos<STATE>(R, q.z, pp_face_vertex<LAK>(d, pids, P, pp, fb, fe, Pf, compensated));
    }

    if (LAK && !STATE && optr != nullptr) {
        // refined ptr[q] = 4q, vals[q] = {1, 2, 3, 4}: the block's 16 BS quads by consecutive threads
        const int64_t qb = 16 * (int64_t)y0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int64_t qq = qb + t + (int64_t)j * BS;
            if (qq < d.N) {
                __stcs(ovals + qq, make_int4(1, 2, 3, 4));
                __stcs(optr + qq, (int)(4 * qq));
            }
        }
        if (y0 + t == 0) optr[d.N] = 4 * d.N;
    }
    // the tensor stores have read the staging buffer and their writes are done
    if (t < 2) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
template <bool LAK, bool STATE, bool PQ, int BS>
__global__ void __launch_bounds__(BS, 512 / BS) k_pp(FastDims d, Faces<PQ> pf, const int4* __restrict__ pids,
                                                     const float* __restrict__ P, QState pp, QState c, int wids,
                                                     const __grid_constant__ CUtensorMap otm, float* __restrict__ R,
                                                     SlotScratch z, int* __restrict__ optr, int4* __restrict__ ovals,
                                                     int compensated)
{
    griddep_enter();
    k_pp_body<LAK, STATE, PQ, BS>(blockIdx.x, d, pf, pids, P, pp, c, wids, otm, R, z, optr, ovals, compensated);
}
template <bool LAK, bool STATE, bool PQ, int BS>
struct k_pp_g {
    static constexpr int kBounds = 2, kMaxT = BS, kMinB = 512 / BS;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const
    {
        k_pp_body<LAK, STATE, PQ, BS>(bx, a...);
    }
    static constexpr auto kernel() { return &k_pp<LAK, STATE, PQ, BS>; }
};

}  // namespace slak
