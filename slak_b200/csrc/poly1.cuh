// poly1.cuh -- level 1 of a closed polygon mesh.
//
// P is the polygon input (its state from closed0.cuh), C = refine(P) the level
// being refined: quad x of C is corner x of P, {v, e_out, f, e_in}.  One thread
// per corner does what k_g1, k_gf and k_g2 do for an open polygon parent in
// three launches: where those hand C's face points to each other through
// memory, a thread here loads the quads of its neighbours (next(x), prev(x), and
// across its edge tw(x) and next(tw(x))), whose positions its warp has mostly in
// L1, and recomputes their face points.  The face points' own vertex points
// are sums over whole faces: one thread per face, in the blocks after the corners'.  k_g3 then takes P's vertices from the
// slot records, as at every level.  Numbering, formulas and their order are
// fast.cuh's.
//
// Bound by load latency (the level moves 0.2 GB at 1 M corners).  Measured on
// B200, 512x512 mixed torus, launch by launch: k_g1 + k_gf + k_g2 39 + 29 + 33 ->
// k_p1 62 us; with level 0's corner positions and next(twin) (Faces::nav,
// QState::nt) read by k_pp as well, the whole step 757 -> 733 us (SLAK), 1022 ->
// 1010 us (LAK), a batch of 32 small meshes 125.6 -> 118.8 us.
#pragma once

#include "grand.cuh"

namespace slak {

// Vertex point of P's face point f (position Pf) with corners fb..fe-1: its
// column is the corners' quads, each {v, e_out, f, e_in}, e_in the e_out before.
// SLAK: e_in in corner order, then the face points; LAK: the face points, then
// e_out in ascending id (g3_vertex's order and formulas).
template <bool LAK>
__device__ __forceinline__ float4 p1_face_vertex(const int4* __restrict__ ids, const float* __restrict__ P, int fb,
                                                 int fe, float4 Pf, int compensated)
{
    const int k = fe - fb;
    const float nn = (float)(k * k);
    const bool comp = compensated && k > 4;
    float4 acc = f4_zero(), sh = f4_zero(), sl = f4_zero(), yv = f4_zero();
    const auto add = [&](int, float4 x) { if (comp) dd_acc(sh, sl, x); else acc = f4_add(acc, x); };
    if (!LAK) {
        for_each_loaded(k, [&](int j) { return ldg4(P, __ldg(&ids[fb + j].w)); }, add);
        yv = f4_add(f4_div(acc, nn), f4_div(f4_mul(Pf, (float)(k - 2)), (float)k));
    }
    float4 ei = ldg4(P, __ldg(&ids[fb].w));
    for (int j0 = fb; j0 < fe; j0 += 4) {                // four corners' loads in flight
        float4 pv[4], eo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (j0 + i < fe) {
                const int4 q = __ldg(ids + j0 + i);
                pv[i] = ldg4(P, q.x);
                eo[i] = ldg4(P, q.y);
            }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (j0 + i < fe) {
                const float4 fp = quad_fp(LAK, pv[i], eo[i], Pf, ei);
                if (LAK || comp) add(0, fp);
                else yv = f4_add(yv, f4_div(fp, nn));
                ei = eo[i];
            }
    }
    if (LAK) {
        if (k <= 8) {
            int id[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) id[j] = j < k ? __ldg(&ids[fb + j].y) : INT32_MAX;
            sort_keys<8>(id);
#pragma unroll
            for (int j0 = 0; j0 < 8; j0 += 4) {
                float4 t[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (j0 + i < k) t[i] = ldg4(P, id[j0 + i]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (j0 + i < k) add(0, t[i]);
            }
        } else {
            for (int last = -1;;) {
                int xm = INT32_MAX;
                for (int j = fb; j < fe; ++j) {
                    const int x = __ldg(&ids[j].y);
                    if (x > last && x < xm) xm = x;
                }
                if (xm == INT32_MAX) break;
                add(0, ldg4(P, xm));
                last = xm;
            }
        }
        yv = f4_div_z(f4_add(f4_div_z(acc, (float)k), f4_mul(Pf, __fadd_rn((float)k, -2.0f))), (float)k);
    }
    return comp ? vp_finish(sh, sl, Pf, k) : yv;
}

template <bool LAK, bool STATE, int BS>
__device__ __forceinline__ void k_p1_body(const unsigned bx_, FastDims d, Faces<false> pf, const int4* __restrict__ ids,
                                          const float* __restrict__ P, QState p, QState c, int4* __restrict__ out_ids,
                                          const CUtensorMap& otm, float* __restrict__ R, SlotScratch z,
                                          int* __restrict__ optr, int4* __restrict__ ovals, int compensated, int nb)
{
    if (bx_ >= (unsigned)nb) {          // the blocks after the corners': one thread per face
        const int g = (bx_ - nb) * BS + threadIdx.x;
        if (g >= d.F1) return;
        const int fb = __ldg(pf.ptr + g), fe = __ldg(pf.ptr + g + 1);
        st_pos<STATE>(R, d.V1 + g, p1_face_vertex<LAK>(ids, P, fb, fe, ldg4(P, d.V1 + g), compensated));
        if (STATE) c.sptr[d.V1 + g] = d.N1 + fb;
        return;
    }
    const int x0 = bx_ * BS, t = threadIdx.x;
    const bool valid = x0 + t < d.N1;
    const int x = valid ? x0 + t : 0;                   // idle threads repeat corner 0's loads
    const int VF1 = d.V1 + d.F1, VFc = d.V + d.N1;

    const int4 Q = __ldg(ids + x);
    const int tw = __ldg(p.tw + x), nt = __ldg(p.nt + x), s1 = __ldg(p.slot + x), t1 = LAK ? 0 : __ldg(p.t + x);
    int nx, px;
    pf.around(x, nx, px);
    const int4 qn = __ldg(ids + nx), qp = __ldg(ids + px);
    const int twp = LAK || STATE ? __ldg(p.tw + px) : 0, ntp = STATE ? __ldg(p.nt + px) : 0;
    const bool own = Q.x < qn.x;
    const float4 c0 = ldg4(P, Q.x), c1 = ldg4(P, Q.y), c2 = ldg4(P, Q.z), c3 = ldg4(P, Q.w);
    const float4 Pu = ldg4(P, qn.x), Pen = ldg4(P, qn.y);
    float4 Pf2 = f4_zero(), Pi2 = f4_zero(), Po3 = f4_zero();
    int fh2 = 0;
    if (own) {                                          // across the edge: quads tw and next(tw)
        const int4 q2 = __ldg(ids + tw);
        const int eo3 = __ldg(&ids[nt].y);
        fh2 = q2.z;
        Pf2 = ldg4(P, q2.z); Pi2 = ldg4(P, q2.w); Po3 = ldg4(P, eo3);
    }

    // edge ids of C's corners 4x+k
    const int eo = Q.y - VF1, ei = Q.w - VF1;
    int e0, e1, e2, e3;
    if (!LAK) {
        e0 = s1; e1 = d.N1 + nx; e2 = d.N1 + x; e3 = t1;
    } else {
        e0 = 4 * eo + (Q.x > qn.x);
        e1 = 4 * eo + 2 + (x > tw);                     // faces compare as their corners do
        e2 = 4 * ei + 2 + (x > twp);
        e3 = 4 * ei + (Q.x > qp.x);
    }
    const int fpid = d.V + x;
    if constexpr (STATE) {
        if (valid) {
            int4* dst = out_ids + 4 * (int64_t)x;
            st8_cs(dst, make_int4(Q.x, VFc + e0, fpid, VFc + e3), make_int4(Q.y, VFc + e1, fpid, VFc + e0));
            st8_cs(dst + 2, make_int4(Q.z, VFc + e2, fpid, VFc + e1), make_int4(Q.w, VFc + e3, fpid, VFc + e2));
            write_state<LAK>(d, c, x, nx, px, tw, twp, nt, ntp, s1, t1, eo, ei);
        }
    } else if (out_ids != nullptr) {
        // staged in the tensor map's 64-byte swizzle and stored by one TMA tensor store, as k_g1's
        __shared__ __align__(1024) int4 sq[4 * BS];
        const int sw = (t >> 1) & 3;
        sq[4 * t + (0 ^ sw)] = make_int4(Q.x, VFc + e0, fpid, VFc + e3);
        sq[4 * t + (1 ^ sw)] = make_int4(Q.y, VFc + e1, fpid, VFc + e0);
        sq[4 * t + (2 ^ sw)] = make_int4(Q.z, VFc + e2, fpid, VFc + e1);
        sq[4 * t + (3 ^ sw)] = make_int4(Q.w, VFc + e3, fpid, VFc + e2);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (t == 0) {
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
                         :: "l"(reinterpret_cast<uint64_t>(&otm)), "r"(0), "r"(x0),
                            "r"((uint32_t)__cvta_generic_to_shared(sq))
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    }

    const float4 fp = quad_fp(LAK, c0, c1, c2, c3);
    if (valid) {
        st_pos<STATE>(R, (int64_t)d.V + x, fp);
        st8_keep(z.Z + 2 * (int64_t)s1, fp, LAK ? c3 : c1);
        if (LAK) z.T[s1] = Q.w;
        else z.rot[t1] = s1;
        if (!LAK) {             // edge point N1 + x: quads x and prev(x)
            const float4 fpp = quad_fp(LAK, ldg4(P, qp.x), c3, c2, ldg4(P, qp.w));
            st4_cs(R, (int64_t)VFc + d.N1 + x, ep_slak(c2, fp, c3, fpp));
        }
    }
    if (valid && own) {
        const float4 fn = quad_fp(LAK, Pu, Pen, c2, c1);
        const float4 F2 = quad_fp(LAK, Pu, c1, Pf2, Pi2), Fn2 = quad_fp(LAK, c0, Po3, Pf2, c1);
        edge_point_vertex<LAK, STATE>(d, c, R, x, nx, tw, nt, Q.y, Q.z, fh2, c0, Pu, c1, c2, Pf2, fp, fn, F2, Fn2);
    }
    if (LAK && !STATE && optr != nullptr) {
        const int64_t q0 = 4 * (int64_t)x0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t qq = q0 + t + (int64_t)j * BS;
            if (qq < d.N) {
                __stcs(ovals + qq, make_int4(1, 2, 3, 4));
                __stcs(optr + qq, (int)(4 * qq));
            }
        }
        if (x0 + t == 0) optr[d.N] = 4 * d.N;
    }
    if constexpr (!STATE) {
        if (t == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
}
// RT: the resident threads per SM the registers are capped for.
template <bool LAK, bool STATE, int BS, int RT>
__global__ void __launch_bounds__(BS, RT / BS) k_p1(FastDims d, Faces<false> pf, const int4* __restrict__ ids,
                                                     const float* __restrict__ P, QState p, QState c,
                                                     int4* __restrict__ out_ids, const __grid_constant__ CUtensorMap otm,
                                                     float* __restrict__ R, SlotScratch z, int* __restrict__ optr,
                                                     int4* __restrict__ ovals, int compensated, int nb)
{
    griddep_enter();
    k_p1_body<LAK, STATE, BS>(blockIdx.x, d, pf, ids, P, p, c, out_ids, otm, R, z, optr, ovals, compensated, nb);
}
template <bool LAK, bool STATE, int BS, int RT>
struct k_p1_g {
    static constexpr int kBounds = 2, kMaxT = BS, kMinB = RT / BS;
    template <class... A> __device__ __forceinline__ void operator()(unsigned bx, const A&... a) const
    {
        k_p1_body<LAK, STATE, BS>(bx, a...);
    }
    static constexpr auto kernel() { return &k_p1<LAK, STATE, BS, RT>; }
};

}  // namespace slak
