// levels.cu -- launches of the closed-form levels (fast.cuh, grand.cuh).
//
// Compiled once per SLAK_UNIT (1 to 7), each with the kernels of one kind of
// parent, so that the kinds build side by side.
#include <cstring>
#include <mutex>
#include <cudaTypedefs.h>

#include "plan.cuh"
#include "grand.cuh"
#include "poly1.cuh"

namespace slak {
namespace {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 enc = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            enc = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    });
    return enc;
}

// The tensor map of a level's refined quads for k_g1's tensor store: `rows`
// rows of 16 int32 (thread x's four quads at out + 16 x), boxes of `bs` rows,
// 64-byte swizzle (the layout k_g1 stages them in).  A null `out` (a launch
// sequence recorded before any memory exists) leaves the map zeroed.
bool quad_store_map(CUtensorMap& m, int* out, int64_t rows, int bs)
{
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (out == nullptr) return true;
    if (enc == nullptr || rows < 1) {
        g_detail = "cuTensorMapEncodeTiled unavailable";
        return false;
    }
    const cuuint64_t dims[2] = {16, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {64};
    const cuuint32_t box[2] = {16, (cuuint32_t)bs};
    const cuuint32_t es[2] = {1, 1};
    const CUresult r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, out, dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) g_detail = "cuTensorMapEncodeTiled: error " + std::to_string((int)r);
    return r == CUDA_SUCCESS;
}

// The same of a PP level (grand.cuh): thread y's 256 bytes as two rows of 128
// (halves of one row of 64 int32), boxes of one half of `bs` threads, 128-byte
// swizzle.
bool quad_store_map2(CUtensorMap& m, int* out, int64_t rows, int bs)
{
    if (out == nullptr) return true;
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (enc == nullptr || rows < 1) {
        g_detail = "cuTensorMapEncodeTiled unavailable";
        return false;
    }
    const cuuint64_t dims[3] = {32, 2, (cuuint64_t)rows};
    const cuuint64_t strides[2] = {128, 256};
    const cuuint32_t box[3] = {32, 1, (cuuint32_t)bs};
    const cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_INT32, 3, out, dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) g_detail = "cuTensorMapEncodeTiled: error " + std::to_string((int)r);
    return r == CUDA_SUCCESS;
}

// One fast level: C = L (refined from its parent level Pl, whose state is
// L.in_state).  BND: Pl has a boundary (quad faces only).
template <bool LAK, bool STATE, bool PQ, bool BND, bool GQ = false, bool SG = false>
void launch_fast_t(const Level& Pl, const Level& L, Faces<PQ> pf, bool comp, Lc& lc)
{
    FastDims d{(int)Pl.N, (int)Pl.V, (int)Pl.F, (int)Pl.E, (int)L.V, (int)L.N, (int)Pl.B};
    if (GQ || SG) { d.N2 = (int)L.gN; d.V2 = (int)L.gV; d.F2 = (int)L.gF; }
    const int nv3 = GQ ? (int)L.gV : (int)Pl.V;      // k_g3's vertices
    const int mode = (comp ? G3_COMP : 0) | (L.longcol ? G3_LONG : 0);
    cudaStream_t str = lc.s;
    // compulsory bytes of each kernel: the level's corner ids and positions it
    // must read once, and the refined ids / positions it alone writes
    const int64_t g1b = 4 * L.N + 16 * L.V + (L.skip_ids ? 0 : 16 * L.N) + 16 * L.F + 16 * Pl.F + (LAK ? 0 : 16 * L.F);
    const int64_t g2b = 16 * Pl.E + (LAK ? 16 * 2 * L.F : 0);
    // LAK's last level: the refined ptr / vals come from k_g1 too
    int* optr = LAK && !STATE ? L.o_ptr : nullptr;
    int4* ovals = LAK && !STATE ? reinterpret_cast<int4*>(L.o_vals) : nullptr;
    bool mapped = true;
    with_block(L.bs[0], [&](auto b) {
        constexpr int BS = decltype(b)::value;
        CUtensorMap otm;
        std::memset(&otm, 0, sizeof otm);
        if constexpr (!STATE && kTmaQuadStore && BS <= 256) mapped = quad_store_map(otm, L.o_ids, Pl.N, BS);
        if (!mapped) return;            // nothing of the level is launched
        launch_g<k_g1_g<LAK, STATE, PQ, BS, BND, GQ, SG>>(grid_for(L.F, BS), BS, str, d, pf, L.ids, L.verts, L.in_state,
                                                          L.out_state, reinterpret_cast<int4*>(L.o_ids), otm, L.o_verts,
                                                          L.slots, optr, ovals);
    });
    if (!mapped) {
        if (!lc.err) lc.err = SLAK_ERR_CUDA;
        return;
    }
    // GQ: k_g1 also writes the vertex points of P's vertices past V2 (and SLAK their slots' edge points)
    const int64_t gqb = GQ ? 16 * (Pl.V - L.gV) + (LAK ? 0 : 16 * (L.F - L.gN)) : 0;
    lc.after("k_g1", 1, (PQ ? g1b + g2b : g1b) + (optr ? 4 * (L.N + 1) + 16 * L.N : 0) + gqb);
    if (!PQ) {      // with quad faces, k_g1 also does k_gf's and k_g2's work
        // k_gf, k_g2 and k_g3 read only k_g1's records and the level's inputs and
        // write disjoint outputs: with side streams they run side by side
        if (lc.conc) { lc.fork(0); lc.fork(1); }
        launch_g<k_gf_g<LAK, STATE>>(grid_for(Pl.F), kBlock, lc.conc ? lc.side[0] : str, d, Pl.ptr, L.ids, L.verts, L.out_state, L.o_verts, comp ? 1 : 0);
        lc.after("k_gf");
        with_block(L.bs[1], [&](auto b) {
            constexpr int BS = decltype(b)::value;
            launch_g<k_g2_g<LAK, STATE, PQ, BS, BND>>(grid_for(L.F, BS), BS, lc.conc ? lc.side[1] : str, d, pf, L.ids, L.verts, L.in_state, L.out_state, L.o_verts);
        });
        lc.after("k_g2", 1, g2b);
    }
    if (!BND && !SG && L.bulk3) {
        launch_g<k_g3_bulk_g<LAK, STATE>>(grid_for(nv3 + 1, kBulkBlock), kBulkBlock, str, d, L.verts, L.in_state, L.out_state, L.slots, L.o_verts, comp ? 1 : 0, nv3, L.st, L.bulk_polls);
    } else {
        with_block(L.bs[2], [&](auto b) {
            constexpr int BS = decltype(b)::value;
            launch_g<k_g3_g<LAK, STATE, BS, BND, SG>>(grid_for(nv3 + 1, BS), BS, str, d, L.verts, L.in_state, L.out_state, L.slots, L.o_verts, mode, nv3, nullptr, 0);
        });
    }
    // compulsory bytes: the vertex points of its vertices, SLAK the edge points of their slots
    const int64_t ns3 = GQ ? L.gN : L.F;
    lc.after("k_g3", 1, 16 * (int64_t)nv3 + (LAK ? 0 : 16 * ns3));
    if (BND && STATE && !LAK) {    // C's edges 0..N1-1 (P's slots): boundary ranks by a scan
        const int nl = scan_launch(L.slots.bscan, L.out_state.brank, Pl.N, L.scan_tmp, str);
        lc.after("scan(boundary)", nl);
    }
    if (!PQ && lc.conc) { lc.join(0); lc.join(1); }
}

template <bool PQ, bool BND, bool GQ = false>
void launch_fast_p(const Level& Pl, const Level& L, Faces<PQ> pf, bool lak, bool comp, Lc& lc)
{
    if constexpr (GQ) {
        if (L.sg) {             // the last level: no state to write
            if (lak) launch_fast_t<true, false, PQ, BND, GQ, true>(Pl, L, pf, comp, lc);
            else launch_fast_t<false, false, PQ, BND, GQ, true>(Pl, L, pf, comp, lc);
            return;
        }
    }
    if (lak) {
        if (L.make_state) launch_fast_t<true, true, PQ, BND, GQ>(Pl, L, pf, comp, lc);
        else launch_fast_t<true, false, PQ, BND, GQ>(Pl, L, pf, comp, lc);
    } else {
        if (L.make_state) launch_fast_t<false, true, PQ, BND, GQ>(Pl, L, pf, comp, lc);
        else launch_fast_t<false, false, PQ, BND, GQ>(Pl, L, pf, comp, lc);
    }
}

// One PP level (grand.cuh): C = L, its parent Pl and its parent's parent PPl,
// whose state is L.in_state.  The block size bs[0] counts C's quads: four per
// thread of k_pp.
template <bool LAK, bool STATE, bool PQ>
void launch_pp_t(const Level& PPl, const Level& Pl, const Level& L, Faces<PQ> pf, bool comp, Lc& lc)
{
    FastDims d{(int)Pl.N, (int)Pl.V, (int)Pl.F, (int)Pl.E, (int)L.V, (int)L.N, 0};
    d.N2 = (int)PPl.N; d.V2 = (int)PPl.V; d.F2 = (int)PPl.F;
    int* optr = LAK && !STATE ? L.o_ptr : nullptr;
    int4* ovals = LAK && !STATE ? reinterpret_cast<int4*>(L.o_vals) : nullptr;
    const int wids = L.skip_ids ? 0 : 1;
    bool mapped = true;
    with_block(L.bs[0], [&](auto b) {
        constexpr int BS = decltype(b)::value / 4;
        CUtensorMap otm;
        std::memset(&otm, 0, sizeof otm);
        if (wids) mapped = quad_store_map2(otm, L.o_ids, PPl.N, BS);
        if (!mapped) return;            // nothing of the level is launched
        launch_g<k_pp_g<LAK, STATE, PQ, BS>>(grid_for(PPl.N, BS), BS, lc.s, d, pf, reinterpret_cast<const int4*>(Pl.ids),
                                             L.verts, L.in_state, L.out_state, wids, otm, L.o_verts, L.slots, optr,
                                             ovals, comp ? 1 : 0);
    });
    if (!mapped) {
        if (!lc.err) lc.err = SLAK_ERR_CUDA;
        return;
    }
    // compulsory bytes: the parent's quads and C's positions in; the refined
    // quads, all refined positions but k_g3's out
    const int64_t g3 = 16 * PPl.V + (LAK ? 0 : 16 * PPl.N);
    lc.after("k_pp", 1, 16 * PPl.N + 16 * L.V + (wids ? 16 * L.N : 0) + 16 * L.Vo - g3 +
                            (optr ? 4 * (L.N + 1) + 16 * L.N : 0));
    const int nv = (int)(PQ ? PPl.V : PPl.V + PPl.F);
    const int mode = (comp ? G3_COMP : 0) | (L.longcol ? G3_LONG : 0);
    with_block(L.bs[2], [&](auto b) {
        constexpr int BS = decltype(b)::value;
        launch_g<k_g3_g<LAK, STATE, BS, false, false, true>>(grid_for(nv + 1, BS), BS, lc.s, d, L.verts, L.in_state,
                                                             L.out_state, L.slots, L.o_verts, mode, nv,
                                                             PQ ? nullptr : PPl.ptr, kPpFace);
    });
    lc.after("k_g3", 1, g3);
}

template <bool PQ>
void launch_pp(const Level& PPl, const Level& Pl, const Level& L, Faces<PQ> pf, bool lak, bool comp, Lc& lc)
{
    if (lak) {
        if (L.make_state) launch_pp_t<true, true, PQ>(PPl, Pl, L, pf, comp, lc);
        else launch_pp_t<true, false, PQ>(PPl, Pl, L, pf, comp, lc);
    } else {
        if (L.make_state) launch_pp_t<false, true, PQ>(PPl, Pl, L, pf, comp, lc);
        else launch_pp_t<false, false, PQ>(PPl, Pl, L, pf, comp, lc);
    }
}

}  // namespace

#if SLAK_UNIT == 1
void launch_fast_quad(const Level& Pl, const Level& L, bool lak, bool comp, Lc& lc)
{
    launch_fast_p<true, false>(Pl, L, Faces<true>{nullptr, nullptr}, lak, comp, lc);
}
#elif SLAK_UNIT == 2
void launch_fast_quad_open(const Level& Pl, const Level& L, bool lak, bool comp, Lc& lc)
{
    launch_fast_p<true, true>(Pl, L, Faces<true>{nullptr, nullptr}, lak, comp, lc);
}
#elif SLAK_UNIT == 3
void launch_fast_gq(const Level& Pl, const Level& L, bool lak, bool comp, Lc& lc)
{
    launch_fast_p<true, false, true>(Pl, L, Faces<true>{nullptr, nullptr}, lak, comp, lc);
}
#elif SLAK_UNIT == 4
// Level 1 of a closed polygon input (poly1.cuh): C = L, its parent Pl the
// input.  k_p1 runs blocks of bs[0] / 2 threads; bs[1] picks its register cap
// (128, 256, 512: for 1024, 768, 512 resident threads).  Bulk-copied records: as
// launch_fast_t's.
template <bool LAK, bool STATE>
static void launch_p1_t(const Level& Pl, const Level& L, Faces<false> pf, bool comp, Lc& lc)
{
    FastDims d{(int)Pl.N, (int)Pl.V, (int)Pl.F, (int)Pl.E, (int)L.V, (int)L.N, 0};
    int* optr = LAK && !STATE ? L.o_ptr : nullptr;
    int4* ovals = LAK && !STATE ? reinterpret_cast<int4*>(L.o_vals) : nullptr;
    const int mode = (comp ? G3_COMP : 0) | (L.longcol ? G3_LONG : 0);
    bool mapped = true;
    with_block(L.bs[0], [&](auto b) {
        constexpr int BS = decltype(b)::value / 2;
        CUtensorMap otm;
        std::memset(&otm, 0, sizeof otm);
        if (!STATE) mapped = quad_store_map(otm, L.o_ids, Pl.N, BS);
        if (!mapped) return;            // nothing of the level is launched
        with_block(L.bs[1], [&](auto r) {
            constexpr int RT = decltype(r)::value == 128 ? 1024 : decltype(r)::value == 256 ? 768 : 512;
            const unsigned nb = grid_for(L.F, BS);
            launch_g<k_p1_g<LAK, STATE, BS, RT>>(nb + grid_for(Pl.F, BS), BS, lc.s, d, pf,
                                                 reinterpret_cast<const int4*>(L.ids), L.verts, L.in_state, L.out_state,
                                                 reinterpret_cast<int4*>(L.o_ids), otm, L.o_verts, L.slots, optr,
                                                 ovals, comp ? 1 : 0, (int)nb);
        });
    });
    if (!mapped) {
        if (!lc.err) lc.err = SLAK_ERR_CUDA;
        return;
    }
    const int64_t g3 = 16 * Pl.V + (LAK ? 0 : 16 * L.F);
    lc.after("k_p1", 1, 4 * L.N + 16 * L.V + (L.skip_ids ? 0 : 16 * L.N) + 16 * L.Vo - g3 +
                            (optr ? 4 * (L.N + 1) + 16 * L.N : 0));
    if (L.bulk3) {
        launch_g<k_g3_bulk_g<LAK, STATE>>(grid_for(Pl.V + 1, kBulkBlock), kBulkBlock, lc.s, d, L.verts, L.in_state,
                                          L.out_state, L.slots, L.o_verts, comp ? 1 : 0, (int)Pl.V, L.st, L.bulk_polls);
    } else {
        with_block(L.bs[2], [&](auto b) {
            constexpr int BS = decltype(b)::value;
            launch_g<k_g3_g<LAK, STATE, BS>>(grid_for(Pl.V + 1, BS), BS, lc.s, d, L.verts, L.in_state, L.out_state, L.slots,
                                             L.o_verts, mode, (int)Pl.V, nullptr, 0);
        });
    }
    lc.after("k_g3", 1, g3);
}

void launch_p1(const Level& Pl, const Level& L, Faces<false> pf, bool lak, bool comp, Lc& lc)
{
    if (lak) {
        if (L.make_state) launch_p1_t<true, true>(Pl, L, pf, comp, lc);
        else launch_p1_t<true, false>(Pl, L, pf, comp, lc);
    } else {
        if (L.make_state) launch_p1_t<false, true>(Pl, L, pf, comp, lc);
        else launch_p1_t<false, false>(Pl, L, pf, comp, lc);
    }
}
#elif SLAK_UNIT == 5
void launch_fast_poly_open(const Level& Pl, const Level& L, const int* cface, bool lak, bool comp, Lc& lc)
{
    launch_fast_p<false, true>(Pl, L, Faces<false>{Pl.ptr, cface}, lak, comp, lc);
}
#elif SLAK_UNIT == 6
void launch_pp_quad(const Level& PPl, const Level& Pl, const Level& L, bool lak, bool comp, Lc& lc)
{
    launch_pp<true>(PPl, Pl, L, Faces<true>{nullptr, nullptr}, lak, comp, lc);
}
#elif SLAK_UNIT == 7
void launch_pp_poly(const Level& PPl, const Level& Pl, const Level& L, Faces<false> pf, bool lak, bool comp, Lc& lc)
{
    launch_pp<false>(PPl, Pl, L, pf, lak, comp, lc);
}
#endif

}  // namespace slak
