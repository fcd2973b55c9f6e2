// One Heun stage of a 256-cell block from packed records (the dense whole-step kernel).
//
// A dense step is bound by issue and barriers, not by bytes, so a block's work is
// laid out for few instructions per edge:
//   * the velocities of every cell the block's edges read (its own and its halo
//     list's) are computed once, by one thread per cell, into float4 (h, u, v, inv)
//     in shared memory, instead of twice per edge from momenta: an edge reads each
//     side with one 16-byte load, and the reciprocal inv serves the side of the face
//     whose depth is the cell's own. A halo cell's state crosses L2 once per block;
//   * an edge record is one float4 (normal, length, both cells as local indices) and
//     one float2 (bed steps): 24 bytes instead of 28 in seven arrays;
//   * an edge's words go back over its own record: (w0, w1, w2, w5) over the float4,
//     (w3, w4) over the float2. The right cell adds -w0, -w3, -w4 (adding -w is
//     subtracting w, bit for bit). An edge that is not computed holds zeros: a sum
//     that starts at +0 is never -0, and adding either zero to it changes nothing.
// The records, the CSR pointers and the local CSR arrive by bulk copies on one
// mbarrier while the threads load the cells' states.
// A stage executes 1534 warp instructions per 32 cells this way (a million wet cells, 20 steps).
#pragma once

#include "swe_tiled.cuh"

namespace swe {

constexpr uint32_t kNoCell = 0xFFFFu;  // local index beyond a boundary edge

struct BlockPlan {
    uint32_t capE, capV, capS, total;
};

__host__ __device__ inline BlockPlan block_plan(uint32_t max_edges, uint32_t max_halo, uint32_t max_slots) {
    BlockPlan L;
    L.capE = (max_edges + 31u) & ~31u;
    L.capV = kBlockCells + max_halo;
    L.capS = (max_slots + 7u) & ~7u;
    L.total = 128u + 24u * L.capE + 16u * L.capV + 1040u + ((2u * L.capS + 15u) & ~15u);
    return L;
}

struct BlockBuf {
    uint64_t *bar;
    float4 *rec;  // records, then the words (w0, w1, w2, w5)
    float4 *V;    // (h, u, v, inv) of the block's cells, then its halo cells
    float2 *dz;   // bed steps, then the words (w3, w4)
    uint32_t *cptr;
    uint16_t *lcsr;
};

__device__ __forceinline__ BlockBuf block_buf(unsigned char *smem, const BlockPlan &L) {
    BlockBuf B;
    B.bar = reinterpret_cast<uint64_t *>(smem);
    B.rec = reinterpret_cast<float4 *>(smem + 128u);
    B.V = B.rec + L.capE;
    B.dz = reinterpret_cast<float2 *>(B.V + L.capV);
    B.cptr = reinterpret_cast<uint32_t *>(B.dz + L.capE);
    B.lcsr = reinterpret_cast<uint16_t *>(B.cptr + 260);
    return B;
}

// What a block's stage needs to know of it: dt bits, first record and records, first
// local-CSR slot and slots, real cells, first halo entry and halo cells, first source and sources.
struct BlockItem {
    uint32_t b, inst, dt, e0, ne, l0, lp, cells, h0, nh, s0, ns;
};

__device__ __forceinline__ BlockItem block_item(const swe_mesh_t &m, const swe_blocks_t &k, uint32_t b, uint32_t inst,
                                                uint32_t dt) {
    BlockItem it;
    it.b = b;
    it.inst = inst;
    it.dt = dt;
    it.e0 = m.tile_ptr[b];
    it.ne = m.tile_count[b];
    it.l0 = m.blk_lcsr_ptr[b];
    it.lp = m.blk_lcsr_ptr[b + 1] - it.l0;
    it.cells = m.block_cells[b];
    it.h0 = k.halo_ptr[b];
    it.nh = k.halo_ptr[b + 1] - it.h0;
    it.s0 = it.ns = 0u;
    if (k.src_ptr) {
        it.s0 = k.src_ptr[b];
        it.ns = k.src_ptr[b + 1] - it.s0;
    }
    return it;
}

// Warp 0: the block's records and CSR into shared memory, one bulk copy per lane.
__device__ __forceinline__ void block_issue(const swe_mesh_t &m, const swe_blocks_t &k, const BlockItem &it, const BlockBuf &B) {
    const uint32_t lane = threadIdx.x & 31u, ep = (it.ne + 31u) & ~31u;  // segments are padded to 32 records
    if (lane == 0) mbar_expect_tx(B.bar, 24u * ep + 1040u + 2u * it.lp);
    __syncwarp();
    if (lane == 0) {
        if (ep) bulk_load(B.rec, k.rec + 4ull * it.e0, 16u * ep, B.bar);
    } else if (lane == 1) {
        if (ep) bulk_load(B.dz, k.dz + 2ull * it.e0, 8u * ep, B.bar);
    } else if (lane == 2) {
        bulk_load(B.cptr, m.cptr + static_cast<size_t>(it.b) * kBlockCells, 1040u, B.bar);
    } else if (lane == 3) {
        if (it.lp) bulk_load(B.lcsr, m.blk_lcsr + it.l0, 2u * it.lp, B.bar);
    }
}

// safe_vel2 of one cell: (h, u, v, inv).
__device__ __forceinline__ float4 cell_velocity(const Phys &p, float h, float hu, float hv) {
    const float inv = vel_inv(p, h), twice = 2.0f * h;
    float u = twice * hu * inv, v = twice * hv * inv;
    if (!(h > p.dry_tol)) u = v = 0.0f;
    return make_float4(h, u, v, inv);
}

// The velocities of the block's cells and of its halo cells (all threads). The block is active:
// its own stage input in the corrector is the predictor. *odd is set when a cell is not plain_cell.
template <int STAGE>
__device__ __forceinline__ void block_velocities(const swe_blocks_t &blocks, const swe_state_t &s,
                                                 const Phys &p, const BlockItem &it, const BlockBuf &B,
                                                 volatile uint32_t *odd) {
    const uint32_t tid = threadIdx.x, i = it.b * kBlockCells + tid;
    const float h = STAGE ? s.h1[i] : s.h[i], hu = STAGE ? s.hu1[i] : s.hu[i], hv = STAGE ? s.hv1[i] : s.hv[i];
    for (uint32_t k = tid; k < it.nh; k += kThreads) {
        float hh, hhu, hhv;
        load_state<STAGE>(s, static_cast<int>(blocks.halo[it.h0 + k]), hh, hhu, hhv);
        const float4 c = cell_velocity(p, hh, hhu, hhv);
        B.V[kBlockCells + k] = c;
        if (!plain_cell(p, c)) *odd = 1u;
    }
    const float4 c = cell_velocity(p, h, hu, hv);
    B.V[tid] = c;
    if (!plain_cell(p, c)) *odd = 1u;
}

// Record j of the block into its words. False, with nothing stored, when M cannot compute it.
template <int STAGE, bool OPEN, class M>
__device__ __forceinline__ bool block_edge(const swe_mesh_t &m, const swe_state_t &s, const Phys &p, const BlockItem &it,
                                           const BlockBuf &B, uint32_t j, float dt) {
    const float4 r = B.rec[j];
    const float2 dz = B.dz[j];
    const uint32_t cells = __float_as_uint(r.w), lL = cells & 0xFFFFu, lR = cells >> 16;
    if (OPEN && M::kPlain && lR == kNoCell) return false;  // an open mesh's boundary edges: after the loop
    const float4 L = B.V[lL];
    float w0 = 0.0f, w1 = 0.0f, w2 = 0.0f, w3 = 0.0f, w4 = 0.0f, w5 = 0.0f;
    bool wall = false;
    float4 R = L;
    if (lR != kNoCell) {
        R = B.V[lR];
    } else {  // a boundary edge, in the block of its left cell: the state beyond it needs the momenta
        wall = true;
        const uint32_t c = it.b * kBlockCells + lL;
        const float hu = STAGE ? s.hu1[c] : s.hu[c], hv = STAGE ? s.hv1[c] : s.hv[c];
        if (OPEN) {
            const int cR = m.tile_cr[it.e0 + j];
            uint32_t kind = kOpenWall;
            float value = 0.0f, hG, huG, hvG;
            boundary_state(m, p, cR, L.x, hu, hv, r.x, r.y, hG, huG, hvG, kind, value);
            if (!(L.x < p.dry_tol && hG < p.dry_tol) || open_forced(kind, value)) {
                if (!edge_words<true, M>(p, cR, r.x, r.y, r.z, dz.x, dz.y, L.x, hu, hv, hG, huG, hvG, w0, w1, w2, w3, w4,
                                         w5, kind, value))
                    return false;
                if (cR < -1) tally_open(s.open_vol, static_cast<uint32_t>(-2 - cR), (0.5f * dt) * w0);
            }
        } else {
            float huR, hvR;
            wall_mirror(hu, hv, r.x, r.y, huR, hvR);
            const float twice = 2.0f * L.x;
            R.y = twice * huR * L.w;
            R.z = twice * hvR * L.w;
            if (!(L.x > p.dry_tol)) R.y = R.z = 0.0f;
        }
    }
    if (!(OPEN && wall) && !(L.x < p.dry_tol && R.x < p.dry_tol)) {
        FaceFlux f = face_flux_from_vel<M, true>(p, r.x, r.y, dz, pr(L.x, R.x), pr(L.y, R.y), pr(L.z, R.z),
                                                    pr(L.w, R.w));
        if (!f.plain) return false;
        if (wall) f.Fh = 0.0f;  // a wall passes no mass
        flux_words(p, r.x, r.y, r.z, pr(L.x, R.x), f.hs, f.Fh, f.Fhn, f.Fht, f.smax, w0, w1, w2, w3, w4, w5);
    }
    B.rec[j] = make_float4(w0, w1, w2, w5);
    B.dz[j] = make_float2(w3, w4);
    return true;
}

// The fluxes of the block's records (all threads; records and velocities are in shared memory). odd: a cell is out
// of the branch-free operations' range (plain_cell), so every edge takes the IEEE ones; else those edges
// whose numerators are, once more after the loop. again: a zeroed word per thread in shared memory (not a
// register of the loop).
template <int STAGE, bool OPEN>
__device__ __forceinline__ void block_fluxes(const swe_mesh_t &m, const swe_state_t &s, const Phys &p,
                                             const BlockItem &it, const BlockBuf &B, float dt, bool odd,
                                             uint32_t *again) {
    const uint32_t tid = threadIdx.x;
    if (!odd) {
        for (uint32_t j = tid; j < it.ne; j += kThreads)
            if (!block_edge<STAGE, OPEN, PlainOps>(m, s, p, it, B, j, dt)) again[tid] |= 1u << (j / kThreads);
    } else {
        again[tid] = 0xFFFFFFFFu;
    }
    uint32_t rounds = again[tid];  // at most 32: the launch refuses larger blocks
    if (rounds) {
        again[tid] = 0u;
        for (; rounds; rounds &= rounds - 1u) {
            const uint32_t j = tid + (__ffs(rounds) - 1) * kThreads;
            if (j < it.ne) block_edge<STAGE, OPEN, IeeeOps>(m, s, p, it, B, j, dt);
        }
    }
}

// Gather and update of the block's cells (all threads, after a barrier). In the corrector the block's
// results come back: whether a cell is wet and the CFL minimum, valid in warp 0.
template <int STAGE, bool COMP, bool CLAMP>
__device__ __forceinline__ void block_update(const swe_mesh_t &m, const swe_state_t &s, const Phys &p, float cfl,
                                             const BlockItem &it, const BlockBuf &B, float dt, uint32_t *red,
                                             bool &any_wet, uint32_t &bmin) {
    const uint32_t tid = threadIdx.x;
    bool wet = false;
    uint32_t bound = kNoBound;
    if (tid < it.cells) {
        const uint32_t i = it.b * kBlockCells + tid;
        float sdh = 0.0f, sdhu = 0.0f, sdhv = 0.0f, lam = 0.0f;
        const uint32_t q0 = B.cptr[tid] - B.cptr[0], q1 = B.cptr[tid + 1] - B.cptr[0];
        for (uint32_t q = q0; q < q1; ++q) {
            const uint32_t v = B.lcsr[q], j = v >> 1;
            const float4 A = B.rec[j];
            const float2 D = B.dz[j];
            const bool right = (v & 1u) != 0u;
            sdh += right ? -A.x : A.x;
            sdhu += right ? -D.x : A.y;
            sdhv += right ? -D.y : A.z;
            if (STAGE == 1) lam += A.w;
        }
        const float hui = STAGE ? s.hu1[i] : s.hu[i], hvi = STAGE ? s.hv1[i] : s.hv[i];
        const float loi = COMP ? (STAGE ? s.h1_lo[i] : s.h_lo[i]) : 0.0f;
        const float h0 = STAGE ? s.h[i] : 0.0f, hu0 = STAGE ? s.hu[i] : 0.0f, hv0 = STAGE ? s.hv[i] : 0.0f;
        const float lo0 = (STAGE && COMP) ? s.h_lo[i] : 0.0f;
        update_cell<STAGE, COMP, CLAMP>(s, p, cfl, dt, i, m.area[i], m.n_mann[i], B.V[tid].x, hui, hvi, loi, h0, hu0,
                                        hv0, lo0, sdh, sdhu, sdhv, lam, wet, bound);
    }
    if (STAGE == 1) tile_outcome(wet, bound, red, any_wet, bmin);
}

inline size_t block_bytes(const swe_mesh_t *m, const swe_blocks_t *k) {
    return block_plan(m->max_tile_edges, k->max_halo, m->max_blk_slots).total;
}

}  // namespace swe
