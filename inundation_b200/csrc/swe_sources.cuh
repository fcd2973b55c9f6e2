// Sparse sources as device functions over a strided range of sources, shared
// by the source kernels and the persistent step kernel.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "swe_common.cuh"

namespace swe {

// ---------------------------------------------------------------------------
// Sparse sources (resident.py:665-733): all increments, then the bounds.
// A source with a hydrograph adds hscale times the hydrograph's value at the
// start of its instance's step to its rate: t = now_ticks / 2^20 s rounded to
// float, piecewise linear between the knots, the end values outside them.
// (The reference's inflows are constant per phase; this is the product's own
// interpolation, restated by the oracle.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float hydrograph_at(const swe_sources_t &src, uint32_t j, float t) {
    const uint32_t k0 = src.knot_ptr[j], k1 = src.knot_ptr[j + 1];
    if (k1 <= k0) return 0.0f;
    if (!(t > src.knot_t[k0])) return src.knot_q[k0];
    if (!(t < src.knot_t[k1 - 1])) return src.knot_q[k1 - 1];
    uint32_t k = k0;
    while (k + 2 < k1 && !(t < src.knot_t[k + 1])) ++k;
    const float t0 = src.knot_t[k], t1 = src.knot_t[k + 1];
    const float q0 = src.knot_q[k], q1 = src.knot_q[k + 1];
    return q0 + (q1 - q0) * ((t - t0) / (t1 - t0));
}

__device__ __forceinline__ float clock_seconds(const swe_ctrl_t *c) {
    return static_cast<float>(c->now_ticks) * (1.0f / kTicksPerSecond);
}

// Sources that the persistent kernel's CTAs add with their tiles: at most four list entries per thread and tile, read
// from L1. Past it every source is a thread's of a grid-wide pass, which needs a barrier, and marks its two-ring one block
// after the other. A step of 30k cells with 1024 sources against 1025: 18.5 and 32.5 us (260k cells: 54 and 73 us).
constexpr uint32_t kFusedSources = 1024;

// Sources whose CFL bounds the step control's CTA takes, in the persistent and the dense kernel. It has 32 groups of
// eight lanes, and a round of them is a chain of five dependent loads, some 3 us, that the whole grid waits for; a
// grid-wide pass costs one barrier and one such chain. A persistent step of 30k cells with 64 sources: 15.0 us by the
// CTA, with 65 17.7 us by the pass (with 256 and 1024: 25.6 and 65 us by the CTA, 18.2 and 18.5 by the pass); a dense
// step of 260k cells: 64 24.9 us, 65 24.4 us (1024: 78 us by the CTA, 27 by the pass).
constexpr uint32_t kCtaBounds = 64;

// Source k's increment of cell i (of an instance whose step is dt), into the committed depth; keep != nullptr:
// the cell's h also goes to keep[0] and its low word to keep[3 x 64] (a tile's state held in shared memory).
// Returns whether the cell is wet after it.
__device__ __forceinline__ bool source_add(const swe_state_t &s, const swe_sources_t &src, uint32_t k, uint32_t i,
                                           uint32_t inst, float dt, float dry_tol, int comp, float *keep = nullptr) {
    float rate = src.rate[k];
    if (src.hydro && src.hydro[k] != 0xFFFFFFFFu)
        rate = rate + src.hscale[k] * hydrograph_at(src, src.hydro[k], clock_seconds(s.ctrl + inst));
    const float inc = dt * rate;
    float h_new;
    if (comp) {
        float lo_new;
        add_compensated(s.h[i], s.h_lo[i], inc, h_new, lo_new);
        s.h_lo[i] = lo_new;
        if (keep) keep[3 * kTileCells] = lo_new;
    } else {
        h_new = gmax(s.h[i] + inc, 0.0f);
    }
    s.h[i] = h_new;
    if (keep) keep[0] = h_new;
    return h_new >= dry_tol;
}

__device__ __forceinline__ void source_apply(const swe_mesh_t &m, const swe_state_t &s, const swe_sources_t &src,
                                             float dry_tol, int comp, uint32_t first, uint32_t stride) {
    for (uint32_t k = first; k < src.count; k += stride) {
        const uint32_t i = src.cells[k];
        const uint32_t inst = m.block_inst[i >> 8];
        const uint32_t dt_bits = s.dt_buf[kDtWords * inst];
        if (dt_bits == 0u) continue;
        if (source_add(s, src, k, i, inst, __uint_as_float(dt_bits), dry_tol, comp))
            s.blk[kBlkWords * (i >> 8) + kBlkWet] = 1u;
    }
}

// One instance's CFL bound from a warp: every lane's (inst, bound), kNoBound for
// none. A warp whose bounds all belong to one instance sends one atomic minimum;
// otherwise every lane sends its own. Called by all 32 lanes.
__device__ __forceinline__ void bound_flush_warp(const swe_state_t &s, uint32_t inst, uint32_t bound) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const bool has = bound != kNoBound;
    const unsigned with = __ballot_sync(kFull, has);
    if (!with) return;
    const int leader = __ffs(with) - 1;
    const uint32_t ref = __shfl_sync(kFull, inst, leader);
    if (__all_sync(kFull, !has || inst == ref)) {
        const uint32_t low = __reduce_min_sync(kFull, bound);
        if (static_cast<int>(threadIdx.x & 31u) == leader) atomicMin(&s.dt_buf[kDtWords * ref + 1], low);
    } else if (has) {
        atomicMin(&s.dt_buf[kDtWords * inst + 1], bound);
    }
}

// The post-source CFL bounds: each thread keeps the minimum of its sources'
// bounds while they belong to one instance, and the warp combines them at the
// end, so the dt word sees few atomics however many sources there are (a
// minimum is the same in any order). Called by every thread of whole warps.
__device__ __forceinline__ void source_bound(const swe_mesh_t &m, const swe_state_t &s, const swe_sources_t &src,
                                             const Phys &p, float cfl, uint32_t first, uint32_t stride) {
    uint32_t acc_inst = 0u, acc = kNoBound;
    for (uint32_t k = first; k < src.count; k += stride) {
        const uint32_t i = src.cells[k];
        const uint32_t inst = m.block_inst[i >> 8];
        if (s.dt_buf[kDtWords * inst] == 0u) continue;
        const float h_new = s.h[i];
        if (!(h_new >= p.dry_tol)) continue;
        const float u = sqrtf(s.hu[i] * s.hu[i] + s.hv[i] * s.hv[i]) / h_new;
        const float c = sqrtf(p.g * h_new);
        const uint32_t base = m.tile_ptr[i >> 8];
        float lam = 0.0f;
        for (uint32_t q = m.cptr[i]; q < m.cptr[i + 1]; ++q) {
            const uint32_t v = m.lcsr[q];
            const uint32_t e = base + (v >> 1);
            const int nb = (v & 1u) ? m.tile_cl[e] : m.tile_cr[e];
            const bool dry_side = nb >= 0 && s.h[nb] < p.dry_tol;
            lam += (u + (dry_side ? 2.0f : 1.0f) * c) * m.tile_len[e];
        }
        const float A = m.area[i];
        if (!(lam > 1e-30f && A > 1e-10f)) continue;
        const uint32_t b = __float_as_uint(cfl * A / lam);
        if (inst != acc_inst && acc != kNoBound) {
            atomicMin(&s.dt_buf[kDtWords * acc_inst + 1], acc);
            acc = kNoBound;
        }
        acc_inst = inst;
        acc = min(acc, b);
    }
    bound_flush_warp(s, acc_inst, acc);
}

// The post-source CFL bounds of a few sources by one CTA, eight lanes per source, one
// CSR slot per lane: the slots' loads are in flight together, and the lanes' terms are
// added in slot order, so the sums are source_bound's bit for bit. All threads.
__device__ __forceinline__ void source_bound_cta(const swe_mesh_t &m, const swe_state_t &s, const swe_sources_t &src,
                                                 const Phys &p, float cfl) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const uint32_t sub = threadIdx.x & 7u, groups = blockDim.x >> 3;
    for (uint32_t k0 = 0; k0 < src.count; k0 += groups) {
        const uint32_t k = k0 + (threadIdx.x >> 3);
        bool run = k < src.count;
        uint32_t i = 0u, inst = 0u, base = 0u, q = 0u, q1 = 0u;
        float h = 0.0f, hu = 0.0f, hv = 0.0f, A = 0.0f;
        if (run) {
            i = __ldg(src.cells + k);
            inst = m.block_inst[i >> 8];
            base = m.tile_ptr[i >> 8];
            q = m.cptr[i];
            q1 = m.cptr[i + 1];
            A = m.area[i];
            h = s.h[i];
            hu = s.hu[i];
            hv = s.hv[i];
            run = s.dt_buf[kDtWords * inst] != 0u && h >= p.dry_tol;
        }
        float u = 0.0f, c = 0.0f;
        if (run) {
            u = sqrtf(hu * hu + hv * hv) / h;
            c = sqrtf(p.g * h);
        }
        float lam = 0.0f;
        while (__any_sync(kFull, run && q < q1)) {
            float term = 0.0f;
            if (run && q + sub < q1) {
                const uint32_t v = m.lcsr[q + sub];
                const uint32_t e = base + (v >> 1);
                const int nb = (v & 1u) ? m.tile_cl[e] : m.tile_cr[e];
                const bool dry_side = nb >= 0 && s.h[nb] < p.dry_tol;
                term = (u + (dry_side ? 2.0f : 1.0f) * c) * m.tile_len[e];
            }
            for (int l = 0; l < 8; ++l) {
                const float t = __shfl_sync(kFull, term, l, 8);
                if (q + l < q1) lam += t;
            }
            q += 8u;
        }
        uint32_t bound = kNoBound;
        if (run && sub == 0u && lam > 1e-30f && A > 1e-10f) bound = __float_as_uint(cfl * A / lam);
        bound_flush_warp(s, inst, bound);
    }
}

}  // namespace swe
