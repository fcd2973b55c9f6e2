// Whole steps of a mesh with many active blocks in one cooperative launch.
//
// The stages take a 256-cell block at a time from packed records (swe_block.cuh).
// What one launch for all steps saves against three launches a step (two stages and
// the dilation):
//   * the dilation: before its predictor a block looks at the wet flags of its own
//     two-ring, which the last corrector (and sources) left, while the block before it is staged;
//   * launch gaps and ramps: the phases are separated by grid barriers, the records and
//     CSR of a CTA's first block, which no step changes, are copied while the CTA waits
//     at the barrier, and the first block's predictor needs its dt only after its
//     fluxes (the step control publishes it after the release, as in swe_persist.cu);
//   * the steps after the last instance's window is done, and the capture of a graph.
// The predictor's CTAs go through the blocks in the order the last dilation left, the
// blocks that were active first: CTA k starts with the k-th and takes further ones from a
// counter, so that the active blocks spread evenly over the SMs, wherever they lie, and every
// CTA ends within about a block of the others; its corrector repeats the blocks it took.
// Sources come by block: a block's are added right after its corrector's update. Those of
// inactive blocks wait for one more barrier, in the steps that have any. The CFL bounds of up
// to kCtaBounds sources are taken by the step control's CTA; those of more by a pass over all of them
// after a barrier, which looks only at the cells whose bound can be below the smallest one so far:
// a source's wave speeds are at most u + 2c on its whole perimeter.
// Bound: issue and the waits at CTA barriers. Over a launch of 20 steps of a million wet cells 63 % of the issue slots
// are used, and of the 12.7 cycles between two instructions of a warp 3.4 are waits at a CTA barrier (three or four a
// block, one buffer per CTA), 2.1 for loads, 1.7 fixed latencies and 1.5 not selected; DRAM moves 285 B per cell and
// step, 33 % of the copy bandwidth. One step: 600k cells all wet 81 us, 260k cells 44 % active 21.5 us (as two staged
// stage kernels and a dilation 105 and 33.5 us). With blocks dealt to CTAs in turn instead of taken, a phase of the
// first waits 15 us for its last CTA (49 us instead of 41.7), and one of the second takes 16 us instead of 13.
//
// Every barrier and staged-data wait is bounded, as in the other kernels. The results
// are the other kernels' bit for bit: the same expressions, the same blocks active.
#include <cuda_runtime.h>

#include <cstdint>

#include "swe_block.cuh"
#include "swe_grid.cuh"
#include "swe_sources.cuh"

namespace swe {

// CTAs an SM must hold: with 4, 64 registers a thread and no spills (600k cells all wet 80.7 us a step, 260k cells
// 44 % active 21.2); with 5, 48 registers (82.7 and 22.5); with 6 they spill.
constexpr int kDenseMinCtas = 4;

constexpr uint32_t kNoBlock = 0xFFFFFFFFu;
constexpr uint32_t kTakenCap = 512;  // blocks a CTA computes besides its first in one step

struct DenseShared {
    BlockItem first;    // the CTA's first block; its dt is this step's, 0 when it is not computed
    BlockItem next[2];
    uint32_t taken[kTakenCap];  // the blocks computed besides the first in this step
    uint32_t n_taken;
    uint32_t candidate;  // the block to look at next (kNoBlock: none left)
    uint32_t odd;       // a cell of the block is out of the branch-free operations' range
    uint32_t again[kThreads];  // block_fluxes
    uint32_t active;    // the first block is active this step
    uint32_t red[2 * kThreads / 32];
    int flag[3];
    uint32_t epoch0;
};

// What a phase leaves for the next: whether the first block's records are (being) staged.
struct DenseStage {
    uint32_t phase;  // parity of the next completion
    bool in_flight;  // copies of the first block's records were issued and not yet waited for
    bool staged;     // they have arrived and are whole
};

// Whether block b is active in the coming step (one warp): a wet or forced block in its two-ring.
__device__ __forceinline__ bool block_pull(const swe_mesh_t &m, const swe_state_t &s, uint32_t b, bool all_active) {
    if (all_active) return true;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t v = 0u;
    if (lane == 0) v = s.blk[kBlkWords * b + kBlkWet] | s.blk[kBlkWords * b + kBlkForced];
    for (uint32_t k = m.ring_ptr[b] + lane, k1 = m.ring_ptr[b + 1]; k < k1; k += 32u) {
        const uint32_t nb = m.ring_idx[k];
        v |= s.blk[kBlkWords * nb + kBlkWet] | s.blk[kBlkWords * nb + kBlkForced];
    }
    return __any_sync(0xFFFFFFFFu, v != 0u);
}

// This step's dt of an instance, as the predictor reads it: published after the last barrier's release.
__device__ __forceinline__ uint32_t dense_dt(const swe_state_t &s, uint32_t inst, uint32_t step, uint32_t epoch) {
    if (step == 0u) return s.dt_buf[kDtWords * inst];
    const uint64_t *pair = dt_pair(s, inst);
    return published_dt(s, pair, epoch, ld_relaxed_u64(pair));
}

// The next block off the predictor's counter (one thread), or kNoBlock.
__device__ __forceinline__ uint32_t take_block(const swe_mesh_t &m, const swe_state_t &s) {
    const uint32_t k = gridDim.x + atomicAdd(&s.sched[kSchedTake], 1u);
    return k < m.n_blocks ? s.active_list[m.n_blocks + k] : kNoBlock;
}

// Block b's active flag in the predictor (one thread), and word that an inactive block has sources.
__device__ __forceinline__ void keep_active(const swe_blocks_t &blocks, const swe_state_t &s, uint32_t b, bool active,
                                            uint32_t epoch) {
    s.blk[kBlkWords * b + kBlkActive] = active ? 1u : 0u;
    if (!active && blocks.src_ptr && blocks.src_ptr[b + 1] != blocks.src_ptr[b]) s.sched[kSchedSrcOut] = epoch;
}

// source_bound over many sources, evaluated only where the bound can be below its instance's smallest so
// far (which another thread may lower meanwhile: an older value only prunes less). The margin in perim
// covers the rounding of the sum over the edges.
__device__ __forceinline__ void source_bound_pruned(const swe_mesh_t &m, const swe_blocks_t &blocks,
                                                    const swe_state_t &s, const swe_sources_t &src, const Phys &p,
                                                    float cfl, uint32_t first, uint32_t stride) {
    for (uint32_t k = first; k < src.count; k += stride) {
        const uint32_t i = src.cells[k], inst = m.block_inst[i >> 8];
        const uint32_t *dtw = s.dt_buf + kDtWords * inst;
        const float h = s.h[i], hu = s.hu[i], hv = s.hv[i], A = m.area[i], around = blocks.perim[i];
        if (dtw[0] == 0u || !(h >= p.dry_tol)) continue;
        const float u = sqrtf(hu * hu + hv * hv) / h;
        const float c = sqrtf(p.g * h);
        if (__float_as_uint(cfl * A / ((u + 2.0f * c) * around)) >= dtw[1]) continue;  // NaN: no bound either
        const uint32_t base = m.tile_ptr[i >> 8];
        float lam = 0.0f;
        for (uint32_t q = m.cptr[i], q1 = m.cptr[i + 1]; q < q1; ++q) {
            const uint32_t v = m.lcsr[q];
            const uint32_t e = base + (v >> 1);
            const int nb = (v & 1u) ? m.tile_cl[e] : m.tile_cr[e];
            const bool dry_side = nb >= 0 && s.h[nb] < p.dry_tol;
            lam += (u + (dry_side ? 2.0f : 1.0f) * c) * m.tile_len[e];
        }
        if (lam > 1e-30f && A > 1e-10f) atomicMin(&s.dt_buf[kDtWords * inst + 1], __float_as_uint(cfl * A / lam));
    }
}

// The predictor's next block into `out` (one warp): candidates are looked at, and their active flags
// kept, until one is active; the candidate after it is taken while they are. with_dt: its dt too
// (else, before the dt is published, 0 for now).
__device__ __forceinline__ void next_predicted(const swe_mesh_t &m, const swe_blocks_t &blocks, const swe_state_t &s,
                                               DenseShared &sh, uint32_t step, uint32_t epoch, bool all_active,
                                               bool with_dt, BlockItem *out) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t c = sh.candidate, n = sh.n_taken;
    for (;;) {
        if (c == kNoBlock || n >= kTakenCap) {  // the other CTAs have room for what is left
            if (lane == 0) out->b = kNoBlock;
            return;
        }
        uint32_t after = 0u;
        if (lane == 0) after = n + 1u < kTakenCap ? take_block(m, s) : kNoBlock;
        const uint32_t inst = m.block_inst[c];
        const bool active = block_pull(m, s, c, all_active);
        if (lane == 0) {
            keep_active(blocks, s, c, active, epoch);
            if (active) {
                *out = block_item(m, blocks, c, inst, with_dt ? dense_dt(s, inst, step, epoch) : 0u);
                sh.taken[n] = c;
                sh.n_taken = n + 1u;
                sh.candidate = after;
            }
        }
        if (active) return;
        c = __shfl_sync(0xFFFFFFFFu, after, 0);
    }
}

// Waits for staged records; on a timeout records error 1 and gives the copies one more bounded wait.
__device__ __forceinline__ bool dense_wait(const swe_state_t &s, const BlockBuf &B, DenseStage &st) {
    const bool ok = mbar_wait(B.bar, st.phase);
    st.phase ^= 1u;
    if (__syncthreads_and(ok)) return true;
    if (threadIdx.x == 0) atomicOr(&s.ctrl->error, 1u);
    mbar_wait(B.bar, st.phase ^ 1u);
    return false;
}

// One stage over this CTA's blocks. Ends with the first block's records on their way for the next phase.
template <int STAGE, bool COMP, bool CLAMP, bool OPEN>
__device__ bool dense_phase(const swe_mesh_t &m, const swe_blocks_t &blocks, const swe_state_t &s, const Phys &p,
                            float cfl, const BlockBuf &B, DenseShared &sh, DenseStage &st, uint64_t &computed,
                            uint32_t step, uint32_t epoch, bool all_active, const swe_sources_t &src) {
    const uint32_t tid = threadIdx.x;
    const bool last_warp = tid >= kThreads - 32u;
    const BlockItem *it = &sh.first;
    for (uint32_t w = 0;; ++w) {
        const bool first = w == 0u;
        BlockItem *next = &sh.next[w & 1u];
        // The predictor starts its first block before its activity and dt are known.
        const bool early = STAGE == 0 && first;
        bool go = early || it->dt != 0u;
        if (go) {
            if (!(first && (st.in_flight || st.staged))) {
                if (tid < 32u) block_issue(m, blocks, *it, B);
                st.in_flight = true;
            }
            if (early && tid >= 32u && tid < 64u) {
                const bool active = block_pull(m, s, it->b, all_active);
                if (tid == 32u) {
                    sh.active = active ? 1u : 0u;
                    keep_active(blocks, s, it->b, active, epoch);
                    // an open mesh's volume tallies need dt with the fluxes
                    if (OPEN) sh.first.dt = active ? dense_dt(s, it->inst, step, epoch) : 0u;
                }
            }
            block_velocities<STAGE>(blocks, s, p, *it, B, &sh.odd);
        }
        // the last warp finds the next block while this one's records arrive
        if (last_warp) {
            if (STAGE == 0) {
                if (first && tid == kThreads - 32u) {
                    sh.n_taken = 0u;
                    sh.candidate = take_block(m, s);
                }
                __syncwarp();
                next_predicted(m, blocks, s, sh, step, epoch, all_active, !first, next);
            } else if (tid == kThreads - 32u) {
                if (w < sh.n_taken) {
                    const uint32_t b = sh.taken[w], inst = m.block_inst[b];
                    *next = block_item(m, blocks, b, inst, s.dt_buf[kDtWords * inst]);
                } else {
                    next->b = kNoBlock;
                }
            }
        }
        if (st.in_flight) {
            st.in_flight = false;
            if (!dense_wait(s, B, st)) return false;
            st.staged = first;
        }
        if (early) {
            __syncthreads();  // the first block may have been staged before
            go = sh.active != 0u && !(OPEN && sh.first.dt == 0u);
        }
        if (go) {
            st.staged = false;  // the words go over the records
            block_fluxes<STAGE, OPEN>(m, s, p, *it, B, __uint_as_float(it->dt), sh.odd != 0u, sh.again);
        }
        if (early && tid == kThreads - 32u) {  // in the last warp, which has the fewest records
            if (!OPEN) sh.first.dt = go ? dense_dt(s, it->inst, step, epoch) : 0u;
            if (next->b != kNoBlock) next->dt = dense_dt(s, next->inst, step, epoch);
        }
        __syncthreads();
        const uint32_t dt_bits = go ? it->dt : 0u;
        if (dt_bits != 0u) {
            const float dt = __uint_as_float(dt_bits);
            bool any_wet;
            uint32_t bmin;
            block_update<STAGE, COMP, CLAMP>(m, s, p, cfl, *it, B, dt, sh.red, any_wet, bmin);
            if (STAGE == 1) {
                bool wet_sources = false;
                if (it->ns) {
                    for (uint32_t k = tid; k < it->ns; k += kThreads)
                        wet_sources |= source_add(s, src, it->s0 + k, src.cells[it->s0 + k], it->inst, dt, p.dry_tol, COMP);
                    wet_sources = __syncthreads_or(wet_sources) != 0;
                }
                if (tid == 0) {
                    s.blk[kBlkWords * it->b + kBlkWet] = (any_wet || wet_sources) ? 1u : 0u;
                    if (bmin != kNoBound) atomicMin(&s.dt_buf[kDtWords * it->inst + 1], bmin);
                    computed += it->cells;
                }
            }
        } else if (early && !go && tid == 0) {
            sh.first.dt = 0u;
        }
        if (tid == 0) sh.odd = 0u;
        // the shared memory is refilled by bulk copies
        fence_proxy_async();
        __syncthreads();
        it = next;
        if (it->b == kNoBlock) break;
        st.staged = false;
    }
    if (!st.staged) {
        if (tid < 32u) block_issue(m, blocks, sh.first, B);
        st.in_flight = true;
    }
    return true;
}

template <bool COMP, bool CLAMP, bool OPEN>
__global__ void __launch_bounds__(kThreads, kDenseMinCtas)
    dense_steps_kernel(swe_mesh_t m, swe_blocks_t blocks, swe_state_t s, swe_sources_t src, Phys p, float cfl, int all_active,
                       uint32_t n_steps) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ DenseShared sh;
    const BlockBuf B = block_buf(smem, block_plan(m.max_tile_edges, blocks.max_halo, m.max_blk_slots));
    CountSync g{s.sync, 0u};  // the launch zeroes the counter before the kernel starts
    const uint32_t tid = threadIdx.x;
    sh.again[tid] = 0u;
    if (tid == 0) {
        sh.odd = 0u;
        mbar_init(B.bar, 1u);
        fence_barrier_init();
        sh.epoch0 = *reinterpret_cast<volatile uint32_t *>(s.sched + kSchedEpoch);  // before any CTA's first barrier
        const uint32_t b = s.active_list[m.n_blocks + blockIdx.x];  // no more CTAs than blocks
        sh.first = block_item(m, blocks, b, m.block_inst[b], 0u);
    }
    if (blockIdx.x == 0)  // no published dt pair of an earlier run or launch carries an epoch of this one
        for (uint32_t i = tid; i < m.n_inst; i += kThreads) *const_cast<uint64_t *>(dt_pair(s, i)) = 0ull;
    __syncthreads();
    const uint32_t first = blockIdx.x * kThreads + tid, stride = gridDim.x * kThreads;
    const bool all = all_active != 0;
    auto nothing = [] {};
    DenseStage st{0u, false, false};
    uint64_t computed = 0;
    bool ok = true;
    for (uint32_t step = 0; step < n_steps; ++step) {
        const uint32_t epoch = sh.epoch0 + step + 1u, next_epoch = epoch + 1u;
        if (!(ok = dense_phase<0, COMP, CLAMP, OPEN>(m, blocks, s, p, cfl, B, sh, st, computed, step, epoch, all, src)))
            break;
        if (!(ok = count_sync(g, sh.flag, nothing))) break;
        // the predictor's counter, whose phase is over, for the next step
        if (blockIdx.x == 0 && tid == 0) s.sched[kSchedTake] = 0u;
        if (!(ok = dense_phase<1, COMP, CLAMP, OPEN>(m, blocks, s, p, cfl, B, sh, st, computed, step, epoch, all, src)))
            break;
        if (src.count && *reinterpret_cast<volatile uint32_t *>(s.sched + kSchedSrcOut) == epoch) {
            // blocks found inactive have sources, on cells whose depth neighbouring correctors read
            if (!(ok = count_sync(g, sh.flag, nothing))) break;
            for (uint32_t b = blockIdx.x; b < m.n_blocks; b += gridDim.x) {
                const uint32_t inst = m.block_inst[b], dt = s.dt_buf[kDtWords * inst];
                if (dt == 0u || block_active(s.blk, b)) continue;
                for (uint32_t k = blocks.src_ptr[b] + tid; k < blocks.src_ptr[b + 1]; k += kThreads)
                    if (source_add(s, src, k, src.cells[k], inst, __uint_as_float(dt), p.dry_tol, COMP))
                        s.blk[kBlkWords * b + kBlkWet] = 1u;
            }
        }
        if (src.count > kCtaBounds) {
            if (!(ok = count_sync(g, sh.flag, nothing))) break;
            source_bound_pruned(m, blocks, s, src, p, cfl, first, stride);
        }
        auto control = [&] {
            if (src.count && src.count <= kCtaBounds) {
                source_bound_cta(m, s, src, p, cfl);
                __syncthreads();  // the bounds land before step_control reads them
            }
            bool runs = false;
            for (uint32_t i = tid; i < m.n_inst; i += kThreads) {
                const uint32_t dt = step_control(s.ctrl + i, s.dt_buf + kDtWords * i, 1);
                runs |= dt != 0u;
                st_relaxed_u64(const_cast<uint64_t *>(dt_pair(s, i)), (static_cast<uint64_t>(next_epoch) << 32) | dt);
            }
            const bool done = __syncthreads_or(runs) == 0;
            if (tid == 0) {
                volatile uint32_t *sched = s.sched;
                sched[kSchedEpoch] = next_epoch;
                if (done) sched[kSchedIdle] = next_epoch;
            }
        };
        if (!(ok = count_sync(g, sh.flag, control, s.sched + kSchedIdle))) break;
        // no instance ran this step: the steps left do nothing either (see persistent_steps_kernel)
        if (static_cast<uint32_t>(sh.flag[2]) == epoch) break;
    }
    if (st.in_flight) mbar_wait(B.bar, st.phase);
    if (tid == 0) {
        if (!ok) atomicOr(&s.ctrl->error, 2u);
        if (computed) atomicAdd(reinterpret_cast<unsigned long long *>(s.sched + kSchedComputed), computed);
    }
}

int launch_handover(const swe_mesh_t *m, const swe_state_t *s, const swe_params_t *p, cudaStream_t st);  // swe_control.cu

template <bool COMP, bool CLAMP, bool OPEN>
int launch_dense(const swe_mesh_t *m, const swe_blocks_t *k, const swe_state_t *s, const swe_params_t *p,
                 const swe_sources_t *src, uint32_t n_steps, cudaStream_t st) {
    auto kern = dense_steps_kernel<COMP, CLAMP, OPEN>;
    const size_t bytes = block_bytes(m, k);
    int rc = set_smem(kern, bytes);
    if (rc) return rc;
    int per_sm = 0, dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, bytes) != cudaSuccess)
        return SWE_ERR_CUDA;
    if (per_sm < 1) return SWE_ERR_TOO_LARGE;
    const uint32_t fit = min(static_cast<uint32_t>(per_sm) * static_cast<uint32_t>(sms), m->n_blocks);
    const uint32_t grid = (p->grid == 0u || p->grid > fit) ? fit : p->grid;
    // the barrier's arrival counter (at most four barriers a step) stays below 2^32
    if (4ull * n_steps * grid >= (1ull << 32)) return SWE_ERR_TOO_LARGE;
    Phys ph = make_phys(p->g, p->dry_tol);
    float cfl = p->cfl;
    int all_active = p->active_set ? 0 : 1;
    swe_mesh_t mm = *m;
    swe_blocks_t bb = *k;
    swe_state_t ss = *s;
    swe_sources_t sc = *src;
    void *args[] = {&mm, &bb, &ss, &sc, &ph, &cfl, &all_active, &n_steps};
    // every block of a step must find a CTA (one with room for its last block may meet an inactive one there and stop)
    if (m->n_blocks > static_cast<uint64_t>(grid) * kTakenCap) return SWE_ERR_TOO_LARGE;
    if (cudaMemsetAsync(s->sync, 0, sizeof(uint32_t), st) != cudaSuccess) return SWE_ERR_CUDA;
    // the counter of taken blocks, and words that carry no epoch of this launch
    if (cudaMemsetAsync(s->sched + kSchedTake, 0, sizeof(uint32_t), st) != cudaSuccess ||
        cudaMemsetAsync(s->sched + kSchedIdle, 0, 2 * sizeof(uint32_t), st) != cudaSuccess)
        return SWE_ERR_CUDA;
    if (cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kern), dim3(grid), dim3(kThreads), args, bytes, st) !=
        cudaSuccess)
        return SWE_ERR_CUDA;
    return launch_handover(m, s, p, st);
}

template <bool OPEN>
int dispatch_dense(const swe_mesh_t *m, const swe_blocks_t *k, const swe_state_t *s, const swe_params_t *p,
                   const swe_sources_t *src, uint32_t n_steps, cudaStream_t st) {
    if (p->compensated)
        return p->track_clamp ? launch_dense<true, true, OPEN>(m, k, s, p, src, n_steps, st)
                              : launch_dense<true, false, OPEN>(m, k, s, p, src, n_steps, st);
    return p->track_clamp ? launch_dense<false, true, OPEN>(m, k, s, p, src, n_steps, st)
                          : launch_dense<false, false, OPEN>(m, k, s, p, src, n_steps, st);
}

inline bool blocks_ok(const swe_mesh_t *m, const swe_blocks_t *k) {
    return k && k->rec && k->dz && k->halo && k->halo_ptr && k->perim && m->blk_lcsr && m->blk_lcsr_ptr;
}

}  // namespace swe

using namespace swe;

extern "C" {

int swe_configure_blocks(const swe_mesh_t *mesh, const swe_blocks_t *blocks, int *blocks_per_sm) {
    if (!mesh_ok(mesh) || !blocks_ok(mesh, blocks) || !blocks_per_sm) return SWE_ERR_ARGUMENT;
    *blocks_per_sm = 0;
    const size_t bytes = block_bytes(mesh, blocks);
    if (bytes > kMaxSmem || kBlockCells + blocks->max_halo >= kNoCell || mesh->max_tile_edges > 32u * kThreads)
        return SWE_OK;
    cudaFuncAttributes own;
    if (cudaFuncGetAttributes(&own, dense_steps_kernel<true, false, false>) != cudaSuccess) return SWE_ERR_CUDA;
    if (bytes + own.sharedSizeBytes > kMaxSmem) return SWE_OK;
    const int rc = set_smem(dense_steps_kernel<true, false, false>, bytes);
    if (rc) return rc;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, dense_steps_kernel<true, false, false>, kThreads,
                                                         bytes) == cudaSuccess
               ? SWE_OK
               : SWE_ERR_CUDA;
}

int swe_steps_blocks(const swe_mesh_t *mesh, const swe_blocks_t *blocks, const swe_state_t *state,
                     const swe_params_t *params, const swe_sources_t *sources, uint32_t n_steps, swe_stream_t stream) {
    if (!mesh_ok(mesh) || !blocks_ok(mesh, blocks) || !state_ok(state) || !open_ok(mesh, state) || !params ||
        !sources_ok(sources))
        return SWE_ERR_ARGUMENT;
    if (!state->sync || (reinterpret_cast<uintptr_t>(state->dt_buf) & 15u)) return SWE_ERR_ARGUMENT;
    if (sources->count && !blocks->src_ptr) return SWE_ERR_ARGUMENT;
    if (mesh->max_sub_edges > 2047u || mesh->max_sub_slots > 2047u || mesh->n_inst > 1023u ||
        mesh->n_blocks > (1u << 23) || kBlockCells + blocks->max_halo >= kNoCell ||
        mesh->max_tile_edges > 32u * kThreads)
        return SWE_ERR_TOO_LARGE;
    if (n_steps == 0u) return SWE_OK;
    return mesh->n_open ? dispatch_dense<true>(mesh, blocks, state, params, sources, n_steps, stream)
                        : dispatch_dense<false>(mesh, blocks, state, params, sources, n_steps, stream);
}

}  // extern "C"
