// track_kernel.cuh -- the tracking kernel (compiled by track_kernel.cu,
// track_kernel_plain.cu, track_kernel_map.cu and track_kernel_full.cu, one
// kind of lattice each).
//
// One thread per particle; the particle's state lives in registers for the
// whole call (all turns).  The compiled element stream is staged into shared
// memory chunk by chunk with cp.async.bulk (the TMA engine's 1-D bulk copy)
// completing on mbarriers; every warp reads the records as broadcasts and
// dispatches on the opcode with a warp-uniform switch.  A lattice that fits
// the shared-memory stages is loaded once and stays resident for all turns;
// a longer one streams through the stages with STAGES-1 chunks in flight.
//
// Loop semantics follow the reference exactly:
//   until-turn      common/track/track.h:610-670
//   line            common/track/track.h:779-822
//   elem-by-elem    common/track/track.h:672-777
// (at_element_id is start + element ordinal while inside a turn and reset at
// the turn end, a failing or lost particle freezes where it stopped, status
// is OR-accumulated, -1 on failure).
//
// These translation units are compiled with -fmad=false; the FAST
// instantiation uses explicit fma() (maps.cuh).
#pragma once

#include <cstdint>

#include "kernel_api.h"
#include "maps.cuh"

namespace stg {

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bulk (TMA) copy global -> shared, completion counted on `bar`.
// src and dst 16-byte aligned, bytes a multiple of 16 (chunks are).
__device__ __forceinline__ void bulk_copy_g2s(void *dst, const void *src, uint32_t bytes,
                                              uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Bounded wait: gives up after ~2^31 clock cycles (~1 s) instead of hanging.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity)
{
    long long const t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > (1ll << 31)) return false;
    }
    return true;
}

__device__ __forceinline__ void load_particle(PState &p, const uint64_t *cols, int64_t n,
                                              int64_t i)
{
    const double *d = reinterpret_cast<const double *>(cols);
    const int64_t *k = reinterpret_cast<const int64_t *>(cols);
    p.q0 = d[0 * n + i];
    p.mass0 = d[1 * n + i];
    p.beta0 = d[2 * n + i];
    p.gamma0 = d[3 * n + i];
    p.p0c = d[4 * n + i];
    p.s = d[5 * n + i];
    p.x = d[6 * n + i];
    p.y = d[7 * n + i];
    p.px = d[8 * n + i];
    p.py = d[9 * n + i];
    p.zeta = d[10 * n + i];
    p.psigma = d[11 * n + i];
    p.delta = d[12 * n + i];
    p.rpp = d[13 * n + i];
    p.rvv = d[14 * n + i];
    p.chi = d[15 * n + i];
    p.charge_ratio = d[16 * n + i];
    p.pid = k[17 * n + i];
    p.at_element = k[18 * n + i];
    p.at_turn = k[19 * n + i];
    p.state = k[20 * n + i];
    p.energy0 = sqrt(p.p0c * p.p0c + p.mass0 * p.mass0);
    refresh_kick_factors(p);
    p.lazy_s = false;
}

// Write one full record (21 columns) to a column block of capacity cap.
__device__ __forceinline__ void store_record(const PState &p, uint64_t *out, int64_t cap,
                                             int64_t j, int64_t at_element, int64_t at_turn,
                                             double s)
{
    double *d = reinterpret_cast<double *>(out);
    int64_t *k = reinterpret_cast<int64_t *>(out);
    d[0 * cap + j] = p.q0;
    d[1 * cap + j] = p.mass0;
    d[2 * cap + j] = p.beta0;
    d[3 * cap + j] = p.gamma0;
    d[4 * cap + j] = p.p0c;
    d[5 * cap + j] = s;
    d[6 * cap + j] = p.x;
    d[7 * cap + j] = p.y;
    d[8 * cap + j] = p.px;
    d[9 * cap + j] = p.py;
    d[10 * cap + j] = p.zeta;
    d[11 * cap + j] = p.psigma;
    d[12 * cap + j] = p.delta;
    d[13 * cap + j] = p.rpp;
    d[14 * cap + j] = p.rvv;
    d[15 * cap + j] = p.chi;
    d[16 * cap + j] = p.charge_ratio;
    k[17 * cap + j] = p.pid;
    k[18 * cap + j] = at_element;
    k[19 * cap + j] = at_turn;
    k[20 * cap + j] = p.state;
}

// be_monitor/track.h:48-110: output index for the current turn, or -1.
__device__ __forceinline__ int64_t monitor_index(const uint64_t *rec, int64_t turn, int64_t pid)
{
    int64_t const nstores = (int64_t)rec[1], start = (int64_t)rec[2], skip = (int64_t)rec[3];
    int64_t const max_pid = (int64_t)rec[4], min_pid = (int64_t)rec[5];
    int64_t const since = turn - start;
    int64_t out = -1;
    if (since >= 0 && (since % skip) == 0) {
        int64_t idx = since / skip;
        if (idx >= nstores && rec[6] != 0) idx = idx % nstores;
        if (idx < nstores) {
            int64_t const off = pid - min_pid;
            int64_t const np = max_pid - min_pid + 1;
            out = (rec[7] != 0) ? np * idx + off : off * np + idx;
        }
    }
    return out;
}

// output/elem_by_elem_config.h:667-763
__device__ __forceinline__ int64_t ebe_index(const EbeDevConfig &c, int64_t pid, int64_t elem,
                                             int64_t turn)
{
    int64_t out = -1;
    if (c.min_particle_id <= pid && c.max_particle_id >= pid && c.min_element_id <= elem &&
        c.max_element_id >= elem && c.min_turn <= turn &&
        (c.max_turn >= turn || c.is_rolling != 0)) {
        int64_t const np = c.num_particles_to_store, ne = c.num_elements_to_store;
        int64_t cap = 0;
        if (c.order == 0) {
            out = (turn - c.min_turn) * np * ne + (elem - c.min_element_id) * np +
                  (pid - c.min_particle_id);
            cap = np * ne * c.num_turns_to_store;
        }
        if (out >= cap && cap > 0 && c.is_rolling != 0) out = out % cap;
    }
    return out;
}

// What became of a particle in an element.
enum Passed : int { PASSED = 0, LOST = 1, FAILED = -1 };

// Apply one element.  FAILED is the reference's status -1; p.state is left
// as the reference's map leaves it.  The kinds other than KIND_FULL compile
// only the maps of kPlainOps; the host chooses them for lattices without any
// other opcode, so their fall-through (failure, particle lost, as for an
// unknown type id) is never taken.  Maps that cannot lose a particle return a
// constant, so the walk tests nothing after them.  OWN: drifts and multipoles
// are the walk's (own_loop).  EBE: the state need not be 1; an aperture leaves
// its lowest bit (state &= inside in the reference).
template <bool FAST, int KIND, bool S_LIVE, bool EBE, bool DENSE, bool OWN>
__device__ __forceinline__ Passed apply(PState &p, const uint64_t *rec, uint64_t hdr,
                                        const TrackParams &prm, const Recip &inv, int64_t start_elem,
                                        int64_t ord)
{
    uint32_t const op = (uint32_t)(hdr & 0xFF);
    uint32_t const aux = (uint32_t)(hdr >> 32);
    auto limit = [&](bool inside) {
        if (EBE) p.state &= 1;
        if (inside) return PASSED;
        p.state = 0;
        return LOST;
    };
    switch (op) {
    case OP_DRIFT:
        if constexpr (OWN) break;
        drift<FAST, S_LIVE, DENSE>(p, W(rec[1]));
        if (!(aux & DRIFT_APERTURE)) return PASSED;
        return limit(inside_global(p, prm.xlim_bits, prm.ylim_bits));
    case OP_MULTIPOLE:
        if constexpr (OWN) break;
        multipole<FAST, false, KIND != KIND_SIMPLE, DENSE>(p, rec, aux);
        return PASSED;
    case OP_SROTATION:
        srotation<FAST>(p, rec);
        return PASSED;
    case OP_XYSHIFT:
        p.x += W(rec[1]);
        p.y += W(rec[2]);
        return PASSED;
    case OP_LIMIT_ELLIPSE:
        return limit(inside_ellipse<FAST>(p, rec, aux));
    case OP_CAVITY:
        cavity<KIND == KIND_MAP>(p, rec, inv);
        return PASSED;
    case OP_MULTIPOLE_CURV:
        multipole<FAST, true, false, false>(p, rec, aux);
        return PASSED;
    case OP_DRIFT_EXACT:
        drift_exact<S_LIVE>(p, W(rec[1]));
        if (!(aux & DRIFT_APERTURE)) return PASSED;
        return limit(inside_global(p, prm.xlim_bits, prm.ylim_bits));
    case OP_LIMIT_RECT:
        return limit(inside_rect(p, rec));
    case OP_LIMIT_RECT_ELLIPSE:
        return limit(inside_rect_ellipse(p, rec));
    case OP_DIPEDGE:
        p.px += W(rec[1]) * p.x;
        p.py += W(rec[2]) * p.y;
        return PASSED;
    case OP_RF_MULTIPOLE:
        if constexpr (KIND != KIND_FULL) break;
        else {
            p = rf_multipole(p, rec, (int)aux);
            return PASSED;
        }
    case OP_BB4D:
        if constexpr (KIND != KIND_FULL) break;
        else {
            p = beam_beam_4d(p, rec);
            return PASSED;
        }
    case OP_BB6D:
        if constexpr (KIND != KIND_FULL) break;
        else {
            if (aux & BB6D_ROUND)
                p = beam_beam_6d<true, FAST>(p, rec, aux);
            else
                p = beam_beam_6d<false, FAST>(p, rec, aux);
            return PASSED;
        }
    case OP_SC_COASTING:
        if constexpr (KIND != KIND_FULL) break;
        else {
            p = sc_coasting(p, rec);
            return PASSED;
        }
    case OP_SC_QGAUSS:
        if constexpr (KIND != KIND_FULL) break;
        else {
            if (aux & SC_PAIR) {
                ScKick const k = sc_qgauss_pair(p.x, p.y, p.px, p.py, p.zeta, p.inv_rvv, p.sc_k,
                                                rec + 1, aux);
                if (k.ok) {
                    p.px = k.px;
                    p.py = k.py;
                    return PASSED;
                }
            }
            p = sc_qgauss<FAST>(p, rec, aux);
            return PASSED;
        }
    case OP_SC_INTERP:
        if constexpr (KIND != KIND_FULL) break;
        else {
            p = sc_interpolated(p, rec, aux);
            return PASSED;
        }
    case OP_TRICUB:
        if constexpr (KIND == KIND_FULL) {
            int64_t const state = p.state;
            if (EBE) p.state = 1;
            p = tricub_element<FAST>(p, rec, aux);
            if (p.state != 1) return FAILED;  // outside the grid: lost, failure
            if (EBE) p.state = state;
            return PASSED;
        } else if constexpr (KIND == KIND_MAP) {
            GridKick const k = tricub<FAST>(p.px, p.py, p.zeta, p.beta0, p.rvv,
                                            p.q0 * p.charge_ratio, p.p0c, p.x, p.y, rec, aux);
            if (!k.inside) {
                p.state = 0;
                return FAILED;
            }
            p.px = k.px;
            p.py = k.py;
            add_energy<true>(p, k.energy, inv);
            return PASSED;
        } else {
            break;
        }
    case OP_MONITOR: {
        uint64_t *out = reinterpret_cast<uint64_t *>(rec[8]);
        if (out == nullptr) return PASSED;
        int64_t const j = monitor_index(rec, p.at_turn, p.pid);
        if (j < 0) return PASSED;
        if (j >= (int64_t)rec[9]) {
            p.state = 0;
            return FAILED;
        }
        store_record(p, out, (int64_t)rec[9], j, start_elem + ord, p.at_turn,
                     p.lazy_s ? prm.s_table[ord] : p.s);
        return PASSED;
    }
    case OP_NOP:
        return PASSED;
    case OP_FAIL:
        return FAILED;
    default:  // OP_FAIL_LOST: unknown type id
        break;
    }
    p.state = 0;
    return FAILED;
}

}  // namespace

// Drifts and multipoles, most of every ring, in a loop of their own: as cases
// of the switch they share its registers and branches.  Measured without and
// with it: 10,000 protons x 20 turns of the FODO ring, exact 2.05 and 1.93 ms,
// fast 1.88 and 1.71; ring with errors, 1,000,000 protons, fast 12.45 and 12.07
// ms; field-map ring 3.77 and 3.71.  Where the FP64 pipe hides the switch it
// only adds code: FODO ring, 200,000 protons, exact 3.30 and 3.43 ms; round
// beam-beam and space charge 3.02 and 3.07.
__host__ __device__ constexpr bool own_loop(int kind, bool dense, bool ebe)
{
    return !ebe && kind != KIND_FULL && !(kind == KIND_SIMPLE && dense);
}

// The records of one staged chunk, in order, for the calling thread's
// particle.  Only lanes that take part walk; one whose particle stops leaves
// the loop, so nothing has to reconverge per element.  The next record's
// header is read before the element is applied: with one or two warps per
// scheduler (10,000 particles) the walk's time is its chain of latencies,
// and the header's shared-memory read was a link of it.
// S_LIVE (block-uniform for the pass): some particle of the block
// accumulates s, so drifts carry the s update.  EBE: element-by-element
// output, whose particles may enter an element already lost (the reference
// checks the state after the map).  DENSE: some FP64 products on the integer
// pipes (mul_rn).
template <bool FAST, int KIND, bool S_LIVE, bool EBE, bool DENSE>
__device__ __forceinline__ void walk_chunk(PState &p, const uint64_t *rec, const TrackParams &prm,
                                           const Recip &inv, bool &part, bool &active, int &status,
                                           int64_t &stop_elem, int64_t &ord, int64_t start_elem)
{
    if (!part) return;
    int64_t const first = ord;
    uint64_t hdr = rec[0];
    uint32_t o = 0;
    // a chunk ends with an OP_END record (or zero padding, which reads as one)
    constexpr bool kOwn = own_loop(KIND, DENSE, EBE);
    auto const stop = [&](Passed rc) {
        if (rc == FAILED) status |= -1;
        part = false;
        active = false;
        stop_elem = first + o;
        if (p.lazy_s) p.s = prm.s_table[first + o + 1];
    };
    while (true) {
        if constexpr (kOwn) {
            while (true) {
                uint32_t const op = (uint32_t)(hdr & 0xFF);
                if (op != OP_DRIFT && op != OP_MULTIPOLE) break;
                const uint64_t *const now = rec;
                uint32_t const aux = (uint32_t)(hdr >> 32);
                rec += (hdr >> 8) & 0xFFFFFFu;
                hdr = rec[0];
                if (op == OP_MULTIPOLE) {
                    multipole<FAST, false, KIND != KIND_SIMPLE, DENSE>(p, now, aux);
                } else {
                    drift<FAST, S_LIVE, DENSE>(p, W(now[1]));
                    if ((aux & DRIFT_APERTURE) && !inside_global(p, prm.xlim_bits, prm.ylim_bits)) {
                        p.state = 0;
                        return stop(LOST);
                    }
                }
                ++o;
            }
        }
        if ((uint32_t)(hdr & 0xFF) == OP_END) break;
        const uint64_t *const next = rec + ((hdr >> 8) & 0xFFFFFFu);
        uint64_t const next_hdr = next[0];
        if constexpr (EBE) {
            int64_t const ae = start_elem + first + o;
            int64_t const j = ebe_index(prm.ebe, p.pid, ae, p.at_turn);
            if (j >= 0 && j < prm.ebe_cap)
                store_record(p, prm.ebe_out, prm.ebe_cap, j, ae, p.at_turn,
                             p.lazy_s ? prm.s_table[first + o] : p.s);
        }
        Passed const rc = apply<FAST, KIND, S_LIVE, EBE, DENSE, kOwn>(p, rec, hdr, prm, inv,
                                                                       start_elem, first + o);
        if (rc != PASSED || (EBE && p.state != 1)) return stop(rc);
        ++o;
        rec = next;
        hdr = next_hdr;
    }
    ord = first + o;
}

__device__ __forceinline__ void mbar_inval(uint64_t *bar)
{
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Above two warps per scheduler (of 152 SMs) the FP64 pipe is the bound and
// some of its multiplications run on the integer pipes beside it; below, a
// warp's own chain of latencies is, and the FP64 instruction's 64 cycles are
// the shorter way to a product.  Measured, integer against FP64 products: a
// FODO ring, exact, 100,000 protons 2.00 against 2.72 ms, 60,000 1.22 / 1.41,
// 32,000 0.75 / 0.77, 10,000 2.27 / 2.09 (more turns); a 2,000-element ring,
// fast, 100,000 2.48 / 2.60, 32,000 1.16 / 1.15.
constexpr int64_t kDenseParticles = 2 * 32 * 4 * 152;

// One CTA's share of a tracking call: particle t of the launch (an index
// into prm.idx, or prm.i0 + t).  The loops over turns and chunks are
// block-uniform; within a chunk only lanes whose particle takes part walk its
// records, and one whose particle stops leaves the walk (walk_chunk), all of
// them back together at the barrier after the chunk or the turn.  `smem` holds
// 16 words of mbarriers followed by prm.stages chunk buffers.  Returns with
// every copy it issued complete; the caller invalidates the barriers before
// the shared memory is used again.
template <bool FAST, int KIND>
__device__ __forceinline__ void track_block(const TrackParams &prm, int64_t t, uint64_t *smem,
                                            int64_t together)
{
    bool const dense = together > kDenseParticles;
    int const stages = prm.stages;
    int const cw = prm.chunk_words;
    uint64_t *bars = smem;                 // `stages` mbarriers (8 B each, padded to 16 words)
    uint64_t *bufs = smem + 16;            // stages * cw words
    __shared__ long long s_tmin;

    int64_t i;
    bool valid;
    if (prm.idx) {  // compacted launch: only the particles with work left
        valid = t < *prm.count;
        i = valid ? prm.idx[t] : 0;
    } else {
        i = prm.i0 + t;
        valid = i < prm.i1;
    }
    PState p;
    Recip inv{};  // KIND_MAP
    if (valid) {
        load_particle(p, prm.cols, prm.n, i);
        if constexpr (KIND == KIND_MAP) inv = Recip{1.0 / p.beta0, 1.0 / p.energy0};
        // s of a turn that starts at +0 comes from the lattice's s table
        p.lazy_s = (prm.mode != MODE_LINE) && (__double_as_longlong(p.s) == 0);
    }

    // ---------------------------------------------------- per-mode setup
    int64_t const start_elem = valid ? p.at_element : 0;
    bool active;   // still has work in this call
    if (prm.mode == MODE_UNTIL) {
        active = valid && p.state == 1 && p.at_turn < prm.until_turn;
    } else if (prm.mode == MODE_LINE) {
        active = valid && p.state == 1;
    } else {  // MODE_EBE: the reference does not check state here
        active = valid && prm.until_turn > p.at_turn && p.at_turn >= 0 && start_elem >= 0 &&
                 p.pid >= 0;
    }
    int status = 0;
    int64_t stop_elem = -1;  // element ordinal where tracking stopped
    bool const started = active;

    if (threadIdx.x == 0) {
        s_tmin = 0x7FFFFFFFFFFFFFFFll;
        for (int s = 0; s < stages; ++s) mbar_init(&bars[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (active && prm.mode != MODE_LINE) atomicMin(&s_tmin, (long long)p.at_turn);
    bool any = __syncthreads_or(active);
    int64_t turn = (prm.mode == MODE_LINE) ? 0 : (int64_t)s_tmin;

    int const nch = prm.n_chunks;
    bool const resident = nch <= stages;
    int64_t issued = 0;    // chunk loads issued (meaningful in thread 0 only)
    int64_t consumed = 0;  // chunk loads waited for (block-uniform)
    bool timed_out = false;
    if (any) {
        if (threadIdx.x == 0) {
            int const first = resident ? nch : stages;
            for (int g = 0; g < first; ++g) {
                mbar_arrive_expect_tx(&bars[g], (uint32_t)(cw * 8));
                bulk_copy_g2s(bufs + (size_t)g * cw, prm.stream + (size_t)(g % nch) * cw,
                              (uint32_t)(cw * 8), &bars[g]);
            }
            issued = first;
        }
        if (resident) {  // the whole lattice stays in shared memory
            // consumed = the first chunk not seen complete: after a timeout
            // the drain below waits for it and every later one
            int first_bad = nch;
            for (int g = 0; g < nch; ++g)
                if (!mbar_wait_bounded(&bars[g], 0u) && first_bad == nch) first_bad = g;
            consumed = first_bad;
            timed_out = __syncthreads_or(first_bad < nch);
        }
    }

    while (any && !timed_out) {
        bool part = (prm.mode == MODE_LINE) ? active : (active && (p.at_turn == turn));
        // some particle of the block accumulates s in this pass (block-uniform)
        bool const s_live = __syncthreads_or(part && !p.lazy_s);
        int64_t ord = 0;  // element ordinal within the turn / line
        for (int c = 0; c < nch; ++c) {
            int buf = c;
            if (!resident) {
                buf = (int)(consumed % stages);
                uint32_t const parity = (uint32_t)((consumed / stages) & 1);
                bool const ok = mbar_wait_bounded(&bars[buf], parity);
                if (ok) ++consumed;  // a chunk that timed out is left to the drain
                if (__syncthreads_or(!ok)) {
                    timed_out = true;
                    break;
                }
            }
            const uint64_t *rec = bufs + (size_t)buf * cw;
            if (prm.mode == MODE_EBE)
                walk_chunk<FAST, KIND, true, true, false>(p, rec, prm, inv, part, active, status,
                                                          stop_elem, ord, start_elem);
            else if (s_live)
                walk_chunk<FAST, KIND, true, false, false>(p, rec, prm, inv, part, active, status,
                                                           stop_elem, ord, start_elem);
            else if (dense)
                walk_chunk<FAST, KIND, false, false, true>(p, rec, prm, inv, part, active, status,
                                                           stop_elem, ord, start_elem);
            else
                walk_chunk<FAST, KIND, false, false, false>(p, rec, prm, inv, part, active, status,
                                                            stop_elem, ord, start_elem);
            if (!resident) {
                __syncthreads();  // every warp is done with this stage buffer
                if (threadIdx.x == 0) {
                    int64_t const g = issued;  // next chunk of the cyclic stream
                    int const b = (int)(g % stages);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_arrive_expect_tx(&bars[b], (uint32_t)(cw * 8));
                    bulk_copy_g2s(bufs + (size_t)b * cw, prm.stream + (size_t)(g % nch) * cw,
                                  (uint32_t)(cw * 8), &bars[b]);
                    issued = g + 1;
                }
            }
        }
        if (timed_out) break;
        if (prm.mode == MODE_LINE) {
            if (part && prm.finish_turn) {  // track/track.h:813-819
                p.at_turn += 1;
                p.s = 0.0;
            }
            active = false;
        } else if (part) {  // turn completed
            p.at_turn += 1;
            p.s = 0.0;
            p.lazy_s = true;
            if (p.at_turn >= prm.until_turn) active = false;
        }
        ++turn;
        any = __syncthreads_or(active);
        // every particle of the block is at a turn boundary here: a capped
        // launch may stop, the next launch resumes from the stored state
        if (prm.mode == MODE_UNTIL && prm.turn_cap > 0 && turn >= (int64_t)s_tmin + prm.turn_cap)
            any = false;
    }

    // drain bulk copies still in flight before the CTA exits (a resident
    // lattice has none left unless a wait timed out)
    if (threadIdx.x == 0 && (!resident || timed_out)) {
        while (consumed < issued) {
            int const buf = (int)(consumed % stages);
            uint32_t const parity = (uint32_t)((consumed / stages) & 1);
            if (!mbar_wait_bounded(&bars[buf], parity)) {
                timed_out = true;
                break;
            }
            ++consumed;
        }
    }
    if (timed_out) {
        if (threadIdx.x == 0) atomicOr(prm.error, ERR_PIPELINE_TIMEOUT);
        return;  // particle columns are left untouched
    }

    if (!valid) return;
    // ------------------------------------------------ final bookkeeping
    if (prm.mode == MODE_UNTIL) {
        if (stop_elem >= 0) {
            p.state = 0;  // track/track.h:663-666
            p.at_element = start_elem + stop_elem;
        }
    } else if (prm.mode == MODE_LINE) {
        if (started) {  // particles lost before the call are left as they are
            int64_t const done = (stop_elem >= 0) ? stop_elem : prm.num_elements;
            p.at_element = start_elem + done;
            if (stop_elem < 0 && prm.finish_turn && p.state == 1) p.at_element = 0;
        }
    } else {  // EBE
        if (stop_elem >= 0) p.at_element = start_elem + stop_elem;
    }
    if (status != 0) atomicOr(prm.status, status);

    double *d = reinterpret_cast<double *>(prm.cols);
    int64_t *k = reinterpret_cast<int64_t *>(prm.cols);
    int64_t const n = prm.n;
    d[5 * n + i] = p.s;
    d[6 * n + i] = p.x;
    d[7 * n + i] = p.y;
    d[8 * n + i] = p.px;
    d[9 * n + i] = p.py;
    d[10 * n + i] = p.zeta;
    d[11 * n + i] = p.psigma;
    d[12 * n + i] = p.delta;
    d[13 * n + i] = p.rpp;
    d[14 * n + i] = p.rvv;
    k[18 * n + i] = p.at_element;
    k[19 * n + i] = p.at_turn;
    k[20 * n + i] = p.state;
}

template <bool FAST, int MIN_BLOCKS, int KIND>
__global__ void __launch_bounds__(kMaxThreads, MIN_BLOCKS) track_kernel(TrackParams prm)
{
    extern __shared__ __align__(128) uint64_t smem[];
    track_block<FAST, KIND>(prm, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, smem,
                            prm.idx ? *prm.count : prm.i1 - prm.i0);
}

// Persistent batched kernel: each CTA takes work items (a tile of
// blockDim.x particles of one lattice variant) from a global counter until
// none is left, and tracks the tile until turn *base_turn + turn_offset with
// that variant's lattice.  Items are ordered longest first by the host.
template <bool FAST, int MIN_BLOCKS, int KIND>
__global__ void __launch_bounds__(kMaxThreads, MIN_BLOCKS)
    batch_kernel(const TrackParams *variants, const BatchItem *items, int32_t num_items,
                 int32_t *counter, const int64_t *base_turn, int64_t turn_offset)
{
    extern __shared__ __align__(128) uint64_t smem[];
    __shared__ int32_t s_item;
    int64_t const until = *base_turn + turn_offset;
    while (true) {
        __syncthreads();  // previous item done (barriers invalidated, s_item read)
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        int32_t const it = s_item;
        if (it >= num_items) break;
        BatchItem const w = items[it];
        TrackParams prm = variants[w.variant];
        prm.until_turn = until;
        prm.idx = nullptr;
        prm.count = nullptr;
        prm.i0 = w.first;
        prm.i1 = (w.first + blockDim.x < prm.n) ? w.first + blockDim.x : prm.n;
        track_block<FAST, KIND>(prm, threadIdx.x, smem, (int64_t)num_items * blockDim.x);
        __syncthreads();
        if (threadIdx.x == 0)
            for (int b = 0; b < prm.stages; ++b) mbar_inval(&smem[b]);
    }
}

template <bool FAST, int MB, int KIND>
static int launch_one(const TrackParams &prm, unsigned blocks, int threads, size_t smem,
                      cudaStream_t s)
{
    cudaError_t err = cudaFuncSetAttribute(track_kernel<FAST, MB, KIND>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
    track_kernel<FAST, MB, KIND><<<blocks, threads, smem, s>>>(prm);
    return (int)cudaGetLastError();
}

template <int KIND>
int launch_kind(const TrackParams &prm, bool fast, bool two, unsigned blocks, int threads,
                size_t smem, cudaStream_t s)
{
    if (fast)
        return two ? launch_one<true, 2, KIND>(prm, blocks, threads, smem, s)
                   : launch_one<true, 1, KIND>(prm, blocks, threads, smem, s);
    return two ? launch_one<false, 2, KIND>(prm, blocks, threads, smem, s)
               : launch_one<false, 1, KIND>(prm, blocks, threads, smem, s);
}

template <bool FAST, int MB, int KIND>
static cudaError_t batch_occupancy(int threads, size_t smem, int *per_sm)
{
    cudaError_t err = cudaFuncSetAttribute(batch_kernel<FAST, MB, KIND>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, batch_kernel<FAST, MB, KIND>,
                                                         threads, smem);
}

template <int KIND>
cudaError_t batch_occupancy_kind(bool fast, bool two, int threads, size_t smem, int *per_sm)
{
    if (fast)
        return two ? batch_occupancy<true, 2, KIND>(threads, smem, per_sm)
                   : batch_occupancy<true, 1, KIND>(threads, smem, per_sm);
    return two ? batch_occupancy<false, 2, KIND>(threads, smem, per_sm)
               : batch_occupancy<false, 1, KIND>(threads, smem, per_sm);
}

template <bool FAST, int MB, int KIND>
static int launch_batch_one(const BatchLaunch &b, cudaStream_t s)
{
    batch_kernel<FAST, MB, KIND><<<b.grid, b.threads, b.smem, s>>>(
        b.variants, b.items, b.num_items, b.counter, b.base_turn, b.turn_offset);
    return (int)cudaGetLastError();
}

template <int KIND>
int launch_batch_kind(const BatchLaunch &b, cudaStream_t s)
{
    bool const two = b.blocks_per_sm >= 2;
    if (b.fast)
        return two ? launch_batch_one<true, 2, KIND>(b, s) : launch_batch_one<true, 1, KIND>(b, s);
    return two ? launch_batch_one<false, 2, KIND>(b, s) : launch_batch_one<false, 1, KIND>(b, s);
}

#define STG_KIND(PREFIX, K)                                                                   \
    PREFIX template int launch_kind<K>(const TrackParams &, bool, bool, unsigned, int, size_t, \
                                       cudaStream_t);                                          \
    PREFIX template cudaError_t batch_occupancy_kind<K>(bool, bool, int, size_t, int *);       \
    PREFIX template int launch_batch_kind<K>(const BatchLaunch &, cudaStream_t);

}  // namespace stg
