// stream.h -- the device element stream: a CObjects lattice compiled into
// fixed-size chunks of 8-byte words that CTAs stage into shared memory with
// bulk (TMA) copies and walk as warp-uniform records.
//
// Record = header word + parameters.  Header bits: 0-7 opcode, 8-31 record
// length in words (header included), 32-63 auxiliary value (multipole order,
// slice count, flags).  One record per lattice element, in lattice order,
// so the element index is the record ordinal.  Every chunk ends with an
// OP_END record; records never straddle chunks.
#pragma once

#include <cstdint>

namespace stg {

enum Op : uint32_t {
    OP_END = 0,             // end of chunk
    OP_DRIFT = 1,           // [L]            aux bit0: global aperture check
    OP_DRIFT_EXACT = 2,     // [L]            aux bit0: global aperture check
    OP_MULTIPOLE = 3,       // [bal 0..2n+1]  aux = order n | MP_ flags; with
                            // MP_LEAD the lead block follows (leadkick.cuh)
    OP_MULTIPOLE_CURV = 4,  // [bal..., hxl, hyl, length, hxl/length, hyl/length]
                            // aux = order n | MP_ flags
    OP_CAVITY = 5,          // [voltage, k*frequency, deg2rad*lag]
    OP_XYSHIFT = 6,         // [-dx, -dy]
    OP_SROTATION = 7,       // [cos_z, sin_z]
    OP_LIMIT_RECT = 8,      // [min_x, max_x, min_y, max_y]
    OP_LIMIT_ELLIPSE = 9,   // [a_squ, b_squ, a_b_squ]  aux bit0: compare as floats
    OP_LIMIT_RECT_ELLIPSE = 10,  // [max_x, max_y, a_squ, b_squ, a_squ_b_squ]
    OP_DIPEDGE = 11,        // [r21, r43]
    OP_RF_MULTIPOLE = 12,   // [voltage, frequency, lag, bal..., phase...] aux = order
    OP_BB4D = 13,           // [11 BB4D data words]
    OP_BB6D = 14,           // [34 head words, n_part[N], x[N], y[N], sigma[N]]
                            // aux = N | BB6D_ROUND | BB6D_UNCOUPLED
    OP_SC_COASTING = 15,    // [9 SCCoasting words]
    OP_SC_QGAUSS = 16,      // [11 SCQGaussProfile words, sqrt_beta = 1 / (sqrt(2)
                            //  bunchlength_rms), sqrt_beta^2, sqrt_beta / cq,
                            //  1 / (1 - q) (0 when |1 - q| < 1e-6),
                            //  0.5 / sigma^2, 1 / (2 pi eps0 sigma),
                            //  1 / S, 1 / (2 eps0 sqrt(pi) S), sigma_y / sigma_x,
                            //  sigma_x / sigma_y, 1 / (2 sigma_x^2),
                            //  1 / (2 sigma_y^2), length N sqrt_beta / cq /
                            //  (2 pi eps0) and 1 / sigma (round; else 0)],
                            //  S = sqrt(2 |sigma_x^2 - sigma_y^2|)
                            // aux bit0 (SC_ROUND): |sigma_x - sigma_y| <
                            //  min_sigma_diff, sigma = (sigma_x + sigma_y) / 2;
                            // bit1 / bit2 (SC_ELL_X / SC_ELL_Y): elliptic with
                            //  sigma_x > sigma_y / sigma_x < sigma_y;
                            // bit3 (SC_Q1): |1 - q| < 1e-6 (Gaussian profile);
                            // bit4 (SC_PAIR): followed by the 8 words of
                            //  sckick.cuh
    OP_MONITOR = 17,        // [num_stores, start, skip, max_pid, min_pid, rolling,
                            //  turn_ordered, out_ptr, out_capacity]
    OP_NOP = 18,            // success, no effect (disabled beam-beam)
    OP_FAIL = 19,           // failure (map compiled out, e.g. TriCub)
    OP_FAIL_LOST = 20,      // failure and particle lost (unknown type id)
    OP_SC_INTERP = 21,      // [N, sigma_x, sigma_y, length, x_co, y_co, fallback,
                            //  min_sigma_diff, method, num_values, z0, dz,
                            //  values@, derivatives@, nwords, table address]
                            // the table (nwords words, values@ / derivatives@
                            // word offsets into it) lies in device memory
                            // outside the stream; aux bit0: interpolate (else
                            // the fallback density)
    OP_TRICUB = 22,         // [x_shift, y_shift, tau_shift, dipolar_kick_px,
                            //  dipolar_kick_py, dipolar_kick_ptau,
                            //  length / dx, length / dy, length / dz,
                            //  x0, y0, z0, 1 / dx, 1 / dy, 1 / dz,
                            //  nx - 2, ny - 2, nz - 2 (as doubles),
                            //  nx - 1, ny - 1 (cells per row / plane),
                            //  cell coefficient table address]
                            // aux bits 0-2: mirror in x, y, z.  The table (64
                            // coefficients per grid cell, x^i y^j z^k at
                            // k + 4 j + 16 i) lies in device memory outside
                            // the stream, computed there from the node table
    OP_COUNT
};

// Beside the opcodes in a lattice's op mask: some multipole has a lead block.
constexpr uint32_t OPM_LEAD = 1u << 31;
static_assert(OP_COUNT <= 31, "op mask bits");

constexpr uint32_t DRIFT_APERTURE = 1u;
// Multipole aux word: the order and what is known of the coefficients
// (multipole_aux).
constexpr uint32_t MP_ORDER = 0xFFu;
constexpr uint32_t MP_SKEW0 = 1u << 8;   // every skew coefficient is +-0
constexpr uint32_t MP_PLUS = 1u << 9;    // every skew coefficient is +0, no other is -0
constexpr uint32_t MP_DIPOLE0 = 1u << 10;  // bal[0] and bal[1] are +0
constexpr uint32_t MP_LEAD = 1u << 11;     // the quadrupole term leads
// TriCub aux flags: mirror the grid coordinate in x / y / z (mirror_* == 1).
constexpr uint32_t TRICUB_MIRROR_X = 1u;
constexpr uint32_t TRICUB_MIRROR_Y = 2u;
constexpr uint32_t TRICUB_MIRROR_Z = 4u;
// SC q-Gaussian aux flag: the transverse field is the round one.
constexpr uint32_t SC_ROUND = 1u;
constexpr uint32_t SC_ELL_X = 2u;
constexpr uint32_t SC_ELL_Y = 4u;
constexpr uint32_t SC_Q1 = 8u;
constexpr uint32_t SC_PAIR = 16u;
constexpr uint32_t SC_PAIR_AT = 25;  // parameter index of the sckick.cuh words

// BB6D aux flag: the strong beam's Sigma matrix is round and uncoupled
// (S11 = S33, S12 = S34, S22 = S44, S13 = S14 = S23 = S24 = 0) with
// threshold_singular > 0 and min_sigma_diff > 0.  Then R = S13 = 0 at every
// S, and NS(BeamBeam6D_propagate_Sigma_matrix) always takes its singular
// branch with cos theta = 1, sin theta = 0 and no theta derivative, and the
// field is the round one: the map computes only what that branch needs.
constexpr uint32_t BB6D_ROUND = 1u << 31;
// BB6D aux flag: uncoupled (S13 = S14 = S23 = S24 = 0) with threshold_singular
// > 0.  Where R = S11 - S33 is not singular the propagation is S11(S) and
// S33(S) themselves with cos theta = 1, sin theta = 0 and no theta derivative
// (up to the rounding of the general formulas).
constexpr uint32_t BB6D_UNCOUPLED = 1u << 30;
constexpr uint32_t BB6D_SLICES = BB6D_UNCOUPLED - 1u;

inline uint64_t make_header(uint32_t op, uint32_t nwords, uint32_t aux)
{
    return (uint64_t)op | ((uint64_t)(nwords & 0xFFFFFFu) << 8) | ((uint64_t)aux << 32);
}

// The aux word of a multipole of order n with coefficients bal[0..2n+1]; made
// again wherever a coefficient is changed.
inline uint32_t multipole_aux(const uint64_t *bal, uint32_t order)
{
    constexpr uint64_t kMinusZero = (uint64_t)1 << 63;
    uint64_t skew = 0;
    bool minus_zero = false;
    for (uint32_t k = 0; k <= order; ++k) {
        skew |= bal[2 * k + 1];
        minus_zero = minus_zero || bal[2 * k] == kMinusZero;
    }
    return order | ((skew << 1) == 0 ? MP_SKEW0 : 0u) |
           (skew == 0 && !minus_zero ? MP_PLUS : 0u) |
           ((bal[0] | bal[1]) == 0 ? MP_DIPOLE0 : 0u);
}

// Global aperture compare: |x| < limit  <=>  bits(|x|) < bits(limit) for a
// positive finite limit (IEEE doubles of one sign order like their bit
// patterns; NaN and inf compare false, as in the reference's float compare).
inline uint64_t aperture_bits(double limit)
{
    if (!(limit > 0.0)) return 0;  // nothing is inside a non-positive limit
    uint64_t w;
    __builtin_memcpy(&w, &limit, 8);
    return w;
}

struct StreamInfo {
    int64_t num_elements = 0;
    int32_t num_chunks = 0;
    int32_t chunk_words = 0;
    int32_t max_record_words = 0;
    int32_t num_monitors = 0;
    uint32_t op_mask = 0;  // bit per opcode present, OPM_LEAD
};

}  // namespace stg
