// teno_cert.cuh -- a cheap proof that a variable takes the central stencil.
//
// TENO keeps the central stencil when w_0 / (w_0 + sum_d w_d) > 1e-7 with
// w = (SI + 1e-12)^-6, i.e. when sum_d (x_0 / x_d)^6 < 1e7 - 1 for
// x = SI + 1e-12.  In smooth flow the three directional polynomials are
// computed only to lose that comparison.  The proof needs a lower bound of
// each directional SI = c^T OI c, and two linear functionals g = W c of the
// coefficients give one: SI >= g^T (W OI^-1 W^T)^-1 g for every c.  W is the
// mean gradient over the reference triangle, which dominates SI wherever the
// flow varies smoothly, so g is close to the central polynomial's and the
// bound is within a few per cent (the ratio has to differ by 12 in SI for the
// decision to change).  g = sum_j C_j d_j needs 2 numbers per stencil cell
// instead of the pseudo-inverse's K - 1 = 9.
//
// Everything here is FP32 and bounds its own rounding:
//   |g32 - g|        <= eg D sum_j |C_j|          (rounded C and d, the sums; D = max |d_j|)
//   |c_kernel - c|   <= ec D (sum_j |P_kj|)_k     (the kernel's own rounding)
// whose effects on sqrt(SI) add up to D certn, one number per stencil built
// with the tables, and
//   SI_kernel        >= cert_lo SI(c_kernel)            (its quadratic form's rounding)
// The FP64 forms take their differences from FP32 pairs (high, low) of the
// state, (h_j - h_c) + (l_j - l_c): h_j - h_c is exact where it cancels, so
// the error is under 3 u |d| + 2^-45 max |u|, the last term a perturbation of
// the data whose effect on sqrt(SI) is max |u| certu.
// A test that does not prove the decision says nothing: the cell then runs
// the full kernel.  NaN and infinities prove nothing either: every cell has a
// directional stencil to compare with (one lacks where its face is a boundary,
// and a cell with three boundary faces has no neighbours to fill its central
// stencil from, which the set-up refuses).
#pragma once

#include "device.h"

namespace mgpu {
namespace {

// Running sums of one stencil's functionals.
struct CertSum {
    float g0 = 0.0f, g1 = 0.0f, D = 0.0f;
    __device__ __forceinline__ void add(float c0, float c1, float d) {
        g0 = fmaf(c0, d, g0);
        g1 = fmaf(c1, d, g1);
        D = fmaxf(D, fabsf(d));
    }
    // lower bound of the stencil's SI + 1e-12; finite becomes false on a NaN
    // or an infinity in the stencil
    // off: the effect of an absolute error of the differences, else 0
    __device__ __forceinline__ float x_low(const TenoArgs& a, float certn, float off, bool& finite) const {
        const float q = fmaf(g0 * g0, a.cert_b[0], fmaf(g0 * g1, a.cert_b[1], g1 * g1 * a.cert_b[2]));
        finite = finite && q < 3.0e38f;
        const float l = 0.9999f * sqrtf(fmaxf(q, 0.0f)) - fmaf(certn, D, off);
        const float p = fmaxf(l, 0.0f);
        return fmaf(a.cert_lo * p, p, 1.0e-12f);
    }
};

// (x0 / xd)^6
__device__ __forceinline__ float ratio6(float x0, float xd) {
    const float t = x0 / xd, t2 = t * t;
    return t2 * t2 * t2;
}

// Proven: the sum of the three ratios, each with a lower bound of xd, stays
// under half the decision's threshold (the factor two covers the rounding of
// the powers here and in the kernel); or x0 is so small (1.1e-11 against
// xd >= 1e-12: at most 3 x 11^6 = 5.3e6) that no directional SI matters.
__device__ __forceinline__ bool cert_passes(float x0, float r, bool finite) {
    return finite && (r < 5.0e6f || x0 < 1.1e-11f);
}

// Appends the warp's unproven cells (item: what the list holds for a cell) to the list.  Called by all lanes of the
// warp (four per cell); hard: this lane's variable is not proven.  Returns
// whether the lane's cell went on the list.  The list has room for every cell
// (cap); only a list that a failed launch left unread could run past it, and
// is cut there.
__device__ __forceinline__ bool append_hard(uint32_t* list, unsigned* list_n, unsigned cap, uint32_t item, bool hard) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned hb = __ballot_sync(0xffffffffu, hard);
    const bool cell_hard = ((hb >> (lane & ~3u)) & 0xFu) != 0u;
    const bool lead = cell_hard && (lane & 3u) == 0u;
    const unsigned leads = __ballot_sync(0xffffffffu, lead);
    if (leads) {
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(list_n, (unsigned)__popc(leads));
        base = __shfl_sync(0xffffffffu, base, 0);
        const unsigned at = base + (unsigned)__popc(leads & ((1u << lane) - 1u));
        if (lead && at < cap) list[at] = item;
    }
    return cell_hard;
}

// The list's length, read once per block by a kernel that works the list off,
// and the list's reset by its last block (list_n[1] counts the blocks that
// have read it).  Called by every thread of the block, before any leaves.
__device__ __forceinline__ unsigned take_hard_count(unsigned* list_n, unsigned cap) {
    __shared__ unsigned n;
    if (threadIdx.x == 0) {
        n = min(*reinterpret_cast<volatile unsigned*>(list_n), cap);
        __threadfence();
        if (atomicAdd(list_n + 1, 1u) == gridDim.x - 1) {
            list_n[0] = 0u;
            list_n[1] = 0u;
        }
    }
    __syncthreads();
    return n;
}

}  // namespace
}  // namespace mgpu
