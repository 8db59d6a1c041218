// gate_ops.cuh -- element operations shared by the torus blind-rotation kernels: the gate's linear
// combination, a launch item's inputs and the rounding of products to the torus.
#pragma once

#include "torus.cuh"

namespace cbs {

// request holding ragged item `item` (binary search over the offsets)
__device__ __forceinline__ uint32_t gate_req_of(const GateReq* reqs, uint32_t num, uint32_t item) {
    uint32_t lo = 0, hi = num;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (__ldg(&reqs[mid].offset) <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t gate_a(int gate, uint32_t x1, uint32_t x2) {
    const uint32_t s = x1 + x2;
    switch (gate) {
        case 0: case 1: return s;
        case 2: case 3: return 0u - s;
        case 4: return 2u * s;
        case 5: return 0u - 2u * s;
        default: return x1;
    }
}

__device__ __forceinline__ uint32_t gate_b(int gate, uint32_t x1, uint32_t x2) {
    const uint32_t e8 = 1u << 29, e4 = 1u << 30, s = x1 + x2;
    switch (gate) {
        case 0: return e8 + s;
        case 1: return (0u - e8) + s;
        case 2: return (0u - e8) - s;
        case 3: return e8 - s;
        case 4: return e4 + 2u * s;
        case 5: return (0u - e4) - 2u * s;
        default: return x1;
    }
}

// the torus value of the FP64 result v of an integer-valued product: exact for 32-bit
// tori (|v| < 2^52); for 64-bit tori v carries FP64 rounding, reduced mod 2^64 exactly
template <typename TT>
__device__ __forceinline__ TT to_torus(double v);
template <>
__device__ __forceinline__ uint32_t to_torus<uint32_t>(double v) {
    return static_cast<uint32_t>(static_cast<uint64_t>(__double2ll_rn(v)));
}
template <>
__device__ __forceinline__ uint64_t to_torus<uint64_t>(double v) {
    const double k = rint(v * 0x1p-64);
    double r = fma(-k, 0x1p64, v);  // exact: v - k 2^64, |r| <= 2^63
    if (r >= 0x1p63) r -= 0x1p64;
    return static_cast<uint64_t>(__double2ll_rn(r));
}

// inputs of item `item` of a blind-rotation launch: the LWE rows a1 and a2 (a2 = a1 outside
// gate mode) and the combined b
__device__ __forceinline__ void gate_item_inputs(const GateArgs& a, uint32_t item, const uint32_t*& a1,
                                                 const uint32_t*& a2, uint32_t& b) {
    if (a.reqs) {  // ragged: one bootstrap of request r
        const GateReq& rq = a.reqs[gate_req_of(a.reqs, a.num_reqs, item)];
        const uint32_t k = item - rq.offset;
        a1 = rq.a + static_cast<size_t>(k) * a.n;
        a2 = a1;
        b = rq.b[k];
    } else {
        const uint32_t in = item / a.levels_tv;
        a1 = a.a1 + static_cast<size_t>(in) * a.n;
        a2 = a.a2 ? a.a2 + static_cast<size_t>(in) * a.n : a1;
        b = gate_b(a.gate, a.b1[in], a.b2 ? a.b2[in] : 0u);
    }
}

}  // namespace cbs
