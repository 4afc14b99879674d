// Shared host/device helpers of the aurora-pic B200 library.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <stdexcept>
#include <string>

#include "aurorapic_b200.h"

namespace apic {

// A failure that maps onto an apic_status at the C ABI.
struct Error : std::runtime_error {
    int status;
    Error(int s, const std::string& what) : std::runtime_error(what), status(s) {}
};

inline void cuda_check(cudaError_t e, const char* what) {
    if (e != cudaSuccess)
        throw Error(APIC_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define APIC_CUDA(call) ::apic::cuda_check((call), #call)

inline void require(bool ok, const std::string& what, int status = APIC_ERR_INVALID) {
    if (!ok) throw Error(status, what);
}

// Fixed-point charge accumulation: contributions are rounded once to
// multiples of 2^-scale_bits and summed in 64-bit integers, so the deposited
// density does not depend on the order in which particles are processed.
__device__ __forceinline__ long long to_fixed(double value, double scale) {
    return __double2ll_rn(value * scale);
}

// A 64-bit sum in shared memory as two 32-bit words: a 64-bit shared atomicAdd
// is a compare-and-swap loop, which same-node deposits of a warp run one
// lane after another, while 32-bit adds are native.  The low word's add returns its old value,
// so the carry it causes goes to the high word and the pair holds the exact sum
// modulo 2^64 in any order (1D pass over 1 M particles on 64 nodes: 47 -> 37 us;
// step of the FP32 discharge: 62 -> 51 us).
__device__ __forceinline__ void shared_add64(unsigned* lo, unsigned* hi, int i, long long v) {
    const unsigned l = (unsigned)(unsigned long long)v;
    const unsigned old = atomicAdd(lo + i, l);
    const unsigned h = (unsigned)((unsigned long long)v >> 32) + (old + l < old ? 1u : 0u);
    if (h) atomicAdd(hi + i, h);
}
__device__ __forceinline__ unsigned long long join64(unsigned lo, unsigned hi) {
    return (unsigned long long)hi << 32 | lo;
}

// x / d for 0 <= x <= L from the rounded reciprocal rd = 1 / d: a product and
// one Newton correction of the quotient through its exact remainder (Markstein,
// IBM J. Res. Dev. 34 (1990) 111): three operations where the division takes
// about nine and a slow path.  The corrected quotient is the rounding of a
// value within 2^-52 ulp of x / d, for x from 2^-960 on (below, the remainder leaves
// the normal range and the last bits of a quotient near 0 may differ).  rd = 0
// asks for the division (spacings whose reciprocal would leave it).
__host__ __device__ __forceinline__ double cells_of(double x, double d, double rd) {
    if (rd == 0.0) return x / d;
    const double q = x * rd;
    return fma(fma(-q, d, x), rd, q);
}
inline double reciprocal_spacing(double d) { return d > 1e-280 && d < 1e280 ? 1.0 / d : 0.0; }

// Waits on the handle's stream without blocking forever: polls the event
// until it completes or `seconds` elapse.
cudaError_t bounded_wait(cudaStream_t stream, double seconds);

// Device error word -> apic_status (first matching bit wins).
int status_from_device(unsigned word);
std::string describe_device_error(unsigned word);

}  // namespace apic
