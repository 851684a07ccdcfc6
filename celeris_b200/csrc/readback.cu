// Forms the public RGBA32F texels of a state or record (readback.hpp).  Bound by the bus it writes over
// (or, for small reads, by its launch).
//
// Built without flush-to-zero, so that hi + lo is the host's double-precision sum to the last bit.
#include "readback.hpp"

#include <algorithm>

namespace cel {

namespace {

__global__ void __launch_bounds__(256) k_pack(PackArgs a, unsigned first, unsigned count, float4* __restrict__ out) {
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const unsigned t = first + k, y = t / unsigned(a.NX), x = t - y * unsigned(a.NX);
        const size_t e = size_t(y) * a.P + x;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.mode == PACK_AUX) {
            const float2 v = a.aux[e];
            o.x = v.x;
            o.w = v.y;
        } else if (a.mode == PACK_LO) {
            if (a.lo[0]) o = make_float4(a.lo[0][e], a.lo[1][e], a.lo[2][e], 0.f);
        } else if (a.mode == PACK_SUM && a.lo[0]) {
            o.x = float(double(a.hi[0][e]) + double(a.lo[0][e]));
            o.y = float(double(a.hi[1][e]) + double(a.lo[1][e]));
            o.z = float(double(a.hi[2][e]) + double(a.lo[2][e]));
        } else {
            o = make_float4(a.hi[0][e], a.hi[1][e], a.hi[2][e], 0.f);
        }
        out[k] = o;
    }
}

}  // namespace

cudaError_t launch_pack(const PackArgs& a, size_t first, size_t count, float4* out, cudaStream_t s) {
    k_pack<<<unsigned(std::min<size_t>((count + 255) / 256, 1184)), 256, 0, s>>>(a, unsigned(first), unsigned(count), out);
    return cudaGetLastError();
}

}  // namespace cel
