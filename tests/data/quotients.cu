// Counts where the device's corrected quotients differ in bits from the division (two NaNs are equal).
#include "device_math.cuh"
#include "traverse.cuh"

namespace lam {
LAM_DEV bool alpha_accept(const DevScene&, uint32_t, uint32_t, float, float, bool) { return true; }
}  // namespace lam
using namespace lam;

__device__ void differs(float got, float want, unsigned long long* count) {
    if (__float_as_uint(got) != __float_as_uint(want) && !(got != got && want != want)) atomicAdd(count, 1ull);
}

// counts[0]: over_pi, all 2^32 floats; [1]: byte_over_255, all bytes; [2]: unpack_snorm16, all 16-bit words;
// [3]: quotient_f64, 2^26 pairs of floats, a quarter of them with an operand from `edge`; no numerator larger than
// its denominator (the traversal divides by the dominant component of a direction).
__global__ void check(unsigned long long* counts, const uint32_t* edge, uint32_t edges) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t k = first; k < (1ull << 32); k += stride) {
        const float x = __uint_as_float((uint32_t)k);
        differs(over_pi(x), __fdiv_rn(x, PI_F), counts);
    }
    for (uint64_t k = first; k < 256u; k += stride) differs(byte_over_255((uint32_t)k), __fdiv_rn((float)k, 255.0f), counts + 1);
    for (uint64_t k = first; k < 65536u; k += stride)
        differs(unpack_snorm16((uint32_t)k), fmaxf(__fdiv_rn((float)(int16_t)(uint16_t)k, 32767.0f), -1.0f), counts + 2);
    uint32_t s = (uint32_t)first * 747796405u + 2891336453u;
    auto next = [&] {
        s ^= s << 13;
        s ^= s >> 17;
        s ^= s << 5;
        return s;
    };
    if (s == 0u) s = 1u;
    for (uint64_t k = first; k < (1ull << 26); k += stride) {
        uint32_t a = next(), b = next();
        if ((k & 7u) == 0u) a = edge[next() % edges];
        if ((k & 7u) == 1u) b = edge[next() % edges];
        double x = (double)__uint_as_float(a), y = (double)__uint_as_float(b);
        if (fabs(x) > fabs(y)) {
            const double t = x;
            x = y;
            y = t;
        }
        const double got = quotient_f64(x, y, __ddiv_rn(1.0, y)), want = __ddiv_rn(x, y);
        if (__double_as_longlong(got) != __double_as_longlong(want) && !(got != got && want != want))
            atomicAdd(counts + 3, 1ull);
    }
}

extern "C" int run(unsigned long long* host, const uint32_t* edge_host, uint32_t edges) {
    unsigned long long* counts = nullptr;
    uint32_t* edge = nullptr;
    cudaError_t e = cudaMalloc(&counts, 4 * sizeof(*counts));
    if (e == cudaSuccess) e = cudaMalloc(&edge, edges * sizeof(*edge));
    if (e == cudaSuccess) e = cudaMemset(counts, 0, 4 * sizeof(*counts));
    if (e == cudaSuccess) e = cudaMemcpy(edge, edge_host, edges * sizeof(*edge), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        check<<<1184, 256>>>(counts, edge, edges);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(host, counts, 4 * sizeof(*counts), cudaMemcpyDeviceToHost);
    cudaFree(counts);
    cudaFree(edge);
    return (int)e;
}
