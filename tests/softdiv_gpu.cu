// Checks rcp_i, div_of and sqrt_i (fauxgl_gb300/csrc/fgc_softdiv.cuh) against
// __drcp_rn, __ddiv_rn and __dsqrt_rn on the GPU, bit for bit: every FP32 seed
// (all 2^23 truncated significands, both parities for the root) with the
// lowest, highest and a seeded low part, and operands at the ends of the
// exponent range. Prints "ok <cases>" or the first mismatch and exits 1.
// Build: nvcc -gencode arch=compute_103a,code=sm_103a -O3 --fmad=false -std=c++17 softdiv_gpu.cu
#include <cstdint>
#include <cstdio>

#include "../fauxgl_gb300/csrc/fgc_softdiv.cuh"

using namespace fgc;

__device__ uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ bool same(double a, double b) { return (a != a && b != b) || fj_bits(a) == fj_bits(b); }

__global__ void check(unsigned long long* bad, unsigned long long* first) {
    const uint64_t n = 1ull << 23;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        for (int k = 0; k < 8; k++) {
            const uint64_t r = mix(i * 8 + k), r2 = mix(r);
            const uint64_t low = k == 0 ? 0 : k == 1 ? 0x1fffffffull : r & 0x1fffffffull;
            uint64_t e = 1003 + (r >> 40) % 40;
            if (k == 7) e = (r >> 40) & 1 ? (r >> 41) % 4 : 2047 - (r >> 41) % 4;  // zeros, subnormals, infinities, NaN too
            const double w = fj_double(((r >> 63) << 63) | (e << 52) | (i << 29) | low);
            uint64_t ex = k == 6 ? (r2 >> 40) % 2048 : 1003 + (r2 >> 40) % 40;
            double x = fj_double(((r2 >> 63) << 63) | (ex << 52) | (r2 & 0x000fffffffffffffull));
            if (k == 3) x = __dmul_rn(w, 1.0 + (double)(r2 % 64) * 0x1p-52);
            if (k == 4) x = __dmul_rn(w, (double)(r2 % 4096));
            const SoftRcp s = soft_rcp(w);
            const double a = fj_double(fj_bits(w) & 0x7fffffffffffffffull);
            if (!same(rcp_of(w, s), __drcp_rn(w)) || !same(div_of(x, w, s), __ddiv_rn(x, w)) ||
                !same(sqrt_i(a), __dsqrt_rn(a)) || !same(sqrt_i(w), __dsqrt_rn(w))) {
                if (atomicAdd(bad, 1ull) == 0) {
                    first[0] = fj_bits(w);
                    first[1] = fj_bits(x);
                }
            }
        }
    }
}

int main() {
    unsigned long long *d = nullptr, h[3] = {0, 0, 0};
    if (cudaMalloc(&d, 24) != cudaSuccess || cudaMemset(d, 0, 24) != cudaSuccess) return 2;
    check<<<1216, 256>>>(d, d + 1);
    if (cudaMemcpy(h, d, 24, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    cudaFree(d);
    if (h[0]) {
        printf("%llu mismatches, the first with w = %016llx, x = %016llx\n", h[0], h[1], h[2]);
        return 1;
    }
    printf("ok %llu\n", 8ull << 23);
    return 0;
}
