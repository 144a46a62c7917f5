// Compares the conversions on bit patterns (csrc/pair_bits.cuh) with the conversions themselves, bit for
// bit: `pair_bits_check host N` on the CPU, `pair_bits_check device N` on the GPU, N random patterns of
// each kind.  Prints the number of patterns and of differences.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "pair_bits.cuh"

using namespace amdg;

namespace {

__host__ __device__ uint64_t mix(uint64_t x) {  // the finaliser of splitmix64
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__host__ __device__ bool same(float a, float b) { return a != a ? b != b : bits_of(a) == bits_of(b); }

// differences of pattern d
__host__ __device__ int check(double d) {
    float hi, lo;
    split_bits(d, hi, lo);
    const float h = float(d);
    const float l = float(d - double(h));
    int bad = same(hi, h) && same(lo, l) ? 0 : 1;
    const float parts[2] = {h, l};
    for (float f : parts) {
        const double w = widen_bits(f), x = double(f);
        if (x != x ? w == w : bits_of(w) != bits_of(x)) ++bad;
    }
    return bad;
}

// pattern i of kind: 0 all bits; 1 exponents from below the smallest float to above the largest; 2 those
// half way between two floats, just above and just below; 3 the same with a high part of all ones; 4 low
// parts that are themselves half way between two floats
__host__ __device__ double pattern(uint64_t i, int kind) {
    const uint64_t r = mix(5 * i + uint64_t(kind));
    if (kind == 0) return double_of(r);
    uint64_t b = (r & 0x800fffffffffffffull) | (uint64_t(1023 - 165 + (r >> 52) % 300) << 52);
    if (kind == 2 || kind == 3) {
        const uint64_t tail[3] = {0x10000000ull, 0x10000001ull, 0x0fffffffull};
        b = (b & ~0x1fffffffull) | tail[mix(r) % 3];
        if (kind == 3) b |= 0xfffffe0000000ull;
    }
    if (kind == 4) b = (b & ~0xfull) | (mix(r) & 1 ? 0x8ull : 0x4ull);
    return double_of(b);
}
constexpr int kKinds = 5;

__host__ __device__ double special(int i) {
    const uint64_t b[] = {0x0ull, 0x7ff0000000000000ull, 0x7ff8000000000000ull, 0x1ull, 0x000fffffffffffffull,
                          0x0010000000000000ull, 0x36a0000000000000ull, 0x3690000000000000ull, 0x3690000000000001ull,
                          0x369fffffffffffffull, 0x3800000000000000ull, 0x380fffffe0000000ull, 0x380ffffff0000000ull,
                          0x47efffffe0000000ull, 0x47efffffefffffffull, 0x47effffff0000000ull, 0x47f0000000000000ull,
                          0x7fefffffffffffffull, 0x3ff0000000000000ull, 0x3ff0000010000000ull, 0x3ff0000030000000ull,
                          0x3810000000000000ull, 0x3810000000000001ull, 0x39b0000000000001ull, 0x3990000008000000ull};
    const int n = int(sizeof(b) / sizeof(b[0]));
    return i < 2 * n ? double_of(b[i / 2] | (i & 1 ? 0x8000000000000000ull : 0ull)) : 0.0;
}
constexpr int kSpecials = 50;

__global__ void check_kernel(uint64_t n, unsigned long long* bad) {
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    int k = 0;
    if (i < n)
        for (int kind = 0; kind < kKinds; ++kind) k += check(pattern(i, kind));
    if (i < kSpecials) k += check(special(int(i)));
    if (k) atomicAdd(bad, (unsigned long long)k);
}

}  // namespace

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    const uint64_t n = std::strtoull(argv[2], nullptr, 10);
    unsigned long long bad = 0;
    if (std::strcmp(argv[1], "host") == 0) {
        for (uint64_t i = 0; i < n; ++i)
            for (int kind = 0; kind < kKinds; ++kind) bad += check(pattern(i, kind));
        for (int i = 0; i < kSpecials; ++i) bad += check(special(i));
    } else {
        unsigned long long* d = nullptr;
        if (cudaMalloc(&d, sizeof(bad)) != cudaSuccess || cudaMemset(d, 0, sizeof(bad)) != cudaSuccess) return 3;
        check_kernel<<<unsigned((n + 255) / 256), 256>>>(n, d);
        if (cudaMemcpy(&bad, d, sizeof(bad), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
        cudaFree(d);
    }
    std::printf("%llu patterns %llu differences\n", (unsigned long long)(n * kKinds + kSpecials), bad);
    return bad ? 1 : 0;
}
