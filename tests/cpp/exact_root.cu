// Compares root_reciprocal and quotient (msim_device.cuh) with the correctly rounded
// intrinsics on the device and prints the number of mismatches of each:
//   root / reciprocal: every float d2 in [2^-80, 2^80];
//   quotient: random operands, and operands whose quotient lies as near to the middle
//   between two floats as a quotient can (b m = c mod 2^24 for an odd 25-bit middle m
//   and a small c, so that a = (b m - c) / 2^24 is m b up to c).
#include <cstdint>
#include <cstdio>

#include "msim_device.cuh"

using namespace msim;

__global__ void check_root(uint32_t lo, uint32_t count, unsigned long long* bad) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const float d2 = __uint_as_float(lo + i);
        float len, v;
        root_reciprocal(d2, len, v);
        const float ref = __fsqrt_rn(d2);
        if (__float_as_uint(len) != __float_as_uint(ref)) atomicAdd(&bad[0], 1ull);
        if (__float_as_uint(v) != __float_as_uint(__frcp_rn(ref))) atomicAdd(&bad[1], 1ull);
    }
}

__device__ void check_one(float a, float b, unsigned long long* bad) {
    const float q = quotient(a, b, __frcp_rn(b));
    if (__float_as_uint(q) != __float_as_uint(__fdiv_rn(a, b))) atomicAdd(bad, 1ull);
}

__global__ void check_quotients(uint32_t rounds, unsigned long long* bad) {
    const uint64_t t = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t k = 0; k < rounds; k++) {
        const uint64_t x = d_draw(1, 1, t * rounds + k), y = d_draw(1, 2, t * rounds + k);
        // b in [2^-40, 2^40), a in [2^-58, 2^40) of either sign, and zero
        const float b = __uint_as_float(((87u + (uint32_t)(x % 80u)) << 23) | (uint32_t)((x >> 32) & 0x7fffffu));
        float a = __uint_as_float(((69u + (uint32_t)(y % 98u)) << 23) | (uint32_t)((y >> 32) & 0x7fffffu));
        if (fabsf(a) > 2.f * b) a = __fmul_rn(b, __uint_as_float(0x3f800000u | (uint32_t)((y >> 32) & 0x7fffffu)) - 1.f);
        if ((y >> 63) && a != 0.f) a = -a;  // a difference of equal numbers is +0
        if (fabsf(a) >= 3.5e-18f || a == 0.f) check_one(a, b, &bad[2]);
        // nearest to a middle: m odd in [2^24, 2^25), c = +-1 .. +-8
        const uint32_t m = (uint32_t)(0x1000000u | (x & 0xffffffu) | 1u);
        uint32_t inv = m;  // m^-1 mod 2^32 by Newton's iteration
        for (int i = 0; i < 4; i++) inv *= 2u - m * inv;
        const int32_t c = (int32_t)((y & 7u) + 1u) * ((y & 8u) ? -1 : 1);
        const uint32_t bi = ((uint32_t)c * inv) & 0xffffffu;
        if (bi < 0x800000u) continue;
        const int64_t ai = ((int64_t)bi * (int64_t)m - c) >> 24;
        const float af = (float)ai, bf = (float)bi;
        if ((int64_t)af != ai) continue;  // more than 24 bits
        atomicAdd(&bad[4], 1ull);
        check_one(af * 9.5367431640625e-7f, bf, &bad[3]);
    }
}

int main() {
    unsigned long long* bad = nullptr;
    unsigned long long h[5] = {};
    if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess || cudaMemset(bad, 0, sizeof(h)) != cudaSuccess) return 2;
    check_root<<<152 * 16, 256>>>(0x17800000u, 0x50000001u, bad);  // 2^-80 .. 2^80
    check_quotients<<<152 * 16, 256>>>(400u, bad);
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess)
        return 2;
    std::printf("root %llu reciprocal %llu quotient %llu middle %llu of %llu\n", h[0], h[1], h[2], h[3], h[4]);
    cudaFree(bad);
    return 0;
}
