// Check on the GPU that the octahedral mapping of the atlas lookups (oct_uv in
// vulkanexp_gb300/csrc/shade.cuh), which forms its quotients from one refined
// reciprocal, has the bits of the mapping with divisions: directions of length
// one from random normals, along the axes and in their planes, and with
// components down to the smallest normal number.
#include <cstdio>

#include "../../vulkanexp_gb300/csrc/shade.cuh"

using namespace ddgi;

namespace {

__device__ uint32_t mixed(uint32_t x) {  // spreads a counter: products with odd numbers, folded
    x = (x + 1u) * 0x9E3779B9u;
    x = (x ^ (x >> 15)) * 0x2545F491u;
    x = (x ^ (x >> 13)) * 0x9E3779B9u;
    return x ^ (x >> 16);
}

__device__ float2 by_division(float3 d) {
    const float sum = __fadd_rn(__fadd_rn(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
    float x = __fdiv_rn(d.x, sum), y = __fdiv_rn(d.y, sum);
    if (d.z < 0.0f) {
        const float fx = d.x != 0.0f ? copysignf(1.0f - fabsf(y), d.x) : 0.0f;
        const float fy = d.y != 0.0f ? copysignf(1.0f - fabsf(x), d.y) : 0.0f;
        x = fx;
        y = fy;
    }
    return make_float2(fmaf(x, 0.5f, 0.5f), fmaf(y, 0.5f, 0.5f));
}

__global__ void k_check(uint32_t n, uint32_t* differ, float3* first) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float v[3];
    for (uint32_t k = 0; k < 3; ++k) {
        const uint32_t h = mixed(3u * i + k), kind = mixed(h) % 16u;
        v[k] = (float)(int)h * 0x1p-31f;
        if (kind == 0) v[k] = 0.0f;
        if (kind == 1) v[k] = v[k] < 0.0f ? -1.0f : 1.0f;
        if (kind == 2) v[k] = ldexpf(v[k], -(int)(mixed(h + 1u) % 126u));
    }
    const float len = sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    if (!(len > 1e-3f)) return;
    const float3 d = f3(v[0] / len, v[1] / len, v[2] / len);
    const float2 a = oct_uv(d), b = by_division(d);
    if (__float_as_uint(a.x) != __float_as_uint(b.x) || __float_as_uint(a.y) != __float_as_uint(b.y))
        if (atomicAdd(differ, 1u) == 0u) *first = d;
}

}  // namespace

int main() {
    const uint32_t n = 1u << 26;
    uint32_t* differ = nullptr;
    float3* first = nullptr;
    if (cudaMalloc(&differ, sizeof(uint32_t)) != cudaSuccess || cudaMalloc(&first, sizeof(float3)) != cudaSuccess) return 2;
    cudaMemset(differ, 0, sizeof(uint32_t));
    cudaMemset(first, 0, sizeof(float3));
    k_check<<<n / 256, 256>>>(n, differ, first);
    uint32_t count = 0;
    float3 d;
    if (cudaMemcpy(&count, differ, sizeof(count), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    if (cudaMemcpy(&d, first, sizeof(d), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("%u directions, %u differ\n", n, count);
    if (count) {
        std::printf("first: %a %a %a\n", d.x, d.y, d.z);
        return 1;
    }
    std::printf("all ok\n");
    return 0;
}
