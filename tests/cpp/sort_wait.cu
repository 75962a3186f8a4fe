// One pass of the key sort whose block is given the second tile while the first
// is never taken: its look-back must give up after the counted polls, report it
// and leave.  Prints the status word, the milliseconds it took and how many of
// the output keys are not keys of the input.
#include <cstdio>
#include <vector>

#include "scan_sort.cu"

using namespace sphgpu;

int main()
{
    constexpr int n = 2 * RS_TILE, tiles = 2;
    std::vector<uint64_t> k(n);
    for(int i = 0; i < n; ++i) k[i] = (uint64_t)(i * 2654435761u % 251u);
    uint64_t *kin = nullptr, *kout = nullptr;
    uint32_t *vin = nullptr, *vout = nullptr;
    unsigned *hist = nullptr, *next = nullptr, *status = nullptr;
    int* gave_up = nullptr;
    const unsigned second = 1;
    cudaMalloc(&kin, n * 8);
    cudaMalloc(&kout, n * 8);
    cudaMalloc(&vin, n * 4);
    cudaMalloc(&vout, n * 4);
    cudaMalloc(&hist, 256 * 4);
    cudaMalloc(&next, 4);
    cudaMalloc(&status, tiles * 256 * 4);
    cudaMalloc(&gave_up, 4);
    cudaMemcpy(kin, k.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemset(kout, 0, n * 8);
    cudaMemset(vin, 0, n * 4);
    cudaMemset(hist, 0, 256 * 4);
    cudaMemset(status, 0, tiles * 256 * 4);
    cudaMemset(gave_up, 0, 4);
    cudaMemcpy(next, &second, 4, cudaMemcpyHostToDevice);
    k_rs_hist<<<1, RS_BLOCK>>>(kin, n, 1, hist);
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaEventRecord(a);
    k_rs_pass<<<1, RS_BLOCK>>>(kin, vin, kout, vout, n, 0, hist, next, status, gave_up);
    cudaEventRecord(b);
    int flag = -1;
    if(cudaMemcpy(&flag, gave_up, 4, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    std::vector<uint64_t> o(n);
    if(cudaMemcpy(o.data(), kout, n * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    int strange = 0;
    for(uint64_t x : o) strange += x >= 251 ? 1 : 0;
    std::printf("%d %.1f %d\n", flag, ms, strange);
    return 0;
}
