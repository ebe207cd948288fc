// The CTA of the tensor-core inverse transform (volume-compressor_gb300/csrc/
// idct_mma.cuh) with one of its roles slower than the others wait, built with a
// short limit on the waits (VCG_WAIT_TRIES). Test infrastructure: the kernel ends
// in every mode, with the fail word set in all but the first.
//   0 nothing slow, 1 feeders that are not there, 2 a feeder that pauses at its
//   second 32 atoms, 3 a pause at every output of the 16 warps, 4 of one of them
// Output: "<mode> <CUDA error> <fail word>" per mode.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "dct32.cuh"
#include "kernels.cuh"
#include "idct_mma.cuh"

using namespace vcg;

constexpr uint32_t kB = (uint32_t)((kIdctTileBytes + 1023) & ~(size_t)1023);
constexpr size_t kSmem = 1024 + kB + kMmaB + kMmaRing;
constexpr uint32_t kAtoms = 80, kEntries = 40;

__device__ void pause_ms(uint32_t ms) {
    uint64_t t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    while (t - t0 < 1000000ull * ms);
}

__global__ void __launch_bounds__(kMmaCta, 1) k_give_up(const uint32_t *list, const vcd_dq *dq, const uint32_t *place,
                                                        int mode, uint32_t *fail, uint32_t *sums) {
    extern __shared__ uint8_t dyn[];
    __shared__ __align__(16) MmaShared M;
    uint8_t *A = dyn + ((1024u - (smem_u32(dyn) & 1023u)) & 1023u), *B = A + kB, *ring = B + kMmaB;
    const int tid = threadIdx.x;
    mma_setup(M, B);
    if (tid >= kMmaFeed) {
        if (mode != 1)
            mma_feed(M, ring, dq, place, [&](uint32_t i, MmaAtom &a) {
                if (mode == 2 && i >= 32u) pause_ms(50);
                if (i >= kAtoms) return false;
                a.src = list;
                a.n = kEntries;
                a.tensor = 1;
                return true;
            });
    } else if (tid >= kMmaIssuer) {
        if (tid == kMmaIssuer) mma_issue(M, umma_lo(smem_u32(A)), umma_lo(smem_u32(B)));
    } else {
        uint32_t sum = 0;
        const bool ok = mma_atoms(
            A, M, ring,
            [&](const MmaAtom &, int, int, int, uint32_t (&o)[16]) {
                for (int k = 0; k < 16; ++k) sum += o[k];
                if (mode == 3 || (mode == 4 && (tid >> 5) == 5)) pause_ms(10);
            },
            [&](const MmaAtom &, uint8_t *) {});
        sums[blockIdx.x * kMmaThreads + tid] = sum;
        if (!ok) atomicExch(fail, 1u);
    }
    mma_release(M);
    if (tid == 0 && M.starved) atomicExch(fail, 1u);
}

template <class T>
static T *device(const T *src, size_t n) {
    T *p = nullptr;
    if (cudaMalloc(&p, n * sizeof(T)) || cudaMemcpy(p, src, n * sizeof(T), cudaMemcpyHostToDevice)) return nullptr;
    return p;
}

int main() {
    static uint32_t list[kEntries], place[32768], zero[2 * kMmaThreads];
    static vcd_dq dq;
    for (uint32_t i = 0; i < kEntries; ++i) list[i] = i | (1u << 16);
    for (uint32_t p = 0; p < 32768; ++p) place[p] = ((p * 128u) & 0x1FFFFu) | ((p >> 10) << 1);   // even, below 131,072, class 0
    const uint32_t *dlist = device(list, kEntries), *dplace = device(place, 32768);
    const vcd_dq *ddq = device(&dq, 1);
    uint32_t *fail = device(zero, 1), *sums = device(zero, 2 * kMmaThreads);
    if (!dlist || !dplace || !ddq || !fail || !sums) return 3;
    if (cudaFuncSetAttribute((const void *)k_give_up, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem)) return 4;
    for (int mode = 0; mode < 5; ++mode) {
        cudaMemset(fail, 0, 4);
        k_give_up<<<2, kMmaCta, kSmem>>>(dlist, ddq, dplace, mode, fail, sums);
        uint32_t f = 0;
        const cudaError_t e = cudaMemcpy(&f, fail, 4, cudaMemcpyDeviceToHost);
        printf("%d %d %u\n", mode, (int)e, f);
        if (e) return 1;
    }
    return 0;
}
