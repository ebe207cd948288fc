// Host build of the device runtime (volume-compressor_gb300/csrc/vc_device.cu)
// over a stand-in for the CUDA runtime, in which device memory is host memory and
// every queued operation is done at once, and over stand-ins for the launches,
// which leave what the kernels would. Test infrastructure for outcomes that a
// kernel cannot be made to have.
//
// usage: host_device <malformed atom or -1> <a wait ran out: 0 / 1> <output MiB>;
// prints the status of a decode of whole 32-voxel layers into host memory.
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <cuda_runtime.h>

static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline uint32_t __byte_perm(uint32_t, uint32_t, uint32_t) { return 0; }
static inline uint32_t __funnelshift_l(uint32_t, uint32_t, uint32_t) { return 0; }
template <class T> static inline T __ldg(const T *p) { return *p; }
static inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
static inline bool __any_sync(uint32_t, bool v) { return v; }
static inline uint32_t __reduce_max_sync(uint32_t, uint32_t v) { return v; }

#include "vc_device.cu"

// ---- launches
static int64_t g_malformed;
static int g_gave_up;
static int g_transforms;
namespace vcg {
void launch_decode_front(const DecodeJob &J, int, cudaStream_t, const StageEvents *) {
    if (g_malformed >= 0) *J.err = (uint32_t)g_malformed;
}
void launch_idct(const DecodeJob &J, int, cudaStream_t, uint64_t, uint64_t) {
    ++g_transforms;
    if (g_gave_up) *J.fail = 1;
}
void enc_tables(EncTables *, const vcd_tables *) {}
}  // namespace vcg
extern "C" void vch_tables(vcd_tables *) {}

// ---- the CUDA runtime
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof *p);
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaPeekAtLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = 1ull << 34; return cudaSuccess; }
// all host memory is pinned: large outputs take the slabs, without the bounce ring
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
}

int main(int argc, char **argv) {
    if (argc < 4) return 2;
    g_malformed = atoll(argv[1]);
    g_gave_up = atoi(argv[2]);
    const uint64_t bytes = strtoull(argv[3], nullptr, 10) << 20;
    if (vcd_init()) return 3;
    // atoms of 32 KiB, 64 a layer
    const uint64_t n = bytes / 32768;
    vcd_atom *atoms = (vcd_atom *)calloc(n, sizeof(vcd_atom));
    for (uint64_t i = 0; i < n; ++i) atoms[i].kind = VCD_PRESENT, atoms[i].len = 100;
    vcd_archive d;
    memset(&d, 0, sizeof d);
    vcd_region r;
    memset(&r, 0, sizeof r);
    r.acx = r.acy = 8;
    r.atoms = atoms;
    r.bnx = r.bny = 8;
    r.bnz = (uint32_t)(n / 64);
    r.x1 = r.y1 = 256;
    r.z1 = 32 * r.bnz;
    r.n_atoms = n;
    r.present = n;
    r.cap_total = n;
    r.max_len = 100;
    uint8_t *out = (uint8_t *)calloc(1, bytes);
    const int s = vcd_decode_region(&d, &r, nullptr, out, bytes);
    printf("%d %d\n", s, g_transforms);
    free(out);
    free(atoms);
    return 0;
}
