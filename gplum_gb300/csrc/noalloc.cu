// Soft force for callers that cannot allocate device memory.
//
// Some hosts of this library run it inside a runtime that owns every device
// allocation (a memory arena or pool handed out by another framework, or a
// sandboxed process in which cudaMalloc is not permitted).  Those callers can
// pass device buffers they already have, but they cannot let the library call
// cudaMalloc/cudaFree.  p3t_soft_force_noalloc serves them: the caller passes
// the body records, the interaction lists, the superparticles and the output
// buffer (all device-accessible), and the only scratch the computation needs
// -- the packed body records the soft kernel gathers, their FP32 splits, the
// packed superparticles, and one status word -- lives in file-scope static
// device arrays.
//
// Those arrays exist once per GPU that loads this library and stay allocated
// until the process exits (P3T_NOALLOC_MAX_BODIES x 80 B = 5 MiB,
// P3T_NOALLOC_MAX_SPJ x 64 B = 4 MiB, plus the status word and the gate).  Their
// device addresses are looked up once per device, on that device's first call
// (cudaGetSymbolAddress with the device current).  A call waits for its stream
// (for its status), so it cannot be made on a stream that is being captured into a
// CUDA graph.
// Every call shares the arrays: calls that overlap on the GPU (different
// streams, or several host threads) race on them and must be serialised by
// the caller.  The caller's CSR offsets are checked on the device before any
// list is read through them (status bit 2); list entries out of range are
// clamped by the kernel and reported the same way.
#include <cstdio>
#include <mutex>

#include "../../include/gplum_p3t.h"
#include "p3t_common.cuh"
#include "p3t_soft.cuh"

namespace {

static __device__ __align__(256) p3t::SoftPtcl g_noalloc_bodies[P3T_NOALLOC_MAX_BODIES];
static __device__ __align__(256) p3t::SoftSplit g_noalloc_split[P3T_NOALLOC_MAX_BODIES];
static __device__ __align__(256) p3t::SpjPack g_noalloc_spj[P3T_NOALLOC_MAX_SPJ];
static __device__ __align__(256) int g_noalloc_status[2];  // the status word, the gate

struct DeviceScratch {
    bool ready = false;
    p3t::SoftPtcl *bodies = nullptr;
    p3t::SoftSplit *split = nullptr;
    p3t::SpjPack *spj = nullptr;
    int *status = nullptr;
    int calls = 0;             // the gate is closed for a call when it holds the call's number
    bool writes_host = false;  // the device writes any host memory in place
};
constexpr int MAX_DEVICES = 64;
DeviceScratch g_scratch[MAX_DEVICES];
std::mutex g_scratch_mu;

// Device addresses of the static arrays for the current device.  The array
// names are host-side stand-ins: only these looked-up addresses may be
// passed to kernels.
int scratch_for_current_device(DeviceScratch **out, int *call) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return -(int)e;
    if (dev < 0 || dev >= MAX_DEVICES) return -(int)cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    DeviceScratch &s = g_scratch[dev];
    if (!s.ready) {
        e = cudaGetSymbolAddress((void **)&s.bodies, g_noalloc_bodies);
        if (e != cudaSuccess) return -(int)e;
        e = cudaGetSymbolAddress((void **)&s.split, g_noalloc_split);
        if (e != cudaSuccess) return -(int)e;
        e = cudaGetSymbolAddress((void **)&s.spj, g_noalloc_spj);
        if (e != cudaSuccess) return -(int)e;
        e = cudaGetSymbolAddress((void **)&s.status, g_noalloc_status);
        if (e != cudaSuccess) return -(int)e;
        int v = 0;
        s.writes_host = cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccessUsesHostPageTables, dev) == cudaSuccess && v &&
                        cudaDeviceGetAttribute(&v, cudaDevAttrHostNativeAtomicSupported, dev) == cudaSuccess && v;
        s.ready = true;
    }
    s.calls = s.calls == 2147483647 ? 1 : s.calls + 1;
    *call = s.calls;
    *out = &s;
    return 0;
}

}  // namespace

extern "C" int p3t_soft_force_noalloc(int n, const void *epj, int n_group, const int *i_off, const int *i_idx,
                                      const int *j_off, const int *j_idx, const int *s_off, const int *s_idx,
                                      const void *spj, int n_spj, double eps2, int trace_mode, void *force,
                                      void *stream) {
    if (n < 0 || n > P3T_NOALLOC_MAX_BODIES) {
        std::fprintf(stderr,
                     "[gplum_p3t] p3t_soft_force_noalloc: %d bodies exceed the static scratch of %d bodies; "
                     "use p3t_soft_force_host or the resident path for larger systems\n",
                     n, P3T_NOALLOC_MAX_BODIES);
        return -(int)cudaErrorInvalidValue;
    }
    if (n_spj > P3T_NOALLOC_MAX_SPJ) {
        std::fprintf(stderr,
                     "[gplum_p3t] p3t_soft_force_noalloc: %d superparticles exceed the static scratch of %d; "
                     "use p3t_soft_force_host or the resident path for larger systems\n",
                     n_spj, P3T_NOALLOC_MAX_SPJ);
        return -(int)cudaErrorInvalidValue;
    }
    if (n_group < 0 || n_spj < 0 || (trace_mode != 0 && trace_mode != 1)) return -(int)cudaErrorInvalidValue;
    if (n == 0 || n_group == 0) return 0;
    // every buffer the kernels will read or write must be there
    if (!epj || !force || !i_off || !i_idx || !j_off || !j_idx || !s_off || !s_idx || (n_spj > 0 && !spj))
        return -(int)cudaErrorInvalidValue;
    DeviceScratch *s = nullptr;
    int call = 0;
    int r = scratch_for_current_device(&s, &call);
    if (r) return r;
    cudaStream_t st = (cudaStream_t)stream;
    // The kernels set the bits in this call's own word where the device reaches the
    // host's memory; elsewhere in the static word, which keeps the previous call's
    // value: clear it.
    cudaError_t e = cudaSuccess;
    int h = 0;
    int *const status = s->writes_host ? &h : s->status;
    if (!s->writes_host && (e = cudaMemsetAsync(s->status, 0, sizeof(int), st)) != cudaSuccess) return -(int)e;
    // one launch packs bodies and superparticles and checks the offsets; a
    // violation closes the gate, and no list is read through a malformed offset.
    // The host waits once, for the result: 20,000 bodies 112 -> 73 us a call
    // against a launch for each of the check (with a wait), the bodies, their
    // splits and the superparticles.
    p3t::PackArgs K{};
    K.one.epj = epj;
    K.one.nj = n;
    K.one.spj = spj;
    K.one.ns = n_spj;
    K.n_walk = 1;
    K.ptcl = s->bodies;
    K.jsplit = s->split;
    K.spjp = s->spj;
    K.eps2 = (float)eps2;
    K.trace_mode = trace_mode;
    K.chk_i_off = i_off;
    K.chk_j_off = j_off;
    K.chk_s_off = s_off;
    K.chk_groups = n_group;
    K.chk_n = n;
    K.status = status;
    K.gate_call = call;
    K.gate = s->status + 1;
    if ((e = p3t::launch_pack_walks(K, (long long)n + n_spj, st)) != cudaSuccess) {
        cudaStreamSynchronize(st);
        return -(int)e;
    }
    p3t::SoftArgs A{};
    A.i_off = i_off;
    A.i_idx = i_idx;
    A.j_off = j_off;
    A.j_idx = j_idx;
    A.s_off = s_off;
    A.s_idx = s_idx;
    A.group_order = nullptr;
    A.n_group = n_group;
    A.iptcl = s->bodies;
    A.n_iptcl = n;
    A.ptcl = s->bodies;
    A.n_ptcl = n;
    A.spj = (const p3t::SPJRec *)spj;
    A.n_spj = n_spj;
    A.eps2 = (float)eps2;
    A.eps2_d = eps2;
    A.trace_mode = trace_mode;
    A.accumulate = 0;
    A.force = (p3t::ForceRec *)force;
    A.acc64 = nullptr;
    A.cand = nullptr;
    A.cand_cap = 0;
    A.status = status;
    A.jsplit = s->split;
    A.isplit = s->split;
    A.spjp = s->spj;
    A.packed = 1;
    A.gate = s->status + 1;
    A.gate_call = call;
    // the launch shape the setters chose (the same as the allocating path's)
    A.t_ipt2 = p3t::g_soft_shape[0];
    A.t_s1 = p3t::g_soft_shape[1];
    A.t_s2 = p3t::g_soft_shape[2];
    A.occ = p3t::g_soft_shape[3];
    e = launch_soft(A, 0, false, st);
    if (e == cudaSuccess && !s->writes_host) e = cudaMemcpyAsync(&h, s->status, sizeof(int), cudaMemcpyDeviceToHost, st);
    // (also after an error: nothing of this call may still write its word)
    const cudaError_t w = cudaStreamSynchronize(st);
    if (e != cudaSuccess || w != cudaSuccess) return -(int)(e != cudaSuccess ? e : w);
    return *(volatile int *)&h;
}
