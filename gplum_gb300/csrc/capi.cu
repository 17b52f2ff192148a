// C ABI of the P3T soft-force path (declarations and contracts in
// include/gplum_p3t.h).  One process-wide context bound to one GPU.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "../../include/gplum_p3t.h"
#include "p3t_capi_internal.cuh"
#include "p3t_common.cuh"
#include "p3t_soft.cuh"

namespace p3t {

Context *g_ctx = nullptr;
static std::mutex g_mu;

int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return 0;
    std::fprintf(stderr, "[gplum_p3t] CUDA error %d: %s\n", (int)e, cudaGetErrorString(e));
    return -(int)e;
}

Context *ctx_get(int device) {
    if (g_ctx) return g_ctx;
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_ctx) return g_ctx;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= device || device < 0) return nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return nullptr;
    Context *c = new Context();
    c->device = device;
    // the library stream one step below the highest priority: the hard
    // part's side launches that must hold SMs from the start (the lone form)
    // take the highest, so the CTA dispatcher places theirs before the
    // persistent bundle CTAs; work queued beside it at the lowest (the
    // isolated bodies' drift) only takes SMs the step's own launches leave free
    int prio_lo = 0, prio_hi = 0;
    cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi);
    const int prio = (prio_hi < prio_lo) ? prio_hi + 1 : prio_hi;
    if (cudaStreamCreateWithPriority(&c->stream, cudaStreamNonBlocking, prio) != cudaSuccess ||
        cudaStreamCreateWithPriority(&c->side, cudaStreamNonBlocking, prio_hi) != cudaSuccess ||
        cudaStreamCreateWithPriority(&c->pair, cudaStreamNonBlocking, prio) != cudaSuccess) {
        delete c;
        return nullptr;
    }
    if (cudaMalloc(&c->status, sizeof(int)) != cudaSuccess) {
        delete c;
        return nullptr;
    }
    cudaMemsetAsync(c->status, 0, sizeof(int), c->stream);
    int v = 0;
    c->reads_host = cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device) == cudaSuccess && v;
    // default parameters: FPGrav defaults, src/particle.h:917-961
    const double def[21] = {0., 0., 1., 1. / 32., 1. / 8192., 0.01, 0.001, 0.01, 0.001, 1.,
                            0.5, 2., 8., 1., 4., 1., 4., 0., 0., 0., 5.049667e6};
    std::memcpy(c->params, def, sizeof(def));
    g_ctx = c;
    return c;
}

int grow_raw(void **p, size_t *cap, size_t bytes) {
    if (bytes <= *cap) return 0;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    size_t nb = bytes + bytes / 4 + 256;
    cudaError_t e = cudaMalloc(p, nb);
    if (e != cudaSuccess) return cuda_status(e);
    *cap = nb;
    return 0;
}

int grow_host(void **p, size_t *cap, size_t bytes) {
    if (bytes <= *cap) return 0;
    if (*p) cudaFreeHost(*p);
    *p = nullptr;
    *cap = 0;
    size_t nb = bytes + bytes / 4 + 256;
    cudaError_t e = cudaMallocHost(p, nb);
    if (e != cudaSuccess) return cuda_status(e);
    *cap = nb;
    return 0;
}

int check_csr(int n_group, const int *off) {
    if (n_group < 0) return ST_BAD_INDEX;
    if (n_group == 0) return (off && off[0] != 0) ? ST_BAD_INDEX : 0;
    if (!off || off[0] != 0) return ST_BAD_INDEX;
    for (int g = 0; g < n_group; g++)
        if (off[g + 1] < off[g]) return ST_BAD_INDEX;
    return 0;
}

int check_lists(int n_group, const int *i_off, const int *i_idx, const int *j_off, const int *j_idx,
                const int *s_off, const int *s_idx, const void *spj, int n_spj) {
    int r = 0;
    if (n_spj < 0 || (n_spj > 0 && !spj)) return ST_BAD_INDEX;
    if ((r = check_csr(n_group, i_off)) || (r = check_csr(n_group, j_off)) || (r = check_csr(n_group, s_off)))
        return r;
    if (n_group == 0) return 0;
    if ((i_off[n_group] > 0 && !i_idx) || (j_off[n_group] > 0 && !j_idx) || (s_off[n_group] > 0 && !s_idx))
        return ST_BAD_INDEX;
    return 0;
}

int read_status(Context *c) {
    int h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, c->status, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_status(e);
    if (h) cudaMemsetAsync(c->status, 0, sizeof(int), c->stream);
    return h;
}

int take_word(WalkSlot &w) {
    if (!w.h_tab) return 0;
    volatile int *const p = (volatile int *)w.h_tab;
    const int h = *p;
    *p = 0;
    return h;
}

bool is_pinned(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

bool device_reads(Context *c, const void *p, size_t align) {
    if ((uintptr_t)p % align) return false;
    if (c->reads_host) return true;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost && a.devicePointer == p;
}

void Uploader::add(void *dst, const void *src, size_t bytes) {
    if (bytes) items.push_back({dst, src, bytes, c->reads_host || is_pinned(src)});
}

// Several arrays in one launch, read where the caller has them: a copy costs the
// host 4 to 8 us, the launch 4 (upload to download of 30,000 bodies in the FP64
// form, with the download's two waits made one, 812 -> 786 us); the
// link's rate is the same (150-205 GB/s).
constexpr int SEGMENTS = 8;
struct CopySegments {
    const char *src[SEGMENTS];
    char *dst[SEGMENTS];
    size_t bytes[SEGMENTS];  // multiples of 4
};
template <class T>
static __device__ __forceinline__ void copy_words(const char *src, char *dst, size_t n) {
    const T *const s = (const T *)src;
    T *const d = (T *)dst;
    const size_t step = (size_t)gridDim.x * blockDim.x;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * step < n; i += 4 * step) {  // four reads in flight
        const T a = s[i], b = s[i + step], c = s[i + 2 * step], e = s[i + 3 * step];
        d[i] = a;
        d[i + step] = b;
        d[i + 2 * step] = c;
        d[i + 3 * step] = e;
    }
    for (; i < n; i += step) d[i] = s[i];
}
static __global__ void __launch_bounds__(256) k_copy_segments(CopySegments A) {
    for (int k = 0; k < SEGMENTS; k++) {
        const size_t wide = ((uintptr_t)A.src[k] | (uintptr_t)A.dst[k]) % 16 == 0 ? A.bytes[k] / 16 : 0;
        copy_words<uint4>(A.src[k], A.dst[k], wide);
        copy_words<unsigned>(A.src[k] + 16 * wide, A.dst[k] + 16 * wide, (A.bytes[k] - 16 * wide) / 4);
    }
}

// The queued items as one launch where the device reads them all in place.
bool Uploader::in_one_launch(int &r) {
    if (!c->reads_host || items.size() < 2 || items.size() > SEGMENTS) return false;
    CopySegments A{};
    size_t total = 0;
    for (size_t k = 0; k < items.size(); k++) {
        const Item &it = items[k];
        if ((uintptr_t)it.src % 4 || (uintptr_t)it.dst % 4 || it.bytes % 4) return false;
        A.src[k] = (const char *)it.src;
        A.dst[k] = (char *)it.dst;
        A.bytes[k] = it.bytes;
        total += it.bytes;
    }
    const int ctas = (int)std::min<size_t>(1216, total / (256 * 64) + 1);  // 64 bytes a thread, eight CTAs an SM at most
    { P3T_COUNT_LAUNCH(); k_copy_segments<<<ctas, 256, 0, c->stream>>>(A); }
    r = cuda_status(cudaGetLastError());
    items.clear();
    return true;
}

int Uploader::issue() {
    int one = 0;
    if (in_one_launch(one)) return one;
    size_t stage = 0;
    for (auto &it : items)
        if (!it.direct) stage += (it.bytes + 255) / 256 * 256;
    int r = grow_host(&c->h_stage, &c->h_stage_cap, stage);
    if (r) return r;
    char *h = (char *)c->h_stage;
    for (auto &it : items) {
        const void *src = it.src;
        if (!it.direct) {
            std::memcpy(h, it.src, it.bytes);
            src = h;
            h += (it.bytes + 255) / 256 * 256;
        }
        r = cuda_status(cudaMemcpyAsync(it.dst, src, it.bytes, cudaMemcpyHostToDevice, c->stream));
        if (r) return r;
    }
    items.clear();
    return 0;
}

int Uploader::flush() {
    const int r = issue(), e = cuda_status(cudaStreamSynchronize(c->stream));
    return r ? r : e;
}

int d2h(Context *c, void *dst, const void *src, size_t bytes) {
    if (bytes == 0) return 0;
    int r = cuda_status(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
    if (r) return r;
    return cuda_status(cudaStreamSynchronize(c->stream));
}

int h2d(Context *c, void *dst, const void *src, size_t bytes) {
    Uploader u(c);
    u.add(dst, src, bytes);
    return u.flush();
}

// Builds SoftArgs over a set of device buffers.
SoftArgs make_args(Context *c, DevSet &d, int n_group, int n_ptcl, int n_spj, bool accumulate) {
    SoftArgs A;
    std::memset(&A, 0, sizeof(A));
    A.i_off = d.i_off.p; A.i_idx = d.i_idx.p; A.j_off = d.j_off.p; A.j_idx = d.j_idx.p;
    A.s_off = d.s_off.p; A.s_idx = d.s_idx.p;
    A.group_order = d.order_valid ? d.order.p : nullptr;
    A.n_group = n_group;
    A.ptcl = d.ptcl.p; A.mass = d.mass.p; A.r_out = d.r_out.p; A.r_search = d.r_search.p;
    A.n_ptcl = n_ptcl;
    A.iptcl = d.ptcl.p; A.i_r_out = d.r_out.p; A.i_r_search = d.r_search.p;
    A.n_iptcl = n_ptcl;
    A.spj = d.spj.p; A.n_spj = n_spj;
    A.eps2 = (float)c->params[0];
    A.eps2_d = c->params[0];
    A.trace_mode = c->trace_mode;
    A.accumulate = accumulate ? 1 : 0;
    A.force = d.force.p;
    A.acc64 = d.acc64.p;
    A.cand = d.cand.p;
    A.cand_cap = c->cand_cap;
    A.status = c->status;
    A.t_ipt2 = c->tiles[0];
    A.t_s1 = c->tiles[1];
    A.t_s2 = c->tiles[2];
    A.occ = c->soft_occ;
    return A;
}

// The EPJ records of a resident problem -> the soft kernels' arrays, read where
// the caller has them if the device can, otherwise from the staged copy that
// `u` (issued first) makes.  The caller waits for the stream before it returns.
static const void *place(Context *c, Uploader &u, void *stage, const void *src, size_t bytes) {
    if (device_reads(c, src, 8)) return src;
    u.add(stage, src, bytes);
    return stage;
}
static PackArgs pack_resident(DevSet &d, int n, const void *epj) {
    PackArgs A{};
    A.one.epj = epj;
    A.one.nj = n;
    A.n_walk = 1;
    A.ptcl = d.ptcl.p; A.mass = d.mass.p; A.r_out = d.r_out.p; A.r_search = d.r_search.p;
    return A;
}

}  // namespace p3t

using namespace p3t;

#define CTX_OR_FAIL(c)                    \
    Context *c = ctx_get(0);              \
    if (!c) return -(int)cudaErrorNoDevice;

namespace p3t {
unsigned long long g_launch_count = 0;
int g_soft_shape[4] = {128, 64, 32, 5};
}

extern "C" {

unsigned long long p3t_launch_count(void) { return __atomic_load_n(&p3t::g_launch_count, __ATOMIC_RELAXED); }

int p3t_init(int device) {
    Context *c = ctx_get(device);
    return c ? 0 : -(int)cudaErrorNoDevice;
}

int p3t_finalize(void) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_ctx) return 0;
    Context *c = g_ctx;
    cudaStreamSynchronize(c->stream);
    c->release();
    cudaFree(c->status);
    cudaStreamSynchronize(c->side);
    cudaStreamDestroy(c->side);
    cudaStreamSynchronize(c->pair);
    cudaStreamDestroy(c->pair);
    cudaStreamDestroy(c->stream);
    delete c;
    g_ctx = nullptr;
    return 0;
}

int p3t_set_params(const double *params21) {
    CTX_OR_FAIL(c);
    std::memcpy(c->params, params21, 21 * sizeof(double));
    c->params_version++;
    return 0;
}

int p3t_set_soft_tiles(int t_ipt2, int t_s1, int t_s2) {
    CTX_OR_FAIL(c);
    if (t_s2 < 0 || t_s2 > 32 || t_s1 < t_s2 || t_s1 > 64 || t_ipt2 < t_s1 || (t_ipt2 > 128 && t_ipt2 != 256))
        return ST_BAD_INDEX;
    c->tiles[0] = g_soft_shape[0] = t_ipt2;
    c->tiles[1] = g_soft_shape[1] = t_s1;
    c->tiles[2] = g_soft_shape[2] = t_s2;
    return 0;
}

int p3t_set_soft_occupancy(int ctas_per_sm) {
    CTX_OR_FAIL(c);
    if (ctas_per_sm < 4 || ctas_per_sm > 6) return ST_BAD_INDEX;
    c->soft_occ = g_soft_shape[3] = ctas_per_sm;
    return 0;
}

int p3t_set_options(int precision, int trace_mode, int cand_cap) {
    CTX_OR_FAIL(c);
    if (precision < 0 || precision > 1 || trace_mode < 0 || trace_mode > 1 || cand_cap < 1) return ST_BAD_INDEX;
    c->precision = precision;
    c->trace_mode = trace_mode;
    c->cand_cap = cand_cap;
    return 0;
}

void *p3t_stream(void) {
    Context *c = ctx_get(0);
    return c ? (void *)c->stream : nullptr;
}

int p3t_synchronize(void) {
    CTX_OR_FAIL(c);
    return cuda_status(cudaStreamSynchronize(c->stream));
}

int p3t_status(void) {
    CTX_OR_FAIL(c);
    int h = read_status(c);  // (drains the stream: the walks' words are complete)
    if (h < 0) return h;
    for (auto &w : c->walk) h |= take_word(w);
    h |= take_word(c->fun) | c->dropped;
    c->dropped = 0;
    return h;
}

// ---- device-resident soft force ---------------------------------------------
int p3t_upload_particles(int n, const void *epj) {
    if (n < 0 || (n > 0 && !epj)) return ST_BAD_INDEX;
    CTX_OR_FAIL(c);
    DevSet &d = c->res;
    int r = 0;
    if ((r = d.epj_stage.reserve(n)) || (r = d.ptcl.reserve(n)) || (r = d.mass.reserve(n)) ||
        (r = d.r_out.reserve(n)) || (r = d.r_search.reserve(n)) || (r = d.force.reserve(n)) ||
        (r = d.acc64.reserve(n)))
        return r;
    Uploader u(c);
    const void *src = place(c, u, d.epj_stage.p, epj, (size_t)n * sizeof(EPJRec));
    r = u.issue();
    if (!r && n > 0) r = cuda_status(launch_pack_walks(pack_resident(d, n, src), n, c->stream));
    const int e = cuda_status(cudaStreamSynchronize(c->stream));  // the caller's records are read
    if (r || e) return r ? r : e;
    c->res_n = n;
    return 0;
}

int p3t_upload_lists(int n_group, const int *i_off, const int *i_idx, const int *j_off, const int *j_idx,
                     const int *s_off, const int *s_idx, const void *spj, int n_spj) {
    if (const int e = check_lists(n_group, i_off, i_idx, j_off, j_idx, s_off, s_idx, spj, n_spj)) return e;
    CTX_OR_FAIL(c);
    DevSet &d = c->res;
    const long long ni = n_group ? i_off[n_group] : 0, nj = n_group ? j_off[n_group] : 0,
                    ns = n_group ? s_off[n_group] : 0;
    int r = 0;
    if ((r = d.i_off.reserve(n_group + 1)) || (r = d.j_off.reserve(n_group + 1)) || (r = d.s_off.reserve(n_group + 1)) ||
        (r = d.i_idx.reserve(ni)) || (r = d.j_idx.reserve(nj)) || (r = d.s_idx.reserve(ns)) ||
        (r = d.spj.reserve(n_spj)) || (r = d.order.reserve(n_group)))
        return r;
    Uploader u(c);
    u.add(d.i_off.p, i_off, i_off ? (n_group + 1) * sizeof(int) : 0);
    u.add(d.j_off.p, j_off, j_off ? (n_group + 1) * sizeof(int) : 0);
    u.add(d.s_off.p, s_off, s_off ? (n_group + 1) * sizeof(int) : 0);
    u.add(d.i_idx.p, i_idx, ni * sizeof(int));
    u.add(d.j_idx.p, j_idx, nj * sizeof(int));
    u.add(d.s_idx.p, s_idx, ns * sizeof(int));
    u.add(d.spj.p, spj, (size_t)n_spj * sizeof(SPJRec));
    d.order_valid = false;
    r = u.issue();
    if (!r) r = cuda_status(launch_group_order(n_group, d.i_off.p, d.j_off.p, d.s_off.p, nullptr, d.order.p, nullptr, c->stream));
    const int e = cuda_status(cudaStreamSynchronize(c->stream));  // the caller's lists are read
    if (r || e) return r ? r : e;
    c->res_groups = n_group;
    c->res_spj = n_spj;
    d.order_valid = true;
    return 0;
}

int p3t_soft_run(int emit_candidates) {
    CTX_OR_FAIL(c);
    DevSet &d = c->res;
    int r = 0;
    if (emit_candidates && (r = d.cand.reserve((size_t)c->res_n * c->cand_cap))) return r;
    SoftArgs A = make_args(c, d, c->res_groups, c->res_n, c->res_spj, false);
    if (!emit_candidates) A.cand = nullptr;
    return cuda_status(launch_soft(A, c->precision, emit_candidates != 0, c->stream));
}

int p3t_download_forces(void *force, int n) {
    CTX_OR_FAIL(c);
    if (n > c->res_n || n < 0) return ST_BAD_INDEX;
    if (c->reads_host || is_pinned(force)) {
        // (the status read waits for both)
        if (n > 0)
            if (const int r = cuda_status(cudaMemcpyAsync(force, c->res.force.p, (size_t)n * sizeof(ForceRec),
                                                          cudaMemcpyDeviceToHost, c->stream)))
                return r;
    } else {
        int r = grow_host(&c->h_out, &c->h_out_cap, (size_t)n * sizeof(ForceRec));
        if (r || (r = d2h(c, c->h_out, c->res.force.p, (size_t)n * sizeof(ForceRec)))) return r;
        std::memcpy(force, c->h_out, (size_t)n * sizeof(ForceRec));
    }
    return read_status(c);
}

// The pair kernel over groups as their bodies arrive.  The lists and the
// superparticles are on the stream already; the bodies follow in up to GO_STAGES parts
// on the side stream, and a group runs with the part that holds the last body it
// needs, every second part on a stream of its own, so that a part's last CTAs
// share the chip with the next part's first.  Bodies in tree order (as FDPS
// passes them) make a group's bodies near each other; any other order is right
// too, and ends with most groups in the last part.  The host waits once for the
// parts' sizes, while the bodies travel.
// A part costs its launches and the tail of its last groups (a group of 256 bodies
// takes some 75 us alone), so it has PART_GROUPS groups or more: groups of up to
// 256, 1M bodies (8,590 groups) 1.86 -> 1.61 ms in eight parts (four: 1.76), 800,000
// 1.43 -> 1.29, 600,000 (5,050 groups) 1.09 -> 1.00, 400,000 (3,568) 0.74 -> 0.75: not
// below STAGED_GROUPS or STAGED_BODIES.
constexpr int STAGED_BODIES = 524288, STAGED_GROUPS = 4500, PART_GROUPS = 1000;
static int run_staged(Context *c, DevSet &d, const PackArgs &K, SoftArgs A) {
    const int n = K.one.nj, ng = A.n_group, parts = std::max(2, std::min(GO_STAGES, ng / PART_GROUPS));
    const int per = (n + parts - 1) / parts;
    int r = 0;
    for (auto &e : c->stage_ev)
        if (!e && (r = cuda_status(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)))) return r;
    cudaEvent_t *const ev = c->stage_ev, lists = ev[GO_STAGES], sizes = ev[GO_STAGES + 1];
    if ((r = d.stage.reserve((size_t)ng + GO_STAGES)) || (r = grow_host(&c->h_out, &c->h_out_cap, GO_STAGES * sizeof(int))))
        return r;
    int *const start = d.stage.p + ng, *const h = (int *)c->h_out;
    PackArgs S = K;  // the superparticles
    S.one.nj = 0;
    if ((r = cuda_status(launch_pack_walks(S, S.one.ns, c->stream))) || (r = cuda_status(cudaEventRecord(lists, c->stream))) ||
        (r = cuda_status(cudaStreamWaitEvent(c->side, lists, 0))))
        return r;
    for (int s = 0; s < parts; s++) {
        PackArgs B = K;
        const int first = std::min(n, s * per);
        B.one.ns = 0;
        B.one.epj = (const EPJRec *)K.one.epj + first;
        B.one.nj = std::min(per, n - first);
        B.one.jo = first;
        if ((r = cuda_status(launch_pack_walks(B, B.one.nj, c->side))) || (r = cuda_status(cudaEventRecord(ev[s], c->side))))
            return r;
    }
    if ((r = cuda_status(launch_group_stage(ng, d.i_off.p, d.i_idx.p, d.j_off.p, d.j_idx.p, n, per, d.stage.p, c->stream))) ||
        (r = cuda_status(launch_group_order(ng, d.i_off.p, d.j_off.p, d.s_off.p, d.stage.p, d.order.p, start, c->stream))) ||
        (r = cuda_status(cudaMemcpyAsync(h, start, GO_STAGES * sizeof(int), cudaMemcpyDeviceToHost, c->stream))) ||
        (r = cuda_status(cudaEventRecord(sizes, c->stream))) || (r = cuda_status(cudaStreamWaitEvent(c->pair, sizes, 0))) ||
        (r = cuda_status(cudaEventSynchronize(sizes))))
        return r;
    A.n_group_all = ng;
    for (int s = 0; s < parts; s++) {
        const int first = h[s], last = s + 1 < parts ? h[s + 1] : ng;
        const cudaStream_t st = s & 1 ? c->pair : c->stream;
        A.group_order = d.order.p + first;
        A.n_group = last - first;
        if ((r = cuda_status(cudaStreamWaitEvent(st, ev[s], 0))) || (r = cuda_status(launch_soft(A, c->precision, false, st))))
            return r;
    }
    if ((r = cuda_status(cudaEventRecord(sizes, c->pair)))) return r;
    return cuda_status(cudaStreamWaitEvent(c->stream, sizes, 0));
}

// One call, host buffers in and out, with a single wait.  The link bounds what
// the pair kernel does not: the lists go by the copy engine, one launch packs
// bodies and superparticles from the caller's memory, the launch order is made on
// the device, and the pair kernel writes each force into the caller's pinned
// buffer as well as to the device.  1M bodies: 2.19 -> 1.92 ms with the pair kernel
// (0.93) behind the link (0.88 at its 205 GB/s, 180 MB in), 1.63 ms with the groups run
// as their bodies arrive (run_staged).
int p3t_soft_force_host(int n, const void *epj, int n_group, const int *i_off, const int *i_idx, const int *j_off,
                        const int *j_idx, const int *s_off, const int *s_idx, const void *spj, int n_spj,
                        void *force) {
    if (n < 0 || (n > 0 && (!epj || !force))) return ST_BAD_INDEX;
    if (const int e = check_lists(n_group, i_off, i_idx, j_off, j_idx, s_off, s_idx, spj, n_spj)) return e;
    CTX_OR_FAIL(c);
    DevSet &d = c->res;
    const long long ni = n_group ? i_off[n_group] : 0, nj = n_group ? j_off[n_group] : 0,
                    ns = n_group ? s_off[n_group] : 0;
    int r = 0;
    if ((r = d.epj_stage.reserve(n)) || (r = d.ptcl.reserve(n)) || (r = d.mass.reserve(n)) ||
        (r = d.r_out.reserve(n)) || (r = d.r_search.reserve(n)) || (r = d.force.reserve(n)) ||
        (r = d.acc64.reserve(n)) || (r = d.i_off.reserve(n_group + 1)) || (r = d.j_off.reserve(n_group + 1)) ||
        (r = d.s_off.reserve(n_group + 1)) || (r = d.i_idx.reserve(ni)) || (r = d.j_idx.reserve(nj)) ||
        (r = d.s_idx.reserve(ns)) || (r = d.spj.reserve(n_spj)) || (r = d.order.reserve((size_t)n_group)) ||
        (r = d.jsplit.reserve(n)) || (r = d.spjp.reserve(n_spj)))
        return r;
    const bool f64 = c->precision == 1;
    Uploader u(c);
    u.add(d.i_off.p, i_off, i_off ? (n_group + 1) * sizeof(int) : 0);
    u.add(d.j_off.p, j_off, j_off ? (n_group + 1) * sizeof(int) : 0);
    u.add(d.s_off.p, s_off, s_off ? (n_group + 1) * sizeof(int) : 0);
    u.add(d.i_idx.p, i_idx, ni * sizeof(int));
    u.add(d.j_idx.p, j_idx, nj * sizeof(int));
    u.add(d.s_idx.p, s_idx, ns * sizeof(int));
    PackArgs K = pack_resident(d, n, place(c, u, d.epj_stage.p, epj, (size_t)n * sizeof(EPJRec)));
    K.one.spj = place(c, u, d.spj.p, spj, (size_t)n_spj * sizeof(SPJRec));
    K.one.ns = n_spj;
    if (K.one.spj != d.spj.p) K.spj = d.spj.p;  // kept for later runs on the resident lists
    if (!f64) {
        K.jsplit = d.jsplit.p;
        K.spjp = d.spjp.p;
        K.eps2 = (float)c->params[0];
        K.trace_mode = c->trace_mode;
    }
    // an early return leaves no copy of this call running (the caller's
    // buffers and the staging buffer are reused afterwards)
    auto fail = [&](int e) {
        for (cudaStream_t s : {c->side, c->pair, c->stream}) cudaStreamSynchronize(s);
        return e;
    };
    const bool staged = n >= STAGED_BODIES && n_group >= STAGED_GROUPS && K.one.epj == epj;
    if ((r = u.issue())) return fail(r);
    if (!staged &&
        ((r = cuda_status(launch_group_order(n_group, d.i_off.p, d.j_off.p, d.s_off.p, nullptr, d.order.p, nullptr, c->stream))) ||
         (r = cuda_status(launch_pack_walks(K, (long long)n + n_spj, c->stream)))))
        return fail(r);
    c->res_n = n;
    c->res_groups = n_group;
    c->res_spj = n_spj;
    d.order_valid = true;
    SoftArgs A = make_args(c, d, n_group, n, n_spj, false);
    A.cand = nullptr;
    A.packed = 1;
    A.isplit = A.jsplit = d.jsplit.p;
    A.spjp = d.spjp.p;
    // every body is in a group: the forces need no download of their own
    const bool copy = ni == n && is_pinned(force) && device_reads(c, force, 4);
    if (copy) A.force_copy = (ForceRec *)force;
    if (staged) r = run_staged(c, d, K, A);
    else r = cuda_status(launch_soft(A, c->precision, false, c->stream));
    if (r) return fail(r);
    return copy ? read_status(c) : p3t_download_forces(force, n);
}

}  // extern "C"
