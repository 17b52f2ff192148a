// Library context shared by the C-ABI translation units.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cuda_runtime.h>
#include <vector>

#include "p3t_common.cuh"
#include "p3t_soft.cuh"

namespace p3t {

int cuda_status(cudaError_t e);
int grow_raw(void **p, size_t *cap, size_t bytes);
int grow_host(void **p, size_t *cap, size_t bytes);

// Grow-only device array.
template <class T>
struct DevBuf {
    T *p = nullptr;
    size_t cap = 0;  // bytes
    int reserve(size_t n) { return grow_raw((void **)&p, &cap, std::max<size_t>(n, 1) * sizeof(T)); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
};

// One set of device buffers for a soft-force problem.
struct DevSet {
    DevBuf<EPJRec> epj_stage;
    DevBuf<SoftPtcl> iptcl;
    DevBuf<double> i_r_out, i_r_search;
    DevBuf<SoftPtcl> ptcl;
    DevBuf<double> mass, r_out, r_search;
    DevBuf<SPJRec> spj;
    DevBuf<SoftSplit> isplit, jsplit;
    DevBuf<SpjPack> spjp;
    DevBuf<int> i_off, i_idx, j_off, j_idx, s_off, s_idx, order, stage;
    DevBuf<ForceRec> force;
    DevBuf<D4> acc64;
    DevBuf<int> cand;
    bool order_valid = false;
    void release() {
        epj_stage.release(); iptcl.release(); i_r_out.release(); i_r_search.release(); ptcl.release(); mass.release(); r_out.release();
        r_search.release(); spj.release(); isplit.release(); jsplit.release(); spjp.release(); i_off.release(); i_idx.release(); j_off.release(); j_idx.release();
        s_off.release(); s_idx.release(); order.release(); stage.release(); force.release(); acc64.release(); cand.release();
    }
};

constexpr int MAX_TAGS = 8;

// State of one in-flight multiwalk dispatch (or of the functor calls).
struct WalkSlot {
    DevSet d;
    void *h_tab = nullptr;  // pinned: the kernels' status word, then the walks' records table
    size_t h_tab_cap = 0;
    void *h_in = nullptr;  // pinned: records that the device cannot read in place
    size_t h_in_cap = 0;
    void *h_out = nullptr;  // pinned: the forces, written by the kernel
    size_t h_out_cap = 0;
    cudaEvent_t read = nullptr, done = nullptr;  // the caller's records read; the forces there
    int n_i = 0;
    bool busy = false;
    void release() {
        d.release();
        if (h_tab) cudaFreeHost(h_tab);
        if (h_in) cudaFreeHost(h_in);
        if (h_out) cudaFreeHost(h_out);
        if (read) cudaEventDestroy(read);
        if (done) cudaEventDestroy(done);
        *this = WalkSlot();
    }
};

struct Context {
    int device = 0;
    bool reads_host = false;  // the device reads any host memory in place (it walks the host's page tables)
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;  // the soft calls' reads and writes of the caller's arrays
    cudaStream_t pair = nullptr;  // every second stage of the host call's pair kernel
    cudaEvent_t stage_ev[10] = {};  // the host call's stages (see p3t_soft_force_host)
    int *status = nullptr;  // device status bits
    double params[21];
    int params_version = 0;
    int precision = 0;
    int trace_mode = 0;
    int cand_cap = 64;
    int tiles[3] = {128, 64, 32};  // soft-kernel work split (SoftArgs::t_ipt2, t_s1, t_s2)
    int soft_occ = 5;              // mixed soft kernel: resident CTAs per SM (SoftArgs::occ)
    // resident problem
    DevSet res;
    int res_n = 0, res_groups = 0, res_spj = 0;
    // index-form multiwalk: EPJ/SPJ arrays resident across dispatches
    DevSet idx;
    int idx_nj = 0, idx_ns = 0;
    float idx_eps2 = 0.f;  // what idx.spjp was packed with
    int idx_trace = -1;
    // pinned staging
    void *h_stage = nullptr;
    size_t h_stage_cap = 0;
    void *h_out = nullptr;
    size_t h_out_cap = 0;
    WalkSlot walk[MAX_TAGS];
    WalkSlot fun;  // the single-group functor calls
    int dropped = 0;  // status bits of dispatches that were never retrieved

    void release() {
        res.release();
        idx.release();
        if (h_stage) cudaFreeHost(h_stage);
        if (h_out) cudaFreeHost(h_out);
        h_stage = h_out = nullptr;
        h_stage_cap = h_out_cap = 0;
        for (auto &e : stage_ev) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        for (auto &w : walk) w.release();
        fun.release();
    }
};

extern Context *g_ctx;
Context *ctx_get(int device);
int read_status(Context *c);
// The status bits that a slot's kernels have set, cleared (no kernel of the slot may run).
int take_word(WalkSlot &w);
// Host checks of caller lists before any copy or kernel: CSR offsets start at
// 0 and never decrease; index arrays and records are present where the
// offsets say there are entries.  ST_BAD_INDEX otherwise.  (GPLUM trusts
// FDPS's lists; a C caller here can hand any pointer.)
int check_csr(int n_group, const int *off);
int check_lists(int n_group, const int *i_off, const int *i_idx, const int *j_off, const int *j_idx,
                const int *s_off, const int *s_idx, const void *spj, int n_spj);
// Host->device uploads issued as one batch: sources that are pinned, or that
// the device reads through the host's page tables, are copied by the DMA engine
// directly (150-205 GB/s; a copy into pinned memory by a core, 14-24 GB/s),
// others are first gathered into the context's pinned staging buffer.
struct Uploader {
    Context *c;
    struct Item { void *dst; const void *src; size_t bytes; bool direct; };
    std::vector<Item> items;
    explicit Uploader(Context *cc) : c(cc) {}
    void add(void *dst, const void *src, size_t bytes);
    // queues the copies; returns once they are on the stream (the caller's
    // sources and the staging buffer must stay untouched until the stream has
    // run them)
    int issue();
    bool in_one_launch(int &r);
    // waits for the copies as well: the caller's and the staging buffers may be
    // reused afterwards
    int flush();
};
// One upload, with its wait.
int h2d(Context *c, void *dst, const void *src, size_t bytes);
// Device -> host copy ordered after the work queued on the library's
// stream (a non-blocking stream, which plain cudaMemcpy does not wait for).
int d2h(Context *c, void *dst, const void *src, size_t bytes);

SoftArgs make_args(Context *c, DevSet &d, int n_group, int n_ptcl, int n_spj, bool accumulate);
// Launch order of the soft kernel's groups: by stage (optional, 0 .. GO_STAGES - 1),
// then most pair work first; start (optional, [GO_STAGES]): the stages' first places.
constexpr int GO_STAGES = 8;
cudaError_t launch_group_order(int n_group, const int *i_off, const int *j_off, const int *s_off, const int *stage,
                               int *order, int *start, cudaStream_t st);
// stage[g]: the last body among group g's own and its EPJ list, / per.
cudaError_t launch_group_stage(int n_group, const int *i_off, const int *i_idx, const int *j_off, const int *j_idx, int n,
                               int per, int *stage, cudaStream_t st);
bool is_pinned(const void *p);
// Host memory that a kernel may read in place, at `align` bytes.
bool device_reads(Context *c, const void *p, size_t align);

}  // namespace p3t
