// FDPS-facing entry points of the soft force: the single-group functor
// calls and the multiwalk dispatch/retrieve pair (pointer and index forms).
// The walks' arrays are read where FDPS has them, packed into the same device
// layout the resident path uses, and go through the same kernels.
#include <cstdint>
#include <cstring>
#include <unistd.h>

#include "../../include/gplum_p3t.h"
#include "p3t_capi_internal.cuh"
#include "p3t_common.cuh"
#include "p3t_soft.cuh"

using namespace p3t;

namespace {

WalkSlot *slot_for(Context *c, int tag) {
    if (tag < 0) return nullptr;
    WalkSlot &w = c->walk[tag % MAX_TAGS];
    if (!w.done && cudaEventCreateWithFlags(&w.done, cudaEventDisableTiming) != cudaSuccess) return nullptr;
    if (!w.read && cudaEventCreateWithFlags(&w.read, cudaEventDisableTiming) != cudaSuccess) return nullptr;
    return &w;
}

// Per-walk counts of a dispatch: non-negative, with a record pointer where a
// count is positive, and totals that fit the int offsets.
int check_walks(int n_walk, const int *cnt, const void *const *ptr) {
    if (n_walk < 0 || (n_walk > 0 && !cnt)) return ST_BAD_INDEX;
    long long tot = 0;
    for (int k = 0; k < n_walk; k++) {
        if (cnt[k] < 0 || (cnt[k] > 0 && (!ptr || !ptr[k]))) return ST_BAD_INDEX;
        tot += cnt[k];
    }
    return tot > 2147483647LL ? ST_BAD_INDEX : 0;
}

// Room for a table behind the slot's status word, whose bits stay until they are read.
int reserve_table(WalkSlot &w, size_t bytes) {
    const size_t had = w.h_tab_cap;
    const int word = had ? *(volatile int *)w.h_tab : 0;
    const int r = grow_host(&w.h_tab, &w.h_tab_cap, 64 + bytes);
    if (!r && w.h_tab_cap != had) *(volatile int *)w.h_tab = word;
    return r;
}

// A call's walks in the slot's pinned table, which the kernels read.
struct WalkTable {
    WalkSlot &w;
    int n_walk;
    size_t size_j, size_s;  // bytes of an EPJ and SPJ entry (records or indices)
    int ni = 0, nj = 0, ns = 0;
    bool staged = false;  // the records lie in the slot's pinned buffer, not where the caller has them

    int *status() const { return (int *)w.h_tab; }
    WalkRecords *rec() const { return (WalkRecords *)((char *)w.h_tab + 64); }

    int reserve() { return reserve_table(w, (size_t)n_walk * sizeof(WalkRecords)); }
    void set(int k, const void *epi, int n_i, const void *epj, int n_j, const void *spj, int n_s) {
        rec()[k] = WalkRecords{(const EPIRec *)epi, epj, spj, n_i, n_j, n_s, ni, nj, ns};
        ni += n_i; nj += n_j; ns += n_s;
    }
    // Where the records are read.  The kernel reads them in the caller's memory
    // where the device can (60,000 bodies in the index form, four dispatches: the
    // host's copies into pinned buffers, 14-24 GB/s, were 1.2 of a pass's 1.5 ms;
    // the link gives 150-200 GB/s; a pass now takes 0.28 ms) and they are aligned as the kernel reads them;
    // otherwise they are first copied into the slot's pinned buffer.
    int place(bool reads_host) {
        uintptr_t bits = 0;
        for (int k = 0; k < n_walk; k++) {
            const WalkRecords &r = rec()[k];
            if (r.ni) bits |= (uintptr_t)r.epi;
            if (r.nj) bits |= (uintptr_t)r.epj << (size_j < 8);
            if (r.ns) bits |= (uintptr_t)r.spj << (size_s < 8);
        }
        if (reads_host && (bits & 7) == 0) return 0;
        staged = true;
        const size_t need = (size_t)ni * sizeof(EPIRec) + (size_t)nj * size_j + (size_t)ns * size_s + 16;
        const int r = grow_host(&w.h_in, &w.h_in_cap, need);
        if (r) return r;
        char *h = (char *)w.h_in;
        auto put = [&](const void *src, size_t bytes) {
            char *to = h;
            if (bytes) std::memcpy(h, src, bytes);
            h += bytes;
            return to;
        };
        // records of one kind after another: the 8-byte ones first
        for (int k = 0; k < n_walk; k++) rec()[k].epi = (const EPIRec *)put(rec()[k].epi, (size_t)rec()[k].ni * sizeof(EPIRec));
        for (int k = 0; k < n_walk; k++) rec()[k].epj = put(rec()[k].epj, (size_t)rec()[k].nj * size_j);
        for (int k = 0; k < n_walk; k++) rec()[k].spj = put(rec()[k].spj, (size_t)rec()[k].ns * size_s);
        return 0;
    }
};

// Device arrays of a call's i-bodies and lists, and the pack arguments that fill them.
int pack_args(Context *c, WalkTable &t, bool index, PackArgs &A) {
    DevSet &d = t.w.d;
    const bool f64 = c->precision == 1;
    int r = 0;
    if ((r = d.i_off.reserve(t.n_walk + 1)) || (r = d.j_off.reserve(t.n_walk + 1)) ||
        (r = d.s_off.reserve(t.n_walk + 1)) || (r = d.i_idx.reserve(t.ni)) || (r = d.j_idx.reserve(t.nj)) ||
        (r = d.s_idx.reserve(t.ns)) || (r = d.iptcl.reserve(t.ni)))
        return r;
    A = PackArgs{};
    A.walk = t.rec();
    A.n_walk = t.n_walk;
    A.index = index;
    A.i_off = d.i_off.p; A.j_off = d.j_off.p; A.s_off = d.s_off.p;
    A.i_idx = d.i_idx.p; A.j_idx = d.j_idx.p; A.s_idx = d.s_idx.p;
    A.iptcl = d.iptcl.p;
    A.eps2 = (float)c->params[0];
    A.trace_mode = c->trace_mode;
    if (f64) {
        if ((r = d.i_r_out.reserve(t.ni)) || (r = d.i_r_search.reserve(t.ni))) return r;
        A.i_r_out = d.i_r_out.p; A.i_r_search = d.i_r_search.p;
    } else {
        if ((r = d.isplit.reserve(t.ni))) return r;
        A.isplit = d.isplit.p;
    }
    if (index) return 0;
    if ((r = d.ptcl.reserve(t.nj))) return r;
    A.ptcl = d.ptcl.p;
    if (f64) {
        if ((r = d.mass.reserve(t.nj)) || (r = d.r_out.reserve(t.nj)) || (r = d.r_search.reserve(t.nj)) ||
            (r = d.spj.reserve(t.ns)))
            return r;
        A.mass = d.mass.p; A.r_out = d.r_out.p; A.r_search = d.r_search.p;
        A.spj = d.spj.p;
    } else {
        if ((r = d.jsplit.reserve(t.nj)) || (r = d.spjp.reserve(t.ns))) return r;
        A.jsplit = d.jsplit.p;
        A.spjp = d.spjp.p;
    }
    return 0;
}

// Forces of at least this many bytes stay on the device until the retrieve, whose
// kernel writes them into the caller's arrays; smaller ones go to the slot's
// pinned buffer and are copied by the host (14-24 GB/s, from a few us; the kernel
// takes a launch and a wait, 10 us).  60,000 bodies in four dispatches: 360 -> 277 us
// with the records read on the side stream.
constexpr size_t SCATTER_BYTES = 192 << 10;
bool on_device(Context *c, int n_i) { return c->reads_host && (size_t)n_i * sizeof(ForceRec) >= SCATTER_BYTES; }

// The soft kernel over packed walks: the j side from x (the slot's own arrays, or
// the resident ones of the index form), the forces into the slot's pinned buffer.
SoftArgs walk_args(Context *c, WalkTable &t, DevSet &x, int n_j, int n_s, bool accumulate) {
    DevSet &d = t.w.d;
    d.order_valid = false;
    SoftArgs A = make_args(c, d, t.n_walk, n_j, n_s, accumulate);
    A.ptcl = x.ptcl.p; A.mass = x.mass.p; A.r_out = x.r_out.p; A.r_search = x.r_search.p;
    A.spj = x.spj.p;
    A.iptcl = d.iptcl.p; A.i_r_out = d.i_r_out.p; A.i_r_search = d.i_r_search.p; A.n_iptcl = t.ni;
    A.isplit = d.isplit.p; A.jsplit = x.jsplit.p; A.spjp = x.spjp.p;
    A.packed = 1;
    // the kernels' status bits: the slot's own pinned word (a copy behind the kernels was 4 us)
    A.status = t.status();
    A.force = !accumulate && on_device(c, t.ni) ? d.force.p : (ForceRec *)t.w.h_out;
    A.cand = nullptr;
    return A;
}

// the forces of one walk and where the caller wants them
struct ForceOut {
    int *dst;
    int off, n;
};
__global__ void __launch_bounds__(256) k_scatter_forces(const ForceOut *__restrict__ out, const ForceRec *__restrict__ f) {
    constexpr int W = sizeof(ForceRec) / sizeof(int);
    const ForceOut o = out[blockIdx.x];
    const int *const src = (const int *)(f + o.off);
    const long long n = (long long)o.n * W;
    for (long long t = blockIdx.y * 256 + threadIdx.x; t < n; t += gridDim.y * 256) o.dst[t] = src[t];
}

// Functor call: one group, accumulate into the caller's ForceGrav records.  Two
// launches and one wait; the pack kernel reads the records where they are.
int functor_call(const void *epi, int ni, const void *epj, int nj, const void *spj, int ns, void *force) {
    Context *c = ctx_get(0);
    if (!c) return -(int)cudaErrorNoDevice;
    if (ni <= 0) return 0;
    if (!epi || !force || nj < 0 || ns < 0 || (nj > 0 && !epj) || (ns > 0 && !spj)) return ST_BAD_INDEX;
    WalkSlot &w = c->fun;
    WalkTable t{w, 1, sizeof(EPJRec), sizeof(SPJRec)};
    const size_t bytes = (size_t)ni * sizeof(ForceRec);
    int r = 0;
    if ((r = t.reserve()) || (r = grow_host(&w.h_out, &w.h_out_cap, bytes)) || (r = w.d.acc64.reserve(ni))) return r;
    t.set(0, epi, ni, epj, nj, spj, ns);
    PackArgs K;
    if ((r = t.place(c->reads_host)) || (r = pack_args(c, t, false, K))) return r;
    std::memcpy(w.h_out, force, bytes);
    if (c->precision == 1) {
        // FP64 form accumulates in double: seed it from the caller's records
        K.seed = (const ForceRec *)w.h_out;
        K.acc64 = w.d.acc64.p;
    }
    if (!(r = cuda_status(launch_pack_walks(K, (long long)ni + nj + ns, c->stream))))
        r = cuda_status(launch_soft(walk_args(c, t, w.d, nj, ns, true), c->precision, false, c->stream));
    // also after an error: nothing of this call may still read the caller's records
    const int e = cuda_status(cudaStreamSynchronize(c->stream));
    if (r || e) {
        take_word(w);
        return r ? r : e;
    }
    std::memcpy(force, w.h_out, bytes);
    return take_word(w);
}

// Common tail of both dispatch forms: kernels, events.  Returns once
// the caller's records have been read (in_place: by the kernels, where they are).
int launch_walks(Context *c, WalkTable &t, const PackArgs &K, DevSet &x, int n_j, int n_s, long long n_records,
                 bool in_place) {
    WalkSlot &w = t.w;
    int r = 0;
    auto run = [&]() {
        int e = 0;
        // on the side stream: the records are read while an earlier dispatch computes
        if ((e = cuda_status(launch_pack_walks(K, n_records, c->side)))) return e;
        if ((e = cuda_status(cudaEventRecord(w.read, c->side)))) return e;
        if ((e = cuda_status(cudaStreamWaitEvent(c->stream, w.read, 0)))) return e;
        if ((e = cuda_status(launch_soft(walk_args(c, t, x, n_j, n_s, false), c->precision, false, c->stream)))) return e;
        return cuda_status(cudaEventRecord(w.done, c->stream));
    };
    if ((r = run())) {
        cudaStreamSynchronize(c->side);
        cudaStreamSynchronize(c->stream);
        return r;
    }
    w.n_i = t.ni;
    w.busy = true;
    return in_place ? cuda_status(cudaEventSynchronize(w.read)) : 0;
}

// Writes a byte of every page of the walks' result arrays, as it is: a kernel's first
// touch of fresh pages is slow, the host's is not (retrieve into an array that nobody has
// written yet: 6,200 records 111 -> 51 us, 60,000 236 -> 111; into a used one 20 and 42).
// The walks of one allocation lie end to end as a rule, which costs no look at each.
void touch_range(uintptr_t a, uintptr_t e) {
    static const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    for (uintptr_t p = a; p < e; p = (p & ~(page - 1)) + page) {
        volatile char *const c = (volatile char *)p;
        *c = *c;
    }
}
void touch_pages(int n_walk, const int *n_epi, void **force, bool end_to_end, long long n) {
    if (end_to_end) {
        if (n > 0) touch_range((uintptr_t)force[0], (uintptr_t)force[0] + (size_t)n * sizeof(ForceRec));
        return;
    }
    for (int k = 0; k < n_walk; k++)
        if (n_epi[k] > 0) touch_range((uintptr_t)force[k], (uintptr_t)force[k] + (size_t)n_epi[k] * sizeof(ForceRec));
}

// The forces' place: the slot's pinned buffer or device array.
int reserve_force(Context *c, WalkSlot &w, int n_i) {
    return on_device(c, n_i) ? w.d.force.reserve(n_i) : grow_host(&w.h_out, &w.h_out_cap, (size_t)n_i * sizeof(ForceRec));
}

// A dispatch's slot, free of earlier work (a skipped retrieve: the slot is reused in
// order, and the status bits of the dispatch that it drops are left to p3t_status).
int claim_slot(Context *c, WalkSlot &w) {
    int r = 0;
    if (w.busy) {
        w.busy = false;
        r = cuda_status(cudaEventSynchronize(w.done));
    }
    c->dropped |= take_word(w);
    return r;
}

}  // namespace

extern "C" {

int p3t_epep(const void *epi, int ni, const void *epj, int nj, void *force) {
    return functor_call(epi, ni, epj, nj, nullptr, 0, force);
}

int p3t_epsp(const void *epi, int ni, const void *spj, int nj, void *force) {
    return functor_call(epi, ni, nullptr, 0, spj, nj, force);
}

int p3t_soft_dispatch(int tag, int n_walk, const void **epi, const int *n_epi, const void **epj, const int *n_epj,
                      const void **spj, const int *n_spj) {
    int e = 0;
    if ((e = check_walks(n_walk, n_epi, epi)) || (e = check_walks(n_walk, n_epj, epj)) ||
        (e = check_walks(n_walk, n_spj, spj)))
        return e;
    Context *c = ctx_get(0);
    if (!c) return -(int)cudaErrorNoDevice;
    WalkSlot *ws = slot_for(c, tag);
    if (!ws) return ST_BAD_INDEX;
    WalkSlot &w = *ws;
    WalkTable t{w, n_walk, sizeof(EPJRec), sizeof(SPJRec)};
    int r = 0;
    if ((r = claim_slot(c, w)) || (r = t.reserve())) return r;
    for (int k = 0; k < n_walk; k++)
        t.set(k, n_epi[k] ? epi[k] : nullptr, n_epi[k], n_epj[k] ? epj[k] : nullptr, n_epj[k], n_spj[k] ? spj[k] : nullptr,
              n_spj[k]);
    PackArgs K;
    if ((r = t.place(c->reads_host)) || (r = pack_args(c, t, false, K)) || (r = w.d.acc64.reserve(t.ni)) ||
        (r = reserve_force(c, w, t.ni)))
        return r;
    return launch_walks(c, t, K, w.d, t.nj, t.ns, (long long)t.ni + t.nj + t.ns, !t.staged);
}

int p3t_soft_dispatch_index(int tag, int n_walk, const void **epi, const int *n_epi, const int **id_epj,
                            const int *n_epj, const int **id_spj, const int *n_spj, const void *epj, int n_epj_tot,
                            const void *spj, int n_spj_tot, int send_flag) {
    int e = 0;
    if ((e = check_walks(n_walk, n_epi, epi)) || (e = check_walks(n_walk, n_epj, (const void *const *)id_epj)) ||
        (e = check_walks(n_walk, n_spj, (const void *const *)id_spj)))
        return e;
    if (send_flag && (n_epj_tot < 0 || n_spj_tot < 0 || (n_epj_tot > 0 && !epj) || (n_spj_tot > 0 && !spj)))
        return ST_BAD_INDEX;
    Context *c = ctx_get(0);
    if (!c) return -(int)cudaErrorNoDevice;
    WalkSlot *ws = slot_for(c, tag);
    if (!ws) return ST_BAD_INDEX;
    WalkSlot &w = *ws;
    WalkTable t{w, n_walk, sizeof(int), sizeof(int)};
    int r = 0;
    if ((r = claim_slot(c, w))) return r;
    DevSet &x = c->idx;
    bool sent = false;  // the resident records are being read in place, on the library's stream
    if (send_flag) {
        // resident for the dispatches that follow, which may switch the
        // precision: the arrays of both forms
        if ((r = x.ptcl.reserve(n_epj_tot)) || (r = x.mass.reserve(n_epj_tot)) || (r = x.r_out.reserve(n_epj_tot)) ||
            (r = x.r_search.reserve(n_epj_tot)) || (r = x.jsplit.reserve(n_epj_tot)) ||
            (r = x.spj.reserve(n_spj_tot)) || (r = x.spjp.reserve(n_spj_tot)))
            return r;
        WalkTable s{w, 1, sizeof(EPJRec), sizeof(SPJRec)};
        if ((r = s.reserve())) return r;
        s.set(0, nullptr, 0, n_epj_tot ? epj : nullptr, n_epj_tot, n_spj_tot ? spj : nullptr, n_spj_tot);
        if ((r = s.place(c->reads_host))) return r;
        PackArgs K{};
        K.one = s.rec()[0];
        K.n_walk = 1;
        K.ptcl = x.ptcl.p; K.mass = x.mass.p; K.r_out = x.r_out.p; K.r_search = x.r_search.p;
        K.jsplit = x.jsplit.p;
        K.spj = x.spj.p; K.spjp = x.spjp.p;
        K.eps2 = (float)c->params[0];
        K.trace_mode = c->trace_mode;
        if ((r = cuda_status(launch_pack_walks(K, (long long)n_epj_tot + n_spj_tot, c->stream)))) return r;
        // the walks' records may take the same pinned buffer, and an early
        // return leaves nothing reading the caller's arrays
        if (s.staged && (r = cuda_status(cudaStreamSynchronize(c->stream)))) return r;
        sent = !s.staged;
        c->idx_nj = n_epj_tot;
        c->idx_ns = n_spj_tot;
        c->idx_eps2 = K.eps2;
        c->idx_trace = K.trace_mode;
    } else if (c->idx_ns > 0 && (c->idx_eps2 != (float)c->params[0] || c->idx_trace != c->trace_mode)) {
        c->idx_eps2 = (float)c->params[0];
        c->idx_trace = c->trace_mode;
        if ((r = cuda_status(launch_spj_pack(x.spj.p, c->idx_ns, c->idx_eps2, c->idx_trace, x.spjp.p, c->stream)))) return r;
    }
    PackArgs K;
    auto walks = [&]() {
        int f = 0;
        if ((f = t.reserve())) return f;
        for (int k = 0; k < n_walk; k++)
            t.set(k, n_epi[k] ? epi[k] : nullptr, n_epi[k], n_epj[k] ? id_epj[k] : nullptr, n_epj[k],
                  n_spj[k] ? id_spj[k] : nullptr, n_spj[k]);
        if ((f = t.place(c->reads_host)) || (f = pack_args(c, t, true, K)) || (f = w.d.acc64.reserve(t.ni))) return f;
        return reserve_force(c, w, t.ni);
    };
    if ((r = walks())) {
        cudaStreamSynchronize(c->stream);
        return r;
    }
    // the walks' records are read behind the resident ones, so that one event tells of both
    if (sent && ((r = cuda_status(cudaEventRecord(w.done, c->stream))) ||
                 (r = cuda_status(cudaStreamWaitEvent(c->side, w.done, 0))))) {
        cudaStreamSynchronize(c->stream);
        return r;
    }
    return launch_walks(c, t, K, x, c->idx_nj, c->idx_ns, t.ni + ((long long)t.nj + t.ns) / 8, sent || !t.staged);
}

int p3t_soft_retrieve(int tag, int n_walk, const int *n_epi, void **force) {
    Context *c = ctx_get(0);
    if (!c) return -(int)cudaErrorNoDevice;
    WalkSlot *ws = slot_for(c, tag);
    if (!ws || !ws->busy) return ST_BAD_INDEX;
    WalkSlot &w = *ws;
    uintptr_t bits = 0, apart = 0;  // apart: 0 while the walks' arrays lie end to end
    int walks = n_walk;             // those that the dispatch covers
    long long off = 0;
    for (int k = 0; k < walks; k++) {
        if (off + n_epi[k] > w.n_i) walks = k;
        else {
            apart |= (uintptr_t)force[k] - (uintptr_t)force[0] - (uintptr_t)off * sizeof(ForceRec);
            off += n_epi[k];
            if (n_epi[k] > 0) bits |= (uintptr_t)force[k];
        }
    }
    const bool device = on_device(c, w.n_i), direct = device && (bits & 3) == 0;
    if (direct) touch_pages(walks, n_epi, force, apart == 0, off);  // while the kernels run
    int r = cuda_status(cudaEventSynchronize(w.done));
    w.busy = false;
    if (r) return r;
    const int status = take_word(w);  // this dispatch's own bits
    if (direct) {
        if ((r = reserve_table(w, (size_t)walks * sizeof(ForceOut)))) return r;
        ForceOut *out = (ForceOut *)((char *)w.h_tab + 64);
        off = 0;
        for (int k = 0; k < walks; k++) {
            out[k] = ForceOut{(int *)force[k], (int)off, n_epi[k]};
            off += n_epi[k];
        }
        // four words a thread of an average walk
        const int slices = walks > 0 ? (int)std::min<long long>(4096, off * 8 / (1024LL * walks) + 1) : 0;
        if (walks > 0) { P3T_COUNT_LAUNCH(); k_scatter_forces<<<dim3(walks, slices), 256, 0, c->side>>>(out, w.d.force.p); }
        if ((r = cuda_status(cudaGetLastError())) || (r = cuda_status(cudaStreamSynchronize(c->side)))) return r;
    } else {
        if (device) {
            const size_t bytes = (size_t)w.n_i * sizeof(ForceRec);
            if ((r = grow_host(&w.h_out, &w.h_out_cap, bytes)) ||
                (r = cuda_status(cudaMemcpyAsync(w.h_out, w.d.force.p, bytes, cudaMemcpyDeviceToHost, c->side))) ||
                (r = cuda_status(cudaStreamSynchronize(c->side))))
                return r;
        }
        const ForceRec *h = (const ForceRec *)w.h_out;
        for (int k = 0; k < walks; k++) {
            std::memcpy(force[k], h, (size_t)n_epi[k] * sizeof(ForceRec));
            h += n_epi[k];
        }
    }
    return walks < n_walk ? status | ST_BAD_INDEX : status;
}

}  // extern "C"
