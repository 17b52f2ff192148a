// Exclusive prefix sums in one launch (decoupled look-back): each tile
// publishes its sum as soon as it has it and adds up its predecessors' until
// it meets one whose prefix is complete.  A status word holds epoch, flag and
// value together, so neither fences nor a reset between launches are needed:
// words of other launches have another epoch.  Tiles are numbered by a ticket
// in the order they start, so a tile only waits for tiles that already run;
// every wait has a limit, after which the launch reports ST_ITER_CAP.
//
// One launch and one pass over the data instead of three to five launches
// (block sums, their scan, the addition): 200,000 flags in 6.4 us (ncu).
#pragma once
#include "p3t_capi_internal.cuh"
#include "p3t_common.cuh"

namespace p3t {

constexpr int LB_T = 256, LB_K = 8, LB_TILE = LB_T * LB_K;  // threads, items a thread, items a tile
constexpr int LB_SPIN = 1 << 24;
enum : unsigned { LB_SUM = 1, LB_PREFIX = 2 };

// Status words (zeroed when they grow) and tickets of the launches on one stream.
struct LookBack {
    DevBuf<unsigned long long> st;
    DevBuf<unsigned> ticket;  // one per scan of a launch, back at zero after every launch
    unsigned epoch = 0;
    int reserve(Context *c, size_t words) {
        int r = 0;
        if (!ticket.p) {
            if ((r = ticket.reserve(2))) return r;
            cudaMemsetAsync(ticket.p, 0, ticket.cap, c->stream);
        }
        if (words * sizeof(unsigned long long) > st.cap) {
            if ((r = st.reserve(words))) return r;
            cudaMemsetAsync(st.p, 0, st.cap, c->stream);
        }
        epoch = (epoch + 1) & 0x3fffffffu;
        if (epoch == 0) {  // a full turn: no word of the last one may be taken for a new one
            cudaMemsetAsync(st.p, 0, st.cap, c->stream);
            epoch = 1;
        }
        return 0;
    }
};

__device__ __forceinline__ void lb_put(unsigned long long *p, unsigned epoch, unsigned flag, unsigned v) {
    *(volatile unsigned long long *)p = ((unsigned long long)(epoch << 2 | flag) << 32) | v;
}
// the value of a word of this epoch (flag in `flag`), waiting for it; 0 and
// LB_PREFIX when the limit is reached
__device__ __forceinline__ unsigned lb_get(const unsigned long long *p, unsigned epoch, unsigned &flag, int *status) {
    for (int k = 0; k < LB_SPIN; k++) {
        const unsigned long long w = *(const volatile unsigned long long *)p;
        if ((unsigned)(w >> 34) == epoch) {
            flag = (unsigned)(w >> 32) & 3u;
            return (unsigned)w;
        }
    }
    atomicOr(status, ST_ITER_CAP);
    flag = LB_PREFIX;
    return 0u;
}

// the launch's next tile, for the whole CTA (sh: one shared int); the last
// tile leaves the ticket at zero
__device__ __forceinline__ int lb_tile(unsigned *ticket, int ntiles, int *sh) {
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(ticket, 1u);
        if ((int)t == ntiles - 1) *ticket = 0u;
        *sh = (int)t;
    }
    __syncthreads();
    return *sh;
}

// dst(i, prefix, value) for every i < n of src(i)'s exclusive prefix sums,
// dst.total(sum) once.  gridDim.y: independent scans y (src.y, dst.y), each
// with its own status words and ticket.
template <class Src, class Dst>
__global__ void __launch_bounds__(LB_T) k_scan_lb(Src src, Dst dst, int n, int ntiles, unsigned long long *st,
                                                  unsigned *ticket, unsigned epoch, int *status) {
    __shared__ int sh_tile, sh_ex, ws[LB_T / 32];
    const int y = blockIdx.y;
    st += (size_t)y * ntiles;
    const int tile = lb_tile(ticket + y, ntiles, &sh_tile);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int base = tile * LB_TILE + tid * LB_K;
    int v[LB_K], sum = 0;
#pragma unroll
    for (int k = 0; k < LB_K; k++) {
        v[k] = base + k < n ? src(y, base + k) : 0;
        sum += v[k];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    int off = x - sum, tot = 0;
#pragma unroll
    for (int k = 0; k < LB_T / 32; k++) {
        off += k < w ? ws[k] : 0;
        tot += ws[k];
    }
    if (w == 0) {  // look back, 32 tiles at a time
        if (lane == 0) lb_put(st + tile, epoch, tile == 0 ? LB_PREFIX : LB_SUM, (unsigned)tot);
        unsigned ex = 0;
        for (int p = tile - 1; p >= 0; p -= 32) {
            unsigned flag = LB_PREFIX, val = 0;
            if (p - lane >= 0) val = lb_get(st + p - lane, epoch, flag, status);
            const unsigned done = __ballot_sync(0xffffffffu, flag == LB_PREFIX);
            const int last = done ? __ffs(done) - 1 : 31;
            unsigned a = lane <= last ? val : 0u;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            ex += a;
            if (done) break;
        }
        if (lane == 0) {
            if (tile > 0) lb_put(st + tile, epoch, LB_PREFIX, ex + (unsigned)tot);
            sh_ex = (int)ex;
        }
    }
    __syncthreads();
    off += sh_ex;
#pragma unroll
    for (int k = 0; k < LB_K; k++) {
        if (base + k < n) dst(y, base + k, off, v[k]);
        off += v[k];
    }
    if (tile == ntiles - 1 && tid == LB_T - 1) dst.total(y, off);
}

template <class Src, class Dst>
int launch_scan_lb(Context *c, LookBack &lb, Src src, Dst dst, int n, int ny = 1) {
    const int ntiles = (n + LB_TILE - 1) / LB_TILE;
    int r = lb.reserve(c, (size_t)ntiles * ny);
    if (r) return r;
    { P3T_COUNT_LAUNCH(); k_scan_lb<<<dim3(ntiles, ny), LB_T, 0, c->stream>>>(src, dst, n, ntiles, lb.st.p, lb.ticket.p, lb.epoch, c->status); }
    return cuda_status(cudaGetLastError());
}

}  // namespace p3t
