// Device octree and interaction lists for the soft force.
//
// The caller side of the soft-force path, on the device: the contract of the
// host builder (csrc/tree.cpp, include/p3t_tree.h; in GPLUM, FDPS's
// TreeForForce with LONG_SYMMETRY search and quadrupole moments, called at
// src/main_p3t.cpp:344-355,581-587,672-676):
//   * 63-bit Morton keys on the root cube (side = 1.0001 x the largest
//     extent, anchored at the bodies' lower corner with margin
//     (side - extent)/2 on every axis), bodies in key order (ties by index);
//   * a node splits into one child per occupied octant while it holds more
//     than min(n_leaf_limit, n_group_limit) bodies (21 levels at most);
//   * i-groups are the highest nodes with at most n_group_limit bodies (or
//     leaves), in Morton order;
//   * a cell is opened when its search box (bodies +- 1.1 r_search) overlaps
//     the group's body box, or the group's search box overlaps the cell's
//     body box, or size^2 > theta^2 d^2 (d: cell centre of mass to the
//     group's body box); opened leaves give EPJ entries, unopened cells SPJ
//     entries (quadrupole about the centre of mass).
// Steps: bounding box; keys; a stable LSD radix sort of (key, index) in 8
// passes of 8 bits, one launch each (k_radix_pass), or all of these in one CTA
// for small systems (k_small_sort); the nodes of every level
// at once from the sorted keys (k_node_levels: which levels' nodes a body
// heads follows from the common prefixes of the keys around it); groups;
// moments and boxes bottom-up (leaves sum their bodies in key order, as the
// host builder; inner nodes combine children by the parallel-axis rule); and
// the walks, breadth first, one CTA per group over an order-keeping frontier
// (k_walk_bfs), with the walk of (group, node of the upper three levels) tasks
// as the fallback, taken in pre-order, each walking its subtree with the host
// builder's stack discipline (count, then fill).  Both give the host
// builder's lists entry for entry (SPJ entries name the same cells; node
// numbers are in level order here).  The lists go straight into the resident
// soft-force buffers.  The host waits three times a build, for the sizes of
// the node table, of the group table and of the lists.  Compiled with
// -fmad=false so the box and opening arithmetic rounds as the host builder's
// (-ffp-contract=off).
//
// Small builds are bound by launches and waits, large ones by memory passes.
// With the nodes one level at a time (five launches, a scan and a host wait for
// each of the up to 21 levels), a sort of three to five launches a pass and a
// second sort for the launch order, a build took 179 launches and 1.10 ms at
// 3000 bodies, 2.68 ms at 1,048,576 (ring) and 4.11 ms at 2,097,152 (0.3-3 AU);
// now 16 launches (24 above 8,192 bodies) and those of the levels' moments, 0.26,
// 1.37 and 2.36 ms.
#include <algorithm>
#include <cstdint>
#include <vector>

#include "../../include/gplum_p3t.h"
#include "p3t_capi_internal.cuh"
#include "p3t_engine.cuh"
#include "p3t_exact.cuh"

namespace p3t {

struct TNode {
    double ilo[3], ihi[3], olo[3], ohi[3];  // body box, search box (bodies +- 1.1 r_search)
    double com[3], size;
    int first, count, child0, nchild;
};

// FP32 copy of the walk's fields (rounded to nearest), for the ternary
// opening test below
struct TNodeF {
    float ilo[3], ihi[3], olo[3], ohi[3], com[3], size;
    int first, count, child0, nchild;
};

constexpr int RADIX_T = 256, RADIX_K = 8, RADIX_TILE = RADIX_T * RADIX_K;  // keys of a radix tile
constexpr int MAX_LEVEL = 21;                                             // levels below the root
constexpr int WALK_STACK = 256;

static inline int nblocks(long long n, int t = 256) { return (int)std::max<long long>(1, (n + t - 1) / t); }

// ---- bounding box and keys ------------------------------------------------------
// doubles as integers of the same order, for minima and maxima beside the FP64 pipe
__device__ __forceinline__ long long box_key(double x) {
    const long long b = __double_as_longlong(x);
    return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}
__device__ __forceinline__ double box_value(long long k) {
    return __longlong_as_double(k ^ (long long)((unsigned long long)(k >> 63) >> 1));
}
// b: box keys, the three minima and the three maxima -> the CTA's, in s[d][0]
struct BoxSmem {
    long long s[6][32];
};
__device__ __forceinline__ void box_none(long long *b) {
    for (int d = 0; d < 3; d++) {
        b[d] = box_key(1e300);
        b[3 + d] = box_key(-1e300);
    }
}
__device__ __forceinline__ void box_add(long long *b, int d, double x) {
    if (x != x) return;  // as fmin and fmax, which pass over NaN
    b[d] = min(b[d], box_key(x));
    b[3 + d] = max(b[3 + d], box_key(x));
}
__device__ __forceinline__ void box_reduce(long long *b, BoxSmem &B) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int d = 0; d < 6; d++)
        for (int o = 16; o > 0; o >>= 1) {
            const long long x = __shfl_xor_sync(0xffffffffu, b[d], o);
            b[d] = d < 3 ? min(b[d], x) : max(b[d], x);
        }
    if (lane == 0)
        for (int d = 0; d < 6; d++) B.s[d][w] = b[d];
    __syncthreads();
    if (threadIdx.x < 6) {
        const int d = threadIdx.x;
        long long x = B.s[d][0];
        for (int k = 1; k < nw; k++) x = d < 3 ? min(x, B.s[d][k]) : max(x, B.s[d][k]);
        B.s[d][0] = x;
    }
    __syncthreads();
}
// root cube as the host builder: out = {base.xyz, size, scale}; anchored at
// the lower corner, so a thin axis is not cut at coarse levels
__device__ __forceinline__ void root_cube(const BoxSmem &B, double *out) {
    double lo[3], ext = 0.;
    for (int d = 0; d < 3; d++) {
        lo[d] = box_value(B.s[d][0]);
        ext = fmax(ext, box_value(B.s[3 + d][0]) - lo[d]);
    }
    const double size = ext * 1.0001 + 1e-300;
    for (int d = 0; d < 3; d++) out[d] = lo[d] - 0.5 * (size - ext);
    out[3] = size;
    out[4] = double(1 << 21) / size;
}
// The last CTA to finish combines the partial boxes.
__global__ void __launch_bounds__(256) k_bbox(const double *pos, int n, double *part, unsigned *done, double *out) {
    __shared__ BoxSmem B;
    __shared__ bool last;
    const int tid = threadIdx.x;
    long long b[6];
    box_none(b);
    for (int i = blockIdx.x * blockDim.x + tid; i < n; i += gridDim.x * blockDim.x)
        for (int d = 0; d < 3; d++) box_add(b, d, pos[3 * i + d]);
    box_reduce(b, B);
    if (tid < 6) {
        __stcg(&part[6 * blockIdx.x + tid], box_value(B.s[tid][0]));
        __threadfence();
    }
    __syncthreads();
    if (tid == 0) {
        last = atomicAdd(done, 1u) == gridDim.x - 1;
        if (last) *done = 0u;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    box_none(b);
    for (int k = tid; k < (int)gridDim.x; k += 256)
        for (int d = 0; d < 3; d++) {
            b[d] = min(b[d], box_key(__ldcg(&part[6 * k + d])));
            b[3 + d] = max(b[3 + d], box_key(__ldcg(&part[6 * k + 3 + d])));
        }
    box_reduce(b, B);
    if (tid == 0) root_cube(B, out);
}

__device__ __forceinline__ unsigned long long spread21(unsigned long long v) {
    v &= 0x1fffffULL;
    v = (v | v << 32) & 0x1f00000000ffffULL;
    v = (v | v << 16) & 0x1f0000ff0000ffULL;
    v = (v | v << 8) & 0x100f00f00f00f00fULL;
    v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
    v = (v | v << 2) & 0x1249249249249249ULL;
    return v;
}

__device__ __forceinline__ unsigned long long morton_key(const double *pos, int i, double b0, double b1, double b2, double sc) {
    unsigned long long c[3];
    for (int d = 0; d < 3; d++) {
        const double u = (pos[3 * i + d] - (d == 0 ? b0 : (d == 1 ? b1 : b2))) * sc;
        long long v = (long long)u;
        v = v < 0 ? 0 : (v > (1 << 21) - 1 ? (1 << 21) - 1 : v);
        c[d] = (unsigned long long)v;
    }
    return (spread21(c[0]) << 2) | (spread21(c[1]) << 1) | spread21(c[2]);
}

// keys and the counts of each of their eight digits (ghist[8][256], zeroed)
__global__ void __launch_bounds__(256) k_keys(const double *pos, int n, const double *root, unsigned long long *key,
                                              int *idx, unsigned *ghist) {
    __shared__ unsigned h[8][256];
    const int tid = threadIdx.x;
    for (int p = 0; p < 8; p++) h[p][tid] = 0u;
    __syncthreads();
    const double b0 = root[0], b1 = root[1], b2 = root[2], sc = root[4];
    for (int base = blockIdx.x * RADIX_TILE; base < min(n, (int)(blockIdx.x + 1) * RADIX_TILE); base += 256) {
        const int i = base + tid;
        const unsigned in = __ballot_sync(0xffffffffu, i < n);
        if (i >= n) continue;
        const unsigned long long k = morton_key(pos, i, b0, b1, b2, sc);
        key[i] = k;
        idx[i] = i;
#pragma unroll
        for (int p = 0; p < 8; p++) {
            const int d = (int)(k >> (8 * p)) & 255;
            int same;
            const unsigned all = __match_all_sync(in, d, &same);
            if (!same) atomicAdd(&h[p][d], 1u);
            else if ((tid & 31) == __ffs(all) - 1) atomicAdd(&h[p][d], (unsigned)__popc(all));
        }
    }
    __syncthreads();
    for (int p = 0; p < 8; p++)
        if (h[p][tid]) atomicAdd(&ghist[256 * p + tid], h[p][tid]);
}

// ---- stable LSD radix sort of (key, index) -----------------------------------------
// One pass over an 8-bit digit in one launch: a tile ranks its keys by digit
// (warp match, per-warp counts, so equal digits keep their order), publishes
// its digit counts, sums its predecessors' by decoupled look-back (one thread
// a digit) and writes its keys digit by digit from shared memory, so that keys
// are read and written once a pass.  200,000 keys: 11.7 us a pass (ncu) against
// 29 us in three to five launches (counts, scan, scatter).
__global__ void __launch_bounds__(RADIX_T) k_radix_pass(const unsigned long long *__restrict__ key,
                                                        const int *__restrict__ idx, int n, int ntiles, int shift,
                                                        const unsigned *__restrict__ ghist, unsigned long long *st,
                                                        unsigned *ticket, unsigned epoch, int *status,
                                                        unsigned long long *__restrict__ key_out,
                                                        int *__restrict__ idx_out) {
    constexpr int NW = RADIX_T / 32;
    __shared__ unsigned long long sk[RADIX_TILE];
    __shared__ int si[RADIX_TILE], wc[NW][256], dstart[256], dbase[256], ws[2][NW], sh_tile;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int tile = lb_tile(ticket, ntiles, &sh_tile);
    for (int j = 0; j < NW; j++) wc[j][tid] = 0;
    __syncthreads();
    const int base = tile * RADIX_TILE, cnt = min(RADIX_TILE, n - base);
    unsigned long long kv[RADIX_K];
    int iv[RADIX_K], rk[RADIX_K];
#pragma unroll
    for (int r = 0; r < RADIX_K; r++) {
        const int q = w * (32 * RADIX_K) + r * 32 + lane;
        kv[r] = q < cnt ? key[base + q] : 0ULL;
        iv[r] = q < cnt ? idx[base + q] : 0;
    }
#pragma unroll
    for (int r = 0; r < RADIX_K; r++) {
        const bool valid = w * (32 * RADIX_K) + r * 32 + lane < cnt;
        const int d = valid ? (int)(kv[r] >> shift) & 255 : 256;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int before = __popc(peers & ((1u << lane) - 1u));
        int pre = 0;
        if (valid) pre = wc[w][d];
        __syncwarp();
        if (valid && before == 0) wc[w][d] = pre + __popc(peers);
        __syncwarp();
        rk[r] = pre + before;
    }
    __syncthreads();
    // thread d: the digit's keys in the tile, by warp
    int total = 0;
#pragma unroll
    for (int j = 0; j < NW; j++) {
        const int c = wc[j][tid];
        wc[j][tid] = total;
        total += c;
    }
    unsigned long long *const mine = st + (size_t)tile * 256 + tid;
    lb_put(mine, epoch, tile == 0 ? LB_PREFIX : LB_SUM, (unsigned)total);
    // exclusive sums over the digits: of the tile's counts and of all keys'
    const int g = (int)ghist[tid];
    int x = total, y = g;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, x, o), b = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) {
            x += a;
            y += b;
        }
    }
    if (lane == 31) {
        ws[0][w] = x;
        ws[1][w] = y;
    }
    __syncthreads();
    int ds = x - total, gs = y - g;
    for (int k = 0; k < w; k++) {
        ds += ws[0][k];
        gs += ws[1][k];
    }
    unsigned ex = 0;
    for (int p = tile - 1; p >= 0; p--) {
        unsigned flag;
        ex += lb_get(st + (size_t)p * 256 + tid, epoch, flag, status);
        if (flag == LB_PREFIX) break;
    }
    if (tile > 0) lb_put(mine, epoch, LB_PREFIX, ex + (unsigned)total);
    dstart[tid] = ds;
    dbase[tid] = gs + (int)ex - ds;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RADIX_K; r++) {
        if (w * (32 * RADIX_K) + r * 32 + lane >= cnt) continue;
        const int d = (int)(kv[r] >> shift) & 255;
        const int q = dstart[d] + wc[w][d] + rk[r];
        sk[q] = kv[r];
        si[q] = iv[r];
    }
    __syncthreads();
    for (int q = tid; q < cnt; q += RADIX_T) {
        const unsigned long long k = sk[q];
        // (a prefix that the wait's limit cut short stays inside the arrays)
        const int o = min(max(dbase[(int)(k >> shift) & 255] + q, 0), n - 1);
        key_out[o] = k;
        idx_out[o] = si[q];
    }
}

// Root cube, keys and sort of at most SMALL_N bodies by one CTA, keys and indices
// in shared memory: ten launches' work (box, keys, eight passes of 7 us, whose
// tiles hold 2,048 keys: 85 us at 3,000 bodies) in one.  Eight keys a thread and
// 132 KB of shared memory are the limit; above it the passes' tiles spread over
// the SMs.
constexpr int SMALL_T = 1024, SMALL_N = 8192, SMALL_W = SMALL_T / 32;
struct SmallSmem {
    unsigned long long k[SMALL_N];
    int i[SMALL_N];
    int wc[SMALL_W][256];
    int start[256], ws[8], most;
    double root[5];
    BoxSmem box;
};
template <int K>
__device__ __forceinline__ void small_sort(SmallSmem &M, const double *pos, int n, double *root,
                                           unsigned long long *__restrict__ key_out, int *__restrict__ idx_out) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    long long b[6];
    box_none(b);
    for (int i = tid; i < n; i += SMALL_T)
        for (int d = 0; d < 3; d++) box_add(b, d, pos[3 * i + d]);
    box_reduce(b, M.box);
    if (tid == 0) root_cube(M.box, M.root);
    __syncthreads();
    if (tid < 5) root[tid] = M.root[tid];
    unsigned long long kv[K];
    int iv[K], rk[K];
#pragma unroll
    for (int r = 0; r < K; r++) {
        const int q = w * (32 * K) + r * 32 + lane;
        kv[r] = q < n ? morton_key(pos, q, M.root[0], M.root[1], M.root[2], M.root[4]) : 0ULL;
        iv[r] = q;
    }
#pragma unroll 1
    for (int shift = 0; shift < 64; shift += 8) {
        for (int j = lane; j < 256; j += 32) M.wc[w][j] = 0;
        if (tid == 0) M.most = 0;
        __syncwarp();
        // as k_radix_pass: ranks among the warp's keys of the digit, in order
#pragma unroll
        for (int r = 0; r < K; r++) {
            const bool valid = w * (32 * K) + r * 32 + lane < n;
            const int d = valid ? (int)(kv[r] >> shift) & 255 : 256;
            const unsigned peers = __match_any_sync(0xffffffffu, d);
            const int before = __popc(peers & ((1u << lane) - 1u));
            int pre = 0;
            if (valid) pre = M.wc[w][d];
            __syncwarp();
            if (valid && before == 0) M.wc[w][d] = pre + __popc(peers);
            __syncwarp();
            rk[r] = pre + before;
        }
        __syncthreads();
        int total = 0, x = 0;
        if (tid < 256) {
            for (int j = 0; j < SMALL_W; j++) {
                const int c = M.wc[j][tid];
                M.wc[j][tid] = total;
                total += c;
            }
            if (total == n) M.most = 1;  // one digit for all: the order stays
            x = total;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int a = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += a;
            }
            if (lane == 31) M.ws[w] = x;
        }
        __syncthreads();
        if (M.most) {
            __syncthreads();
            continue;
        }
        if (tid < 256) {
            int s = x - total;
            for (int k = 0; k < w; k++) s += M.ws[k];
            M.start[tid] = s;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < K; r++) {
            if (w * (32 * K) + r * 32 + lane >= n) continue;
            const int d = (int)(kv[r] >> shift) & 255, q = M.start[d] + M.wc[w][d] + rk[r];
            M.k[q] = kv[r];
            M.i[q] = iv[r];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < K; r++) {
            const int q = w * (32 * K) + r * 32 + lane;
            if (q < n) {
                kv[r] = M.k[q];
                iv[r] = M.i[q];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < K; r++) {
        const int q = w * (32 * K) + r * 32 + lane;
        if (q >= n) continue;
        key_out[q] = kv[r];
        idx_out[q] = iv[r];
    }
}
__global__ void __launch_bounds__(SMALL_T) k_small_sort(const double *pos, int n, double *root, unsigned long long *key_out,
                                                        int *idx_out) {
    extern __shared__ __align__(16) unsigned char small_raw[];
    SmallSmem &M = *reinterpret_cast<SmallSmem *>(small_raw);
    if (n <= 2 * SMALL_T) small_sort<2>(M, pos, n, root, key_out, idx_out);
    else if (n <= 4 * SMALL_T) small_sort<4>(M, pos, n, root, key_out, idx_out);
    else small_sort<8>(M, pos, n, root, key_out, idx_out);
}

// ---- the nodes of every level --------------------------------------------------------
// 3-bit digits that two keys share from the top (21: equal)
__device__ __forceinline__ int common_digits(unsigned long long a, unsigned long long b) {
    const unsigned long long x = a ^ b;
    return x == 0ULL ? MAX_LEVEL : (__clzll((long long)x) - 1) / 3;
}

// The levels whose node body k (in key order) heads.  The cell of level L
// around k is a node when the cell of level L - 1 around k holds more than
// `limit` bodies, and k heads it when it does not hold k - 1: L from
// common_digits(k - 1, k) + 1 on, up to one below the deepest cell around k of
// more than `limit` bodies (MAX_LEVEL at most).  A cell of level l around k
// holds more than `limit` bodies when some limit + 1 consecutive keys around k
// share l digits.  lo > hi: none.  The root is always a node, headed by body 0.
__device__ __forceinline__ void head_levels(const unsigned long long *__restrict__ key, int n, int k, int limit,
                                            int &lo, int &hi) {
    const unsigned long long me = key[k];
    lo = k == 0 ? 0 : common_digits(key[k - 1], me) + 1;
    int m = -1;  // deepest level of a cell of more than `limit` bodies around k
    if (limit <= 16) {
        for (int j = max(0, k - limit); j <= k && j + limit < n; j++) m = max(m, common_digits(key[j], key[j + limit]));
    } else {
        // bodies around k in the cell of level l, up to `limit` on each side,
        // by bisection; the deepest level by bisection
        int a = -1, b = MAX_LEVEL;
        while (a < b) {
            const int l = (a + b + 1) >> 1;
            int p = max(0, k - limit), q = k;
            while (p < q) {
                const int mid = (p + q) >> 1;
                if (common_digits(key[mid], me) >= l) q = mid;
                else p = mid + 1;
            }
            const int first = p;
            p = k;
            q = min(n - 1, k + limit);
            while (p < q) {
                const int mid = (p + q + 1) >> 1;
                if (common_digits(key[mid], me) >= l) p = mid;
                else q = mid - 1;
            }
            if (p - first + 1 > limit) a = l;
            else b = l - 1;
        }
        m = a;
    }
    hi = m >= 0 ? min(m, MAX_LEVEL - 1) + 1 : (k == 0 ? 0 : -1);
}

// per body its levels, per block and level the bodies that head a node
// (cnt[level][block]); blocks of 256 bodies
__global__ void __launch_bounds__(256) k_node_levels(const unsigned long long *__restrict__ key, int n, int limit,
                                                     unsigned short *lev, int *cnt) {
    __shared__ int wc[8][MAX_LEVEL + 1];
    const int k = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int lo = 1, hi = 0;
    if (k < n) {
        head_levels(key, n, k, limit, lo, hi);
        lev[k] = (unsigned short)(lo | ((hi + 1) << 8));
    }
    for (int L = 0; L <= MAX_LEVEL; L++) {
        const unsigned b = __ballot_sync(0xffffffffu, lo <= L && L <= hi);
        if (lane == 0) wc[w][L] = __popc(b);
    }
    __syncthreads();
    if (threadIdx.x <= MAX_LEVEL) {
        int c = 0;
        for (int j = 0; j < 8; j++) c += wc[j][threadIdx.x];
        cnt[threadIdx.x * gridDim.x + blockIdx.x] = c;
    }
}
// their exclusive sums, level after level: the number of each block's first
// node of a level; lstart[level] (and, last, the node count)
struct LevelScan {
    const int *cnt;
    int *off, *lstart;
    int nblk;
    __device__ int operator()(int, int i) const { return cnt[i]; }
    __device__ void operator()(int, int i, int prefix, int) const {
        off[i] = prefix;
        if (i % nblk == 0) lstart[i / nblk] = prefix;
    }
    __device__ void total(int, int t) const { lstart[MAX_LEVEL + 1] = t; }
};

// The nodes: body k writes those it heads, numbered in level order.  A node
// with a deeper one headed by the same body is split, the body's deepest is
// a leaf.  nch (zeroed) counts children; leaves and each level's inner nodes
// are listed (list[nn..]: the inner nodes of level L from lstart[L] on;
// icnt[L] of them; icnt[MAX_LEVEL + 1] leaves).
__global__ void __launch_bounds__(256) k_nodes(const unsigned long long *__restrict__ key, int n,
                                               const unsigned short *__restrict__ lev, const int *__restrict__ off,
                                               const int *__restrict__ lstart, const double *__restrict__ root, int nn,
                                               TNode *nd, int *parent, int *nch, int *list, int *icnt) {
    __shared__ int wc[8][MAX_LEVEL + 1];
    const int k = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int lo = 1, hi = 0;
    unsigned long long me = 0;
    if (k < n) {
        lo = lev[k] & 255;
        hi = (lev[k] >> 8) - 1;
        me = key[k];
    }
    for (int L = 0; L <= MAX_LEVEL; L++) {
        const unsigned b = __ballot_sync(0xffffffffu, lo <= L && L <= hi);
        if (lane == 0) wc[w][L] = __popc(b);
    }
    __syncthreads();
    const unsigned lt = (1u << lane) - 1u;
    double size = root[3];
    int up = 0, leaf = -1;  // heads of the level above up to k; this body's leaf
    for (int L = 0; L <= MAX_LEVEL; L++, size *= 0.5) {
        const bool head = lo <= L && L <= hi, inner = head && L < hi;
        const unsigned b = __ballot_sync(0xffffffffu, head), bi = __ballot_sync(0xffffffffu, inner);
        int c = off[L * gridDim.x + blockIdx.x] + __popc(b & lt);
        for (int j = 0; j < w; j++) c += wc[j][L];
        int at = 0;
        if (bi) {
            if (lane == 0) at = atomicAdd(&icnt[L], __popc(bi));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(bi & lt);
        }
        if (head) {
            // its end: the first later key outside the cell
            const int sh = 3 * (MAX_LEVEL - L);
            const unsigned long long pre = L == 0 ? 0ULL : me >> sh;
            int p = k, step = 1;  // key[p] inside
            while (p + step < n && (L == 0 || (key[p + step] >> sh) == pre)) {
                p += step;
                step *= 2;
            }
            int q = min(p + step, n);  // n or outside
            while (q - p > 1) {
                const int mid = (p + q) >> 1;
                if (L == 0 || (key[mid] >> sh) == pre) p = mid;
                else q = mid;
            }
            TNode &N = nd[c];
            N.first = k;
            N.count = q - k;
            N.size = size;
            // a split node's first child is headed by the same body, one level down
            N.child0 = -1;
            const int par = L == 0 ? -1 : up - 1;
            parent[c] = par;
            if (L > 0) atomicAdd(&nch[par], 1);
            if (L > lo) nd[par].child0 = c;
            if (inner) list[nn + lstart[L] + at] = c;
            else leaf = c;
        }
        up = c + (head ? 1 : 0);
    }
    const unsigned bl = __ballot_sync(0xffffffffu, leaf >= 0);
    if (bl) {
        int at = 0;
        if (lane == 0) at = atomicAdd(&icnt[MAX_LEVEL + 1], __popc(bl));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(bl & lt);
        if (leaf >= 0) list[at] = leaf;
    }
}

// ---- moments and boxes, bottom-up -------------------------------------------------------
// A node's moments and boxes by NL lanes, one body or child each: a leaf sums its
// bodies in key order (the host builder's sums), an inner node combines its
// children in child order by the parallel-axis rule.  What a body or child adds
// is computed in its own lane; each component's sum then runs in key (child)
// order in a lane of its own, from shared memory, so the sums round as one
// thread's would.  Box bounds do not depend on the order: their minima and maxima
// are integer comparisons of the doubles' ordered bits.
//
// What bounds it: in a large tree the FP64 pipe (one warp instruction per 19
// cycles of an SM), about 10 instructions a node, as one thread per node needs
// once the lanes its warp idles behind the fullest node are counted (with FP64
// minima it needed 12 to 16); in a small one the chain of dependent FP64
// operations, 64 cycles each: about 40 a level instead of 350.  The whole tree,
// with the one-CTA sort below 8,192 bodies: 3,000 bodies 0.36 -> 0.26 ms, 50,000
// 0.47 -> 0.37, 200,000 0.60 -> 0.51, 1M 1.48 -> 1.37, 2M 2.42 -> 2.36.
constexpr int NL = 8, MOM_T = 128;
struct MomentSmem {
    double v[MOM_T / NL][6][NL];
};
// Lane u of node c (c < 0: no node; its lanes only keep the others company).
// Children are read through L2 (ld.cg): other CTAs of the same launch may have
// written them.
__device__ void node_moments(int c, MomentSmem &M, TNode *nd, TNodeF *nf, SPJRec *spj, const int *order,
                             const double *pos, const double *mass, const double *rs) {
    const int u = threadIdx.x % NL, slot = threadIdx.x / NL;
    double(*v)[NL] = M.v[slot];
    int first = 0, count = 0, child0 = 0, nchild = 0;
    double size = 0.;
    if (c >= 0) {
        const TNode &N = nd[c];
        nchild = __ldcg(&N.nchild);
        child0 = __ldcg(&N.child0);
        first = N.first;
        count = N.count;
        size = N.size;
    }
    const bool leaf = nchild == 0;
    const int items = leaf ? count : nchild;
    int most = items;  // of the warp's nodes (a leaf at the deepest level may hold more than NL)
    for (int o = NL; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    const long long inf = box_key(1e300), ninf = box_key(-1e300);
    long long lo[6] = {inf, inf, inf, inf, inf, inf}, hi[6] = {ninf, ninf, ninf, ninf, ninf, ninf};  // inner, outer
    double sum = 0.;  // lanes 0..3: mass and mass-weighted position
    double m = 0., x = 0., y = 0., z = 0.;
    int child = 0;
    for (int k0 = 0; k0 < most; k0 += NL) {
        const bool mine = k0 + u < items;
        if (mine && leaf) {
            const int p = order[first + k0 + u];
            x = pos[3 * p]; y = pos[3 * p + 1]; z = pos[3 * p + 2];
            m = mass[p];
            const double r = 1.1 * rs[p];
            const double w[3] = {x, y, z};
            for (int d = 0; d < 3; d++) {
                const double a = w[d] - r, b = w[d] + r;
                // as fmin and fmax, which pass over NaN
                if (w[d] == w[d]) { lo[d] = min(lo[d], box_key(w[d])); hi[d] = max(hi[d], box_key(w[d])); }
                if (a == a) lo[3 + d] = min(lo[3 + d], box_key(a));
                if (b == b) hi[3 + d] = max(hi[3 + d], box_key(b));
            }
        } else if (mine) {
            child = child0 + u;
            m = __ldcg(&spj[child].mass);
            x = __ldcg(&spj[child].pos[0]); y = __ldcg(&spj[child].pos[1]); z = __ldcg(&spj[child].pos[2]);
            for (int d = 0; d < 3; d++) {
                lo[d] = box_key(__ldcg(&nd[child].ilo[d]));
                hi[d] = box_key(__ldcg(&nd[child].ihi[d]));
                lo[3 + d] = box_key(__ldcg(&nd[child].olo[d]));
                hi[3 + d] = box_key(__ldcg(&nd[child].ohi[d]));
            }
        }
        v[0][u] = m;  // (stale beyond the items, and not summed)
        v[1][u] = m * x;
        v[2][u] = m * y;
        v[3][u] = m * z;
        __syncwarp();
        if (u < 4)
            for (int k = 0; k < min(NL, items - k0); k++) sum += v[u][k];
        __syncwarp();
    }
    const int l0 = (threadIdx.x & 31) - u;
    const double mt = __shfl_sync(0xffffffffu, sum, l0);
    if (mt != 0. && u >= 1 && u < 4) sum = div_rn(sum, mt);
    const double cx = __shfl_sync(0xffffffffu, sum, l0 + 1), cy = __shfl_sync(0xffffffffu, sum, l0 + 2),
                 cz = __shfl_sync(0xffffffffu, sum, l0 + 3);
    double q = 0.;  // lanes 0..5: the quadrupole's components
    for (int k0 = 0; k0 < most; k0 += NL) {
        const bool mine = k0 + u < items;
        if (most > NL && mine && leaf) {
            const int p = order[first + k0 + u];
            x = pos[3 * p]; y = pos[3 * p + 1]; z = pos[3 * p + 2];
            m = mass[p];
        }
        const double dx = x - cx, dy = y - cy, dz = z - cz, mx = m * dx, my = m * dy, mz = m * dz;
        double t[6] = {mx * dx, my * dy, mz * dz, mx * dy, mx * dz, my * dz};
        if (mine && !leaf) {
            const double *Q = &spj[child].xx;
            for (int k = 0; k < 6; k++) t[k] = __ldcg(Q + k) + t[k];
        }
        for (int k = 0; k < 6; k++) v[k][u] = t[k];
        __syncwarp();
        if (u < 6)
            for (int k = 0; k < min(NL, items - k0); k++) q += v[u][k];
        __syncwarp();
    }
    for (int d = 0; d < 6; d++)
        for (int o = 1; o < NL; o <<= 1) {
            lo[d] = min(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = max(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    if (c < 0) return;
    TNode &N = nd[c];
    SPJRec &S = spj[c];
    TNodeF &F = nf[c];  // the walk's FP32 copy
    if (u < 3) {
        auto pick = [&](const long long *a) { return box_value(u == 0 ? a[0] : u == 1 ? a[1] : a[2]); };
        const double il = pick(lo), ih = pick(hi), ol = pick(lo + 3), oh = pick(hi + 3), cd = u == 0 ? cx : u == 1 ? cy : cz;
        N.ilo[u] = il; N.ihi[u] = ih; N.olo[u] = ol; N.ohi[u] = oh;
        N.com[u] = cd;
        S.pos[u] = cd;
        F.ilo[u] = (float)il; F.ihi[u] = (float)ih; F.olo[u] = (float)ol; F.ohi[u] = (float)oh;
        F.com[u] = (float)cd;
    }
    if (u < 6) (&S.xx)[u] = q;
    if (u == 6) {
        S.mass = mt;
        F.size = (float)size;
    }
    if (u == 7) {
        F.first = first;
        F.count = count;
        F.child0 = child0;
        F.nchild = nchild;
    }
}

// one level (nodes lo..hi-1) per launch, deepest level first
__global__ void __launch_bounds__(MOM_T) k_moments(int lo, int hi, TNode *nd, TNodeF *nf, SPJRec *spj, const int *order,
                                                   const double *pos, const double *mass, const double *rs) {
    __shared__ MomentSmem M;
    const int c = lo + (blockIdx.x * MOM_T + threadIdx.x) / NL;
    node_moments(c < hi ? c : -1, M, nd, nf, spj, order, pos, mass, rs);
}

// Moments in lane-dense launches: the nodes of a list, all leaves at once (their
// body sums are the bulk of the FP64 work) or the inner nodes of a level, deepest
// first.  A launch over all nodes of a level, or one climbing thread per finished
// child, left most lanes of the FP64 pipe's warp instructions idle.
__global__ void __launch_bounds__(MOM_T) k_moments_list(const int *list, const int *count, TNode *nd, TNodeF *nf,
                                                        SPJRec *spj, const int *order, const double *pos,
                                                        const double *mass, const double *rs) {
    __shared__ MomentSmem M;
    const int t = (int)(((long long)blockIdx.x * MOM_T + threadIdx.x) / NL), m = *count;
    if ((t & ~(32 / NL - 1)) >= m) return;  // none of the warp's nodes
    node_moments(t < m ? list[t] : -1, M, nd, nf, spj, order, pos, mass, rs);
}
// the inner nodes of levels from..to (deepest first) in one CTA, level after
// level: runs of levels of few nodes -- the top of the tree, and the deep
// chains around close pairs -- whose launches would cost more than their work.
// TOP_NODES: the CTA's SM takes 3 us for 32 nodes, a launch 5 us.
constexpr int TOP_NODES = 32;
__global__ void __launch_bounds__(MOM_T) k_moments_run(int from, int to, const int *lstart, const int *inner,
                                                       const int *icnt, TNode *nd, TNodeF *nf, SPJRec *spj,
                                                       const int *order, const double *pos, const double *mass,
                                                       const double *rs) {
    __shared__ MomentSmem M;
    for (int L = from; L >= to; L--) {
        const int m = icnt[L], t0 = threadIdx.x / NL;
        for (int t = t0; (t & ~(32 / NL - 1)) < m; t += MOM_T / NL)
            node_moments(t < m ? inner[lstart[L] + t] : -1, M, nd, nf, spj, order, pos, mass, rs);
        __threadfence();
        __syncthreads();
    }
}

// ---- groups ---------------------------------------------------------------------------------
// also the children counts into the node records
__global__ void k_group_mark(int nn, TNode *nd, const int *parent, const int *nch, int ngl, int *gmark) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nn) return;
    TNode &N = nd[c];
    const int m = nch[c];
    N.nchild = m;
    const bool cand = N.count <= ngl || m == 0;
    const bool top = (c == 0) || nd[parent[c]].count > ngl;
    if (cand && top) gmark[N.first] = c + 1;
}
// the groups in key order (a scan over the bodies): node and first body
struct GroupScan {
    const int *gmark;
    int *gnode, *i_off, *ng;
    int n;
    __device__ int operator()(int, int k) const { return gmark[k] > 0; }
    __device__ void operator()(int, int k, int prefix, int v) const {
        if (!v) return;
        gnode[prefix] = gmark[k] - 1;
        i_off[prefix] = k;
    }
    __device__ void total(int, int t) const {
        i_off[t] = n;
        *ng = t;
    }
};

// ---- walk --------------------------------------------------------------------------------------
__device__ __forceinline__ bool box_overlap(const double *alo, const double *ahi, const double *blo,
                                            const double *bhi) {
    for (int d = 0; d < 3; d++)
        if (ahi[d] < blo[d] || bhi[d] < alo[d]) return false;
    return true;
}

__device__ __forceinline__ double box_dist2(const double *lo, const double *hi, const double *x) {
    double s = 0.;
    for (int d = 0; d < 3; d++) {
        double e = 0.;
        if (x[d] < lo[d]) e = lo[d] - x[d];
        else if (x[d] > hi[d]) e = x[d] - hi[d];
        s += e * e;
    }
    return s;
}

// The walk split into tasks: pair (group g, top node t) for each of the
// ntop nodes of the upper `depth` levels, taken in the tree's pre-order.  The
// open test of every pair goes first (k_walk_open); then a pair is reached
// when all its top-node ancestors are open for g, and it contributes: an SPJ
// entry (reached, not open), its bodies (reached, open leaf), nothing
// (reached, open, above the split depth: its children are pairs of their
// own), or the depth-first walk of its subtree (reached, open, at the split
// depth).  Pairs in (group, pre-order) order concatenate to the single walk's
// output, entry for entry.
__device__ __forceinline__ bool cell_open(const TNode &C, const double *gilo, const double *gihi,
                                          const double *golo, const double *gohi, double theta2) {
    const bool near = box_overlap(C.olo, C.ohi, gilo, gihi) || box_overlap(golo, gohi, C.ilo, C.ihi);
    return near || (C.size * C.size > theta2 * box_dist2(gilo, gihi, C.com));
}

// Ternary comparisons on FP32 copies of doubles (each within 2^-24 relative
// of its double): +1 when a < b certainly holds for the doubles, -1 when
// a >= b certainly holds, 0 when the copies cannot tell.  b - a differs from
// the FP32 difference of the copies by less than 1.8e-7 (|a| + |b|) (two
// conversions and one rounded subtraction); the margin is 2.5e-7.
__device__ __forceinline__ int lt3(float a, float b) {
    const float d = b - a, e = 2.5e-7f * (fabsf(a) + fabsf(b)) + 1e-30f;
    return d > e ? 1 : (d < -e ? -1 : 0);
}
// box overlap (no dimension separated): +1 yes, -1 no, 0 unknown
__device__ __forceinline__ int overlap3(const float *alo, const float *ahi, const float *blo, const float *bhi) {
    int res = 1;
    for (int d = 0; d < 3; d++) {
        const int s1 = lt3(ahi[d], blo[d]), s2 = lt3(bhi[d], alo[d]);
        if (s1 == 1 || s2 == 1) return -1;  // separated for sure
        if (s1 == 0 || s2 == 0) res = 0;
    }
    return res;
}
// The cell test of the host builder on the FP32 copies: +1 open, -1 closed,
// 0 unknown.  The distance from the group box carries an absolute error
// below E_d = 2.5e-7 (|x| + |lo or hi|) per dimension, so d^2 is within
// B = sum(2 |e_d| E_d + E_d^2) + 4e-7 d^2; sizes and theta^2 carry 2e-7
// relative, covered by the 4e-7 factors.
__device__ __forceinline__ int open3(const TNodeF &C, const float *gilo, const float *gihi, const float *golo,
                                     const float *gohi, float theta2) {
    const int a = overlap3(C.olo, C.ohi, gilo, gihi);
    if (a == 1) return 1;
    const int b = overlap3(golo, gohi, C.ilo, C.ihi);
    if (b == 1) return 1;
    if (a == 0 || b == 0) return 0;
    float d2 = 0.f, bnd = 0.f;
    for (int d = 0; d < 3; d++) {
        const float x = C.com[d];
        float e = 0.f, E = 0.f;
        if (x < gilo[d]) {
            e = gilo[d] - x;
            E = 2.5e-7f * (fabsf(x) + fabsf(gilo[d]));
        } else if (x > gihi[d]) {
            e = x - gihi[d];
            E = 2.5e-7f * (fabsf(x) + fabsf(gihi[d]));
        } else {
            E = 2.5e-7f * (fabsf(x) + fmaxf(fabsf(gilo[d]), fabsf(gihi[d])));
        }
        d2 += e * e;
        bnd += 2.f * e * E + E * E;
    }
    bnd += 4e-7f * d2 + 1e-37f;
    const float s2 = C.size * C.size;
    if (s2 * (1.f - 4e-7f) > theta2 * (d2 + bnd) * (1.f + 4e-7f)) return 1;
    if (s2 * (1.f + 4e-7f) < theta2 * fmaxf(d2 - bnd, 0.f) * (1.f - 4e-7f)) return -1;
    return 0;
}

__global__ void k_walk_open(const TNode *nd, const TNodeF *nf, const int *gnode, int ng, const int *top, int ntop,
                            double theta2, float theta2f, unsigned char *ostat) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (long long)ng * ntop) return;
    const int g = (int)(p / ntop), t = (int)(p - (long long)g * ntop);
    const TNodeF &G = nf[gnode[g]];
    int o = open3(nf[top[t]], G.ilo, G.ihi, G.olo, G.ohi, theta2f);
    if (o == 0) {
        const TNode &Gd = nd[gnode[g]];
        o = cell_open(nd[top[t]], Gd.ilo, Gd.ihi, Gd.olo, Gd.ohi, theta2) ? 1 : -1;
    }
    ostat[p] = o > 0 ? 1 : 0;
}

// Class of each pair and its entry counts: not reached or an open node above
// the split depth (no entries), unopened (one SPJ entry), open leaf (its
// bodies), open node at the split depth (a subtree task, counted later).
// fill == 1 writes the entries of the first three kinds.
__global__ void k_walk_class(const TNode *nd, const int *top, const int *top_anc, const int *top_lvl, long long np,
                             int ntop, int depth, const unsigned char *ostat, const int *order, int fill, int *jc,
                             int *sc, int *task_flag, const int *jo, const int *so, int *j_idx, int *s_idx) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const int g = (int)(p / ntop), t = (int)(p - (long long)g * ntop);
    const unsigned char *os = ostat + (long long)g * ntop;
    bool reached = true;
    for (int a = 0; a < depth; a++) {
        const int ta = top_anc[t * depth + a];
        if (ta >= 0 && !os[ta]) reached = false;
    }
    int nj = 0, ns = 0, task = 0;
    const int c = top[t];
    if (reached) {
        const TNode &C = nd[c];
        if (!os[t]) {
            if (fill) s_idx[so[p]] = c;
            ns = 1;
        } else if (C.nchild == 0) {
            if (fill)
                for (int k = 0; k < C.count; k++) j_idx[jo[p] + k] = order[C.first + k];
            nj = C.count;
        } else if (top_lvl[t] == depth) {
            task = 1;
        }
    }
    if (!fill) {
        jc[p] = nj;
        sc[p] = ns;
        task_flag[p] = task;
    }
}

// the subtree walks of the compacted tasks (pair indices), one per thread;
// the opening test runs on the FP32 copies and falls back to the doubles
// only when the copies cannot decide
__global__ void k_walk_tasks(const TNode *nd, const TNodeF *nf, const int *gnode, const int *top, int ntop,
                             const int *tasks, int ntask, double theta2, float theta2f, const int *order, int fill,
                             int *jc, int *sc, const int *jo, const int *so, int *j_idx, int *s_idx, int *status) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ntask) return;
    const long long p = tasks[q];
    const int g = (int)(p / ntop), t = (int)(p - (long long)g * ntop);
    const int gn = gnode[g];
    float fil[3], fih[3], fol[3], foh[3];
    {
        const TNodeF &G = nf[gn];
        for (int d = 0; d < 3; d++) {
            fil[d] = G.ilo[d];
            fih[d] = G.ihi[d];
            fol[d] = G.olo[d];
            foh[d] = G.ohi[d];
        }
    }
    const TNodeF &C = nf[top[t]];
    int stack[WALK_STACK];
    int sp = 0;
    for (int ch = C.nchild - 1; ch >= 0; ch--) stack[sp++] = C.child0 + ch;
    int nj = 0, ns = 0;
    const int jbase = fill ? jo[p] : 0, sbase = fill ? so[p] : 0;
    for (int guard = 0; sp > 0 && guard < (1 << 26); guard++) {
        const int c = stack[--sp];
        const TNodeF &Q = nf[c];
        int o = open3(Q, fil, fih, fol, foh, theta2f);
        if (o == 0) {
            const TNode &Gd = nd[gn];
            o = cell_open(nd[c], Gd.ilo, Gd.ihi, Gd.olo, Gd.ohi, theta2) ? 1 : -1;
        }
        if (o < 0) {
            if (fill) s_idx[sbase + ns] = c;
            ns++;
        } else if (Q.nchild == 0) {
            if (fill)
                for (int k = 0; k < Q.count; k++) j_idx[jbase + nj + k] = order[Q.first + k];
            nj += Q.count;
        } else {
            if (sp + Q.nchild > WALK_STACK) {
                atomicOr(status, ST_QUEUE_OVERFLOW);
                break;
            }
            for (int ch = Q.nchild - 1; ch >= 0; ch--) stack[sp++] = Q.child0 + ch;
        }
    }
    if (!fill) {
        jc[p] = nj;
        sc[p] = ns;
    }
}

// ---- the walk as one CTA per group, breadth first --------------------------------------------
// The host builder's depth-first walk emits, in visiting order, one SPJ entry
// per unopened cell and the bodies of every opened leaf.  The same sequence
// comes out of a breadth-first sweep that keeps a frontier of items in that
// order: each round replaces every still-untested cell by its outcome -- an
// unopened cell or an opened leaf stays as a final item, an opened inner cell
// gives way to its children in child order -- so that after the last round
// the frontier is the depth-first output sequence.  All the CTA's threads
// test the frontier's cells at once (the subtree walks of one thread each
// ran at ~3 active lanes per instruction).  Items: node << 2 | kind.
constexpr int BFS_T = 128;
constexpr int BFS_CAP = 4096;  // frontier items per group (more: the group takes the task walk)
enum : int { FI_PEND = 0, FI_SPJ = 1, FI_EPJ = 2 };

// exclusive block-wide prefix of v over BFS_T threads (all threads call)
__device__ __forceinline__ int bfs_scan(int v, int *ws, int &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    int off = 0, tot = 0;
#pragma unroll
    for (int k = 0; k < BFS_T / 32; k++) {
        const int c = ws[k];
        off += (k < w) ? c : 0;
        tot += c;
    }
    __syncthreads();
    total = tot;
    return off + x - v;
}

// count pass: the final frontier of group g (blockIdx.x) into store[off[g] ..
// off[g] + len[g]) and its EPJ / SPJ entry counts; a frontier above cap (<= BFS_CAP)
// items or a full store sets *overflow (the lists then come from the task walk)
__global__ void __launch_bounds__(BFS_T) k_walk_bfs(const TNode *nd, const TNodeF *nf, const int *gnode, int ng,
                                                    double theta2, float theta2f, int *jc, int *sc, int *len,
                                                    long long *off, int *store, unsigned long long *cursor,
                                                    long long store_cap, int *overflow, int cap) {
    __shared__ int buf[2][BFS_CAP];
    __shared__ int ws[BFS_T / 32];
    __shared__ long long s_base;
    const int g = blockIdx.x, tid = threadIdx.x;
    if (g >= ng) return;
    const int gn = gnode[g];
    float fil[3], fih[3], fol[3], foh[3];
    {
        const TNodeF &G = nf[gn];
        for (int d = 0; d < 3; d++) {
            fil[d] = G.ilo[d];
            fih[d] = G.ihi[d];
            fol[d] = G.olo[d];
            foh[d] = G.ohi[d];
        }
    }
    if (tid == 0) buf[0][0] = (0 << 2) | FI_PEND;  // the root
    __syncthreads();
    int cur = 0, n = 1;
    bool over = false, pend = true;
    for (int round = 0; pend && round < 64; round++) {
        int run = 0, grown = 0;
        for (int base = 0; base < n; base += BFS_T) {
            const int q = base + tid;
            int item = 0, cnt = 0, kind = FI_SPJ, nch = 0, c0 = 0;
            if (q < n) {
                item = buf[cur][q];
                kind = item & 3;
                cnt = 1;
                if (kind == FI_PEND) {
                    const int c = item >> 2;
                    const TNodeF &Q = nf[c];
                    int o = open3(Q, fil, fih, fol, foh, theta2f);
                    if (o == 0) {
                        const TNode &Gd = nd[gn];
                        o = cell_open(nd[c], Gd.ilo, Gd.ihi, Gd.olo, Gd.ohi, theta2) ? 1 : -1;
                    }
                    if (o < 0) {
                        kind = FI_SPJ;
                    } else if (Q.nchild == 0) {
                        kind = FI_EPJ;
                    } else {
                        nch = Q.nchild;
                        c0 = Q.child0;
                        cnt = nch;
                    }
                    item = (c << 2) | kind;
                }
            }
            int tot = 0;
            const int o = run + bfs_scan(cnt, ws, tot);
            if (q < n && o + cnt <= cap) {
                if (nch) {
                    for (int k = 0; k < nch; k++) buf[cur ^ 1][o + k] = ((c0 + k) << 2) | FI_PEND;
                } else {
                    buf[cur ^ 1][o] = item;
                }
            }
            grown += __syncthreads_or(nch > 0);
            run += tot;
        }
        if (run > cap) {
            over = true;
            break;
        }
        cur ^= 1;
        n = run;
        pend = grown > 0;
        __syncthreads();
    }
    if (pend && !over) over = true;  // deeper than 64 rounds
    if (!over) {
        int nj = 0, ns = 0;
        for (int q = tid; q < n; q += BFS_T) {
            const int it = buf[cur][q];
            if ((it & 3) == FI_EPJ) nj += nf[it >> 2].count;
            else ns += 1;
        }
        int tj = 0, ts = 0;
        bfs_scan(nj, ws, tj);
        bfs_scan(ns, ws, ts);
        if (tid == 0) {
            const long long b = (long long)atomicAdd(cursor, (unsigned long long)n);
            s_base = b;
            if (b + n > store_cap) atomicOr(overflow, 1);
            jc[g] = tj;
            sc[g] = ts;
            len[g] = n;
            off[g] = b;
        }
        __syncthreads();
        const long long b = s_base;
        if (b + n <= store_cap)
            for (int q = tid; q < n; q += BFS_T) store[b + q] = buf[cur][q];
    } else if (tid == 0) {
        atomicOr(overflow, 1);
        jc[g] = 0;
        sc[g] = 0;
        len[g] = 0;
        off[g] = 0;
    }
}

// What the host reads after the walk: lists' sizes, frontier items, whether a
// frontier or the store overflowed, the status bits so far.
struct WalkInfo {
    unsigned long long cursor;
    int n[2], overflow, status;
};
// the groups' list offsets from their counts (scan y = 0: EPJ, 1: SPJ)
struct WalkScan {
    const int *jc, *sc;
    int *j_off, *s_off;
    int ng;
    WalkInfo *info;
    const int *status;
    __device__ int operator()(int y, int g) const { return y ? sc[g] : jc[g]; }
    __device__ void operator()(int y, int g, int prefix, int) const { (y ? s_off : j_off)[g] = prefix; }
    __device__ void total(int y, int t) const {
        (y ? s_off : j_off)[ng] = t;
        info->n[y] = t;
        if (y == 0) info->status = *(const volatile int *)status;
    }
};

// fill pass: group g's entries from its stored frontier, in frontier order
__global__ void __launch_bounds__(BFS_T) k_walk_bfs_fill(const TNodeF *nf, int ng, const int *len, const long long *off,
                                                         const int *store, const int *order, const int *j_off,
                                                         const int *s_off, int *j_idx, int *s_idx) {
    __shared__ int ws[BFS_T / 32];
    const int g = blockIdx.x, tid = threadIdx.x;
    if (g >= ng) return;
    const int n = len[g];
    const int *fr = store + off[g];
    int jrun = j_off[g], srun = s_off[g];
    for (int base = 0; base < n; base += BFS_T) {
        const int q = base + tid;
        int it = 0, nj = 0, ns = 0, first = 0;
        if (q < n) {
            it = fr[q];
            if ((it & 3) == FI_EPJ) {
                const TNodeF &Q = nf[it >> 2];
                nj = Q.count;
                first = Q.first;
            } else {
                ns = 1;
            }
        }
        int tj = 0, ts = 0;
        const int oj = jrun + bfs_scan(nj, ws, tj);
        const int os = srun + bfs_scan(ns, ws, ts);
        for (int k = 0; k < nj; k++) j_idx[oj + k] = order[first + k];
        if (ns) s_idx[os] = it >> 2;
        jrun += tj;
        srun += ts;
    }
}

__global__ void k_task_list(const int *flag, const int *pos, long long np, int *tasks) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < np && flag[p]) tasks[pos[p]] = (int)p;
}

// per-group list offsets from the per-pair offsets
__global__ void k_walk_group_off(const int *jo, const int *so, int ng, int ntop, int nj, int ns, int *j_off,
                                 int *s_off) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g > ng) return;
    j_off[g] = (g < ng) ? jo[(long long)g * ntop] : nj;
    s_off[g] = (g < ng) ? so[(long long)g * ntop] : ns;
}

// Launch order of the soft kernel: groups by the stage they belong to (`stage`, 0
// without one), then by descending weight class (eight classes an octave; the order
// inside a class is arbitrary, and no result depends on it), a counting sort by one
// CTA; start[s]: the first place of stage s.  A full sort of the weights was 40
// launches.
constexpr int GO_T = 1024, GO_CLASSES = 512, GO_PER = GO_STAGES * GO_CLASSES / GO_T;
__global__ void __launch_bounds__(GO_T) k_group_order(int ng, const int *i_off, const int *j_off, const int *s_off,
                                                      const int *stage, int *order, int *start) {
    __shared__ int h[GO_STAGES * GO_CLASSES], ws[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    auto bin = [&](int g) {
        const long long ni = i_off[g + 1] - i_off[g];
        const long long nj = (j_off[g + 1] - j_off[g]) + 2LL * (s_off[g + 1] - s_off[g]);
        const float wt = (float)(((ni + 31) / 32) * 32 * nj + 1);
        const int b = (int)(__float_as_uint(wt) >> 20) - (127 << 3);
        return (stage ? stage[g] : 0) * GO_CLASSES + GO_CLASSES - 1 - min(max(b, 0), GO_CLASSES - 1);
    };
    for (int k = tid; k < GO_STAGES * GO_CLASSES; k += GO_T) h[k] = 0;
    __syncthreads();
    for (int g = tid; g < ng; g += GO_T) atomicAdd(&h[bin(g)], 1);
    __syncthreads();
    int c[GO_PER], sum = 0;
#pragma unroll
    for (int k = 0; k < GO_PER; k++) {
        c[k] = h[GO_PER * tid + k];
        sum += c[k];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    for (int k = 0; k < w; k++) x += ws[k];
    x -= sum;
#pragma unroll
    for (int k = 0; k < GO_PER; k++) {
        h[GO_PER * tid + k] = x;
        x += c[k];
    }
    __syncthreads();
    if (start && tid < GO_STAGES) start[tid] = h[tid * GO_CLASSES];
    __syncthreads();
    for (int g = tid; g < ng; g += GO_T) order[atomicAdd(&h[bin(g)], 1)] = g;
}

cudaError_t launch_group_order(int ng, const int *i_off, const int *j_off, const int *s_off, const int *stage, int *order,
                               int *start, cudaStream_t st) {
    if (ng > 0) { P3T_COUNT_LAUNCH(); k_group_order<<<1, GO_T, 0, st>>>(ng, i_off, j_off, s_off, stage, order, start); }
    return cudaGetLastError();
}

// The stage of a group whose bodies arrive in stages of `per`: the last of its
// bodies' and list entries' (a warp per group; entries out of range are the pair
// kernel's to report).
__global__ void __launch_bounds__(256) k_group_stage(int ng, const int *i_off, const int *i_idx, const int *j_off,
                                                     const int *j_idx, int n, int per, int *stage) {
    const int g = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (g >= ng) return;
    int last = 0;
    for (int k = i_off[g] + lane; k < i_off[g + 1]; k += 32) last = max(last, min(i_idx[k], n - 1));
    for (int k = j_off[g] + lane; k < j_off[g + 1]; k += 32) last = max(last, min(j_idx[k], n - 1));
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0) stage[g] = last / per;
}
cudaError_t launch_group_stage(int ng, const int *i_off, const int *i_idx, const int *j_off, const int *j_idx, int n,
                               int per, int *stage, cudaStream_t st) {
    if (ng > 0) { P3T_COUNT_LAUNCH(); k_group_stage<<<nblocks(32LL * ng), 256, 0, st>>>(ng, i_off, i_idx, j_off, j_idx, n, per, stage); }
    return cudaGetLastError();
}

// ---- host side ----------------------------------------------------------------------------------
struct DTree {
    DevBuf<double> part, root;
    DevBuf<unsigned long long> key, key2;
    DevBuf<unsigned> ghist, done;
    DevBuf<unsigned short> lev;
    DevBuf<int> idx, idx2, lcnt, loff, lstart, nch, list, parent, gmark, gnode, ng;
    DevBuf<TNode> nd;
    DevBuf<TNodeF> nf;
    DevBuf<int> top, pc, tasks;
    DevBuf<unsigned char> ostat;
    DevBuf<int> bjc, bsc, blen, bstore;  // breadth-first walk
    DevBuf<WalkInfo> binfo;
    DevBuf<long long> boff;
    long long bstore_cap = 1LL << 24;
    std::vector<int> level_start;
    int n_nodes = 0, n_groups = 0;
};
static DTree g_dt;
static int g_walk_depth = 3;  // levels above the walk's task split
static int g_walk_bfs = 1;    // walk form: breadth first per group (1) or subtree tasks (0)
static int g_walk_last = -1;  // the form the last build's lists came from
static int g_walk_cap = BFS_CAP;  // frontier items a group's CTA may hold (lower: more groups take the task walk)
static int g_moments_up = 1;  // moments: leaves in one launch, then inner nodes per level (1); all nodes per level (0)


// Builds the tree of the state's bodies and writes the group lists and the
// SPJ array into the resident soft-force set.  *status: the status bits that the
// breadth-first walk's end had seen, -1 when the task walk ran (its own come later).
static int device_tree(Context *c, double theta, int n_leaf_limit, int n_group_limit, int *status) {
    Engine &E = g_eng;
    DTree &T = g_dt;
    DevSet &d = c->res;
    const int n = E.S.n;
    if (n <= 0 || theta <= 0. || n_leaf_limit < 1 || n_group_limit < 1) return ST_BAD_INDEX;
    const int limit = std::min(n_leaf_limit, n_group_limit);
    int r = 0;
    const int pb = std::min(512, nblocks(n)), rt = (n + RADIX_TILE - 1) / RADIX_TILE, lbk = nblocks(n);
    if (!T.done.p) {
        if ((r = T.done.reserve(1))) return r;
        cudaMemsetAsync(T.done.p, 0, T.done.cap, c->stream);
    }
    if ((r = T.part.reserve(6 * (size_t)pb)) || (r = T.root.reserve(8)) || (r = T.key.reserve(n)) ||
        (r = T.key2.reserve(n)) || (r = T.idx.reserve(n)) || (r = T.idx2.reserve(n)) || (r = d.i_idx.reserve(n)) ||
        (r = T.ghist.reserve(8 * 256)) || (r = T.lev.reserve(n)) ||
        (r = T.lcnt.reserve((MAX_LEVEL + 1) * (size_t)lbk)) || (r = T.loff.reserve((MAX_LEVEL + 1) * (size_t)lbk)) ||
        (r = T.lstart.reserve(MAX_LEVEL + 2)) || (r = T.gmark.reserve(n)) || (r = T.ng.reserve(1)))
        return r;
    // 1. root cube, keys, sort (the last pass writes the order into the group lists' bodies)
    if (n <= SMALL_N) {
        // (above 48 KB of shared memory a kernel must be allowed its size)
        if ((r = cuda_status(cudaFuncSetAttribute(k_small_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)sizeof(SmallSmem)))))
            return r;
        { P3T_COUNT_LAUNCH(); k_small_sort<<<1, SMALL_T, sizeof(SmallSmem), c->stream>>>(E.S.pos, n, T.root.p, T.key.p, d.i_idx.p); }
    } else {
        cudaMemsetAsync(T.ghist.p, 0, 8 * 256 * sizeof(unsigned), c->stream);
        { P3T_COUNT_LAUNCH(); k_bbox<<<pb, 256, 0, c->stream>>>(E.S.pos, n, T.part.p, T.done.p, T.root.p); }
        { P3T_COUNT_LAUNCH(); k_keys<<<rt, 256, 0, c->stream>>>(E.S.pos, n, T.root.p, T.key.p, T.idx.p, T.ghist.p); }
        for (int p = 0; p < 8; p++) {
            const bool odd = p & 1;
            if ((r = E.lb.reserve(c, 256 * (size_t)rt))) return r;
            { P3T_COUNT_LAUNCH(); k_radix_pass<<<rt, RADIX_T, 0, c->stream>>>(odd ? T.key2.p : T.key.p, odd ? T.idx2.p : T.idx.p, n, rt, 8 * p,
                                                                         T.ghist.p + 256 * p, E.lb.st.p, E.lb.ticket.p,
                                                                         E.lb.epoch, c->status, odd ? T.key.p : T.key2.p,
                                                                         p == 7 ? d.i_idx.p : (odd ? T.idx.p : T.idx2.p)); }
        }
    }
    const unsigned long long *key = T.key.p;
    const int *idx = d.i_idx.p;
    // 2. nodes of every level
    { P3T_COUNT_LAUNCH(); k_node_levels<<<lbk, 256, 0, c->stream>>>(key, n, limit, T.lev.p, T.lcnt.p); }
    if ((r = launch_scan_lb(c, E.lb, LevelScan{T.lcnt.p, T.loff.p, T.lstart.p, lbk},
                            LevelScan{T.lcnt.p, T.loff.p, T.lstart.p, lbk}, (MAX_LEVEL + 1) * lbk)))
        return r;
    int ls[MAX_LEVEL + 2];
    if ((r = d2h(c, ls, T.lstart.p, sizeof ls))) return r;
    const int base = ls[MAX_LEVEL + 1];
    if (base < 1 || base > (MAX_LEVEL + 1) * (long long)n) return ST_ITER_CAP;
    T.level_start.assign(1, 0);
    for (int L = 1; L <= MAX_LEVEL + 1 && ls[L] > T.level_start.back(); L++) T.level_start.push_back(ls[L]);
    T.n_nodes = base;
    if ((r = T.nd.reserve(base)) || (r = T.parent.reserve(base)) || (r = T.nch.reserve((size_t)base + MAX_LEVEL + 2)) ||
        (r = T.list.reserve(2 * (size_t)base)) || (r = T.nf.reserve(base)) || (r = d.spj.reserve(base)) ||
        (r = T.gnode.reserve(base + 1)) || (r = d.i_off.reserve(base + 1)))
        return r;
    int *icnt = T.nch.p + base;
    cudaMemsetAsync(T.nch.p, 0, ((size_t)base + MAX_LEVEL + 2) * sizeof(int), c->stream);
    cudaMemsetAsync(T.gmark.p, 0, n * sizeof(int), c->stream);
    { P3T_COUNT_LAUNCH(); k_nodes<<<lbk, 256, 0, c->stream>>>(key, n, T.lev.p, T.loff.p, T.lstart.p, T.root.p, base, T.nd.p, T.parent.p,
                                                       T.nch.p, T.list.p, icnt); }
    // 3. groups in Morton order (the host reads their count after the moments' launches)
    { P3T_COUNT_LAUNCH(); k_group_mark<<<nblocks(base), 256, 0, c->stream>>>(base, T.nd.p, T.parent.p, T.nch.p, n_group_limit, T.gmark.p); }
    {
        const GroupScan gs{T.gmark.p, T.gnode.p, d.i_off.p, T.ng.p, n};
        if ((r = launch_scan_lb(c, E.lb, gs, gs, n))) return r;
    }
    // 4. moments: the leaves in one launch, then the inner nodes level by level
    // (or all nodes level by level), deepest first
    const int nlev_all = (int)T.level_start.size() - 1;
    if (g_moments_up) {
        { P3T_COUNT_LAUNCH(); k_moments_list<<<nblocks((long long)base * NL, MOM_T), MOM_T, 0, c->stream>>>(
            T.list.p, icnt + MAX_LEVEL + 1, T.nd.p, T.nf.p, d.spj.p, idx, E.S.pos, E.S.mass, E.S.r_search); }
        for (int L = nlev_all - 2; L >= 0;) {  // the deepest level has leaves only
            int to = L;
            while (to >= 0 && T.level_start[to + 1] - T.level_start[to] <= TOP_NODES) to--;
            const int m = T.level_start[L + 1] - T.level_start[L];
            if (to < L) {  // levels L..to + 1 are small
                { P3T_COUNT_LAUNCH(); k_moments_run<<<1, MOM_T, 0, c->stream>>>(L, to + 1, T.lstart.p, T.list.p + base, icnt, T.nd.p, T.nf.p,
                                                                           d.spj.p, idx, E.S.pos, E.S.mass, E.S.r_search); }
                L = to;
            } else {
                { P3T_COUNT_LAUNCH(); k_moments_list<<<nblocks((long long)m * NL, MOM_T), MOM_T, 0, c->stream>>>(
                    T.list.p + base + T.level_start[L], icnt + L, T.nd.p, T.nf.p, d.spj.p, idx, E.S.pos, E.S.mass,
                    E.S.r_search); }
                L--;
            }
        }
    } else {
        for (int L = nlev_all - 1; L >= 0; L--) {
            const int lo = T.level_start[L], hi = T.level_start[L + 1];
            { P3T_COUNT_LAUNCH(); k_moments<<<nblocks((long long)(hi - lo) * NL, MOM_T), MOM_T, 0, c->stream>>>(lo, hi, T.nd.p, T.nf.p, d.spj.p, idx, E.S.pos,
                                                                                 E.S.mass, E.S.r_search); }
        }
    }
    int ng = 0;
    if ((r = d2h(c, &ng, T.ng.p, sizeof(int)))) return r;
    T.n_groups = ng;
    if ((r = d.j_off.reserve(ng + 1)) || (r = d.s_off.reserve(ng + 1))) return r;
    // 5. walks: breadth first, one CTA per group; if a frontier outgrows its
    // CTA (or the frontier store), the task walk below
    bool walked = false;
    *status = 0;
    if (g_walk_bfs && ng > 0) {
        if ((r = T.bjc.reserve(ng)) || (r = T.bsc.reserve(ng)) || (r = T.blen.reserve(ng)) ||
            (r = T.boff.reserve(ng)) || (r = T.binfo.reserve(1)) || (r = T.bstore.reserve((size_t)T.bstore_cap)))
            return r;
        cudaMemsetAsync(T.binfo.p, 0, sizeof(WalkInfo), c->stream);
        { P3T_COUNT_LAUNCH(); k_walk_bfs<<<ng, BFS_T, 0, c->stream>>>(T.nd.p, T.nf.p, T.gnode.p, ng, theta * theta,
                                                                  (float)(theta * theta), T.bjc.p, T.bsc.p, T.blen.p,
                                                                  T.boff.p, T.bstore.p, &T.binfo.p->cursor, T.bstore_cap,
                                                                  &T.binfo.p->overflow, g_walk_cap); }
        const WalkScan wsn{T.bjc.p, T.bsc.p, d.j_off.p, d.s_off.p, ng, T.binfo.p, c->status};
        if ((r = launch_scan_lb(c, E.lb, wsn, wsn, ng, 2))) return r;
        WalkInfo info;
        if ((r = d2h(c, &info, T.binfo.p, sizeof info))) return r;
        *status = info.status;
        if (!info.overflow) {
            if ((r = d.j_idx.reserve(info.n[0])) || (r = d.s_idx.reserve(info.n[1]))) return r;
            { P3T_COUNT_LAUNCH(); k_walk_bfs_fill<<<ng, BFS_T, 0, c->stream>>>(T.nf.p, ng, T.blen.p, T.boff.p, T.bstore.p,
                                                                           idx, d.j_off.p, d.s_off.p, d.j_idx.p,
                                                                           d.s_idx.p); }
            walked = true;
        } else if ((long long)info.cursor > T.bstore_cap) {
            T.bstore_cap = (long long)(info.cursor + info.cursor / 4);  // room for the next build
        }
    }
    g_walk_last = walked ? 1 : 0;
    // the task walk: the top levels in pre-order (host, from the node table),
    // then (group, top node) pairs: open tests, counts, offsets, entries
    if (!walked) {
        *status = -1;
        const int nlev = (int)T.level_start.size() - 1;
        const int depth = std::min(g_walk_depth, nlev - 1);
        const int ntop_nodes = T.level_start[depth + 1];
        std::vector<TNode> tn(ntop_nodes);
        if ((r = d2h(c, tn.data(), T.nd.p, ntop_nodes * sizeof(TNode)))) return r;
        std::vector<int> top, anc, lvl;
        std::vector<int> path;
        std::vector<int> pos_of(ntop_nodes, -1);
        // pre-order from the root, levels 0..depth
        std::vector<std::pair<int, int>> st{{0, 0}};
        std::vector<int> par_top(ntop_nodes, -1);
        while (!st.empty()) {
            const int nd_id = st.back().first, L = st.back().second;
            st.pop_back();
            pos_of[nd_id] = (int)top.size();
            top.push_back(nd_id);
            lvl.push_back(L);
            if (L < depth)
                for (int ch = tn[nd_id].nchild - 1; ch >= 0; ch--) {
                    par_top[tn[nd_id].child0 + ch] = nd_id;
                    st.push_back({tn[nd_id].child0 + ch, L + 1});
                }
        }
        const int ntop = (int)top.size();
        anc.assign((size_t)ntop * std::max(depth, 1), -1);
        for (int t = 0; t < ntop; t++) {
            int a = par_top[top[t]], k = 0;
            while (a >= 0 && k < depth) {
                anc[(size_t)t * depth + k++] = pos_of[a];
                a = par_top[a];
            }
        }
        const long long np = (long long)ng * ntop;
        if (np > 2000000000LL) return ST_QUEUE_OVERFLOW;
        if ((r = T.top.reserve(3 * (size_t)ntop + (size_t)ntop * std::max(depth, 1))) ||
            (r = T.ostat.reserve(np)) || (r = T.pc.reserve(6 * np + 6)))
            return r;
        int *top_d = T.top.p, *lvl_d = T.top.p + ntop, *anc_d = T.top.p + 2 * ntop;
        if ((r = h2d(c, top_d, top.data(), ntop * sizeof(int))) || (r = h2d(c, lvl_d, lvl.data(), ntop * sizeof(int))) ||
            (r = h2d(c, anc_d, anc.data(), anc.size() * sizeof(int))))
            return r;
        int *jc = T.pc.p, *sc = T.pc.p + np, *jo = T.pc.p + 2 * np, *so = T.pc.p + 3 * np;
        int *tflag = T.pc.p + 4 * np, *tpos = T.pc.p + 5 * np;
        const int wb = (int)std::min<long long>((np + 127) / 128, 1LL << 30);
        const float th2f = (float)(theta * theta);
        { P3T_COUNT_LAUNCH(); k_walk_open<<<wb, 128, 0, c->stream>>>(T.nd.p, T.nf.p, T.gnode.p, ng, top_d, ntop, theta * theta, th2f,
                                               T.ostat.p); }
        { P3T_COUNT_LAUNCH(); k_walk_class<<<wb, 128, 0, c->stream>>>(T.nd.p, top_d, anc_d, lvl_d, np, ntop, depth, T.ostat.p, idx, 0, jc,
                                                sc, tflag, nullptr, nullptr, nullptr, nullptr); }
        int ntask = 0;
        if ((r = g_eng.scan(tflag, tpos, (int)np, &ntask)) || (r = T.tasks.reserve(ntask + 1))) return r;
        { P3T_COUNT_LAUNCH(); k_task_list<<<wb, 128, 0, c->stream>>>(tflag, tpos, np, T.tasks.p); }
        { P3T_COUNT_LAUNCH(); k_walk_tasks<<<nblocks(ntask, 128), 128, 0, c->stream>>>(T.nd.p, T.nf.p, T.gnode.p, top_d, ntop, T.tasks.p,
                                                                 ntask, theta * theta, th2f, idx, 0, jc, sc, nullptr,
                                                                 nullptr, nullptr, nullptr, c->status); }
        int nj = 0, ns = 0;
        if ((r = g_eng.scan(jc, jo, (int)np, &nj)) || (r = g_eng.scan(sc, so, (int)np, &ns))) return r;
        { P3T_COUNT_LAUNCH(); k_walk_group_off<<<nblocks(ng + 1), 256, 0, c->stream>>>(jo, so, ng, ntop, nj, ns, d.j_off.p, d.s_off.p); }
        if ((r = d.j_idx.reserve(nj)) || (r = d.s_idx.reserve(ns))) return r;
        { P3T_COUNT_LAUNCH(); k_walk_class<<<wb, 128, 0, c->stream>>>(T.nd.p, top_d, anc_d, lvl_d, np, ntop, depth, T.ostat.p, idx, 1, jc,
                                                sc, tflag, jo, so, d.j_idx.p, d.s_idx.p); }
        { P3T_COUNT_LAUNCH(); k_walk_tasks<<<nblocks(ntask, 128), 128, 0, c->stream>>>(T.nd.p, T.nf.p, T.gnode.p, top_d, ntop, T.tasks.p,
                                                                 ntask, theta * theta, th2f, idx, 1, jc, sc, jo, so,
                                                                 d.j_idx.p, d.s_idx.p, c->status); }
    }
    // 6. the soft kernel's launch order
    if ((r = d.order.reserve(ng))) return r;
    if ((r = cuda_status(launch_group_order(ng, d.i_off.p, d.j_off.p, d.s_off.p, nullptr, d.order.p, nullptr, c->stream)))) return r;
    d.order_valid = true;
    c->res_groups = ng;
    c->res_spj = base;
    c->res_n = n;
    return cuda_status(cudaGetLastError());
}

}  // namespace p3t

using namespace p3t;

extern "C" {

int p3t_set_walk(int form) {
    if (form < 0 || form > 3) return -(int)cudaErrorInvalidValue;
    g_walk_bfs = form & 1;
    g_moments_up = (form >> 1) ^ 1;
    return 0;
}

int p3t_walk_last(void) { return g_walk_last; }

int p3t_set_walk_limits(int frontier_cap, long long store_items) {
    if (frontier_cap < 1 || frontier_cap > BFS_CAP || store_items < 0) return -(int)cudaErrorInvalidValue;
    g_walk_cap = frontier_cap;
    if (store_items > 0) g_dt.bstore_cap = store_items;
    return 0;
}

// the lists, with no wait at the end where the build has already read clean
// status bits (nothing after the breadth-first walk's count pass sets any)
static int tree_lists(double theta, int n_leaf_limit, int n_group_limit) {
    Context *c = ctx_get(0);
    if (!c || !g_eng.c) return -(int)cudaErrorNoDevice;
    int r = g_eng.pack_soft(), status = -1;
    if (r) return r;
    if ((r = device_tree(c, theta, n_leaf_limit, n_group_limit, &status))) return r;
    return status == 0 ? 0 : read_status(c);
}

int p3t_state_tree(double theta, int n_leaf_limit, int n_group_limit) {
    const int r = tree_lists(theta, n_leaf_limit, n_group_limit);
    return r ? r : read_status(g_eng.c);
}

int p3t_state_tree_soft(double theta, int n_leaf_limit, int n_group_limit) {
    const int r = tree_lists(theta, n_leaf_limit, n_group_limit);
    return r ? r : soft_run_state();
}

int p3t_tree_lists_counts(long long *counts) {
    Context *c = ctx_get(0);
    if (!c) return -(int)cudaErrorNoDevice;
    const int ng = c->res_groups;
    counts[0] = ng;
    counts[1] = c->res_n;
    int nj = 0, ns = 0;
    if (ng > 0) {
        int r = d2h(c, &nj, c->res.j_off.p + ng, sizeof(int));
        if (r || (r = d2h(c, &ns, c->res.s_off.p + ng, sizeof(int)))) return r;
    }
    counts[2] = nj;
    counts[3] = ns;
    counts[4] = c->res_spj;
    return 0;
}

int p3t_tree_lists_get(int *i_off, int *i_idx, int *j_off, int *j_idx, int *s_off, int *s_idx, void *spj) {
    Context *c = ctx_get(0);
    if (!c) return -(int)cudaErrorNoDevice;
    long long k[5];
    int r = p3t_tree_lists_counts(k);
    if (r) return r;
    DevSet &d = c->res;
    const int ng = (int)k[0];
    if ((r = d2h(c, i_off, d.i_off.p, (ng + 1) * sizeof(int))) || (r = d2h(c, j_off, d.j_off.p, (ng + 1) * sizeof(int))) ||
        (r = d2h(c, s_off, d.s_off.p, (ng + 1) * sizeof(int))) || (r = d2h(c, i_idx, d.i_idx.p, k[1] * sizeof(int))) ||
        (r = d2h(c, j_idx, d.j_idx.p, k[2] * sizeof(int))) || (r = d2h(c, s_idx, d.s_idx.p, k[3] * sizeof(int))))
        return r;
    if (spj && (r = d2h(c, spj, d.spj.p, k[4] * sizeof(SPJRec)))) return r;
    return 0;
}

}  // extern "C"
