// Lane-dense form of the hard part: one CTA integrates a "bundle" of many
// clusters at once, all of their state in shared memory.
//
// What bounds it.  An FP64 instruction holds its warp for 64 cycles whatever
// its active lanes, with no overlap inside the warp, and an SM takes one per
// 19 cycles from all its warps.  So (1) the launch's throughput is the number
// of FP64 warp instructions, and (2) the span of a long chain of block steps
// (hundreds of steps of a close pair) is the number of dependent FP64
// instructions of one step, plus whatever the phases wait for in between.
// Hence:
//   - The CTA keeps up to BCAP members of up to bmaxcl(BCAP) clusters and
//     advances every cluster by one block step per iteration, so each phase
//     runs over the union of the bundle's work items, one lane per item:
//     predictor per (member, component), pair terms per live (target, partner)
//     pair, the targets' sun force in warps of its own beside them, sums and
//     corrector per (target, component), the time-step criteria per target.
//   - The members' state of record is shared memory (42 doubles a slot): a
//     block step makes no trip to global memory.  The arrays of struct Hard
//     are written only around a collision, which works on them.
//   - Roots, reciprocals and quotients run on the integer pipe
//     (p3t_exact.cuh), comparisons of positive doubles on their bits, products
//     by powers of two (a block step's length) fused into the following sum
//     where the product is exact; every rounding is that of the plain form.
//   - When a pass has few items, the three components of an item sit in lanes
//     of their own (bundle_terms_split), which shortens the chain; when it has
//     many, one lane takes an item, which is the fewest instructions.
//   - The live pairs are listed once per block step, for its three passes (a
//     margin covers the corrector's displacement, which is checked; a pass
//     that cannot rely on the list makes its own).
// Measured against the form that kept the members in global memory (256 slots,
// 2 CTAs per SM, the library's roots, a list per pass): a block step of a lone
// pair 35 -> 13 us, of a 60-body cluster 49 -> 24 us; the hard launch of a tree
// step 39 -> 24 ms on the 1,048,576-body ring (throughput-bound, 16 M member
// steps), 19 -> 8.9 ms at 50,000 bodies and 28 -> 12 ms on the 2 M-body wide
// disk (both bound by their longest chains).  Rare paths are out of line and work
// loops are not unrolled: what a block step executes has to stay in the
// instruction cache (inlining them cost 15 % of a lone pair's block step).
// Why 128 slots: three such CTAs fill an SM's shared memory (74 KB each), and
// three independent bundles overlap one's waits with the others' FP64 work; a
// bundle of 256 slots fits once per SM.
// Pair terms are added to each target in partner order, the summation order
// of the reference loop (src/gravity_hard.h:203-367), so the sums are
// bit-identical to the one-cluster-per-team form; pairs beyond the cutoff
// contribute exact +-0 terms to accumulators that start at +0.
// Finished clusters leave the bundle and the queue refills it.  Clusters
// larger than a bundle run concurrently in k_hard_wide, alone in a wide bundle
// of BCAP_WIDE slots, or beyond that in k_hard_team, the one-cluster-per-CTA form.
//
// Prefilter margins.  FP32 coordinates are taken relative to the cluster's
// first member, u = fl32(x - ref).  While every stored |x - ref| component
// stays below E (checked at every store; a violation switches the cluster to
// exact FP64 tests for good), a computed FP32 distance exceeds the exact one
// by at most err = 3e-7 E plus 1.6e-7 relative.  A pair whose exact cutoff
// test passes (|dr|^2 r_out_inv^2 <= 1.000001) then has an FP32 value
// <= (1.000001 + err r_out_inv_max)^2 * 1.000001 =: thr_f, and a pair with
// exact R < 1 has FP32 d^2 <= thr_c (r_i + r_j)_32^2 with
// thr_c = (1.000001 + err / (2 min f r_p))^2 * 1.000001 (both rounded up to
// FP32).  Pairs above the thresholds are therefore beyond the cutoff (their
// terms are exact zeros) or have R > 1, so skipping them is exact.  The list
// made from the predicted positions serves the corrected ones too: it holds
// the pairs up to thr_f (1 + 1/64)^2, and every corrected component is
// checked to lie within r_out / 128 of its prediction.
#pragma once

namespace p3t {

constexpr int BPT = 4;          // (target, partner) items a thread tests per round of bundle_build
constexpr int BCAP_MAIN = 256;  // members a cluster may have to stay out of the one-per-CTA form without k_hard_wide
constexpr int BCAP_WIDE = 512;  // member slots of the wide form (one cluster at a time)
// clusters in a bundle at once
__host__ __device__ constexpr int bmaxcl(int cap) { return cap > 256 ? 8 : cap / 2; }
__host__ __device__ constexpr int bundle_threads(int cap) { return cap >= 256 ? 256 : 128; }
// pair terms held at once, entries of the live-pair list
__host__ __device__ constexpr int bundle_terms_cap(int cap) { return 256; }
__host__ __device__ constexpr int bundle_list_cap(int cap) { return cap >= 256 ? 2048 : 1024; }
constexpr int BSURV = 64;    // colliding-pair candidates kept per block step
constexpr int BCLAIM = 8;    // clusters claimed from the queue at a time at most

enum : int { CF_COL = 1, CF_FIN = 2, CF_GONE = 4, CF_EXACT = 8 };  // GONE: goes on in k_hard_wide
enum : unsigned char { MF_ACT = 1, MF_TGT = 2 };
// fields of a member slot (three components from each vector's first); F_N*:
// the running pass's forces of a target, in the order of F_AS..F_JD
enum : int {
    F_POS = 0, F_VEL = 3, F_AS = 6, F_JS = 9, F_AD = 12, F_JD = 15, F_MASS = 18, F_ROI, F_TH, F_DT, F_TE, F_A02,  // F_TE: th + dt, during a step a target's Dt; F_A02: alpha2 acc0 acc0
    F_KEEP = 24,  // the fields above persist between block steps
    F_XP = 24, F_VP = 27, F_NAS = 30, F_NJS = 33, F_NAD = 36, F_NJD = 39, F_N = 42,
    F_PHS = F_XP, F_PHD = F_XP + 1  // potentials of a full pass (the predicted state is dead then)
};

template <int BCAP>
struct BundleSmem {
    static constexpr int S = BCAP;
    static constexpr int NT = bundle_threads(BCAP);
    static constexpr int NCL = bmaxcl(BCAP);
    static constexpr int TC = bundle_terms_cap(BCAP);
    static constexpr int LC = bundle_list_cap(BCAP);
    double d[F_N][S];     // member state by field and slot
    double term[6 * TC];  // pair terms of one drain
    // clusters (bundle index k)
    double c_ts[NCL], c_ref[3][NCL];
    unsigned long long c_key[NCL], c_tm[NCL], c_R[NCL];  // min th + dt, min th, min R of the step
    long long c_pb[NCL], c_work[NCL];
    // colliding-pair candidates
    double sv_R[BSURV];
    long long sv_p[BSURV];
    double q_Kc[8], q_D[8];  // a small pass's 1 - K and dK/dt brackets on their way between warps
    unsigned long long live[2];
    float x32[3][S], roi32[S], fr32[S];  // prefilter copies (x32: of the running pass's positions)
    int hmov[S];                         // high word of r_out / 128
    int gslot[S], pfx[S + 1];
    unsigned list[LC];  // live pairs of the pass: target index << 16 | partner slot, in (target, partner) order
    float c_thrf[NCL], c_thrc[NCL], c_E32[NCL];
    int c_idx[NCL], c_off[NCL], c_n[NCL], c_goff[NCL], c_steps[NCL], c_flags[NCL], c_n0[NCL], c_act[NCL];
    int c_imp[NCL], c_tar[NCL], c_addn[NCL], c_addg[NCL];
    int sv_k[BSURV];
    // claimed, not yet admitted clusters
    int pend_c[BCLAIM], pend_n[BCLAIM];
    int ws[NT / 32];
    int used, ncl, fresh_k, fresh_p, n_sv, n_pend, i_pend, exhausted, any, grew, phase;
    short dn_w[32], dn_b[33];  // bundle_dense: a target's terms of a drain, their places
    int ln, nt, moved, any_dead;  // list entries, targets; a corrected position left the list's margin; dead members
    short tgt[S], cl[S], owner[S], eqc[S], twh[S], twn[S], segb[S], sege[S];
    unsigned char dead[S], merged[S], flag[S];
    long long ph_acc[HP_N], ph_t;  // optional per-phase clock counts (thread 0)
};

// the bundle of this CTA, by its symbol: functions that are not inlined keep
// shared-memory loads (a reference passed to them would make them generic)
template <int BCAP>
__device__ __forceinline__ BundleSmem<BCAP> &bundle_smem() {
    extern __shared__ __align__(16) unsigned char bundle_raw[];
    return *reinterpret_cast<BundleSmem<BCAP> *>(bundle_raw);
}

// the end of a phase of the bundle loop (after its barrier): thread 0 adds
// the clock cycles since the last mark to the phase's count
#define HP_MARK(id)                                            \
    do {                                                       \
        if (A.phase_cycles && threadIdx.x == 0) {              \
            const long long t_ = clock64();                    \
            B.ph_acc[id] += t_ - B.ph_t;                       \
            B.ph_t = t_;                                       \
        }                                                      \
    } while (0)
// member- and cluster-parallel loops over the bundle
#define FOR_SLOTS(p) for (int p = threadIdx.x; p < B.used; p += BT)
#define FOR_CLUSTERS(k) for (int k = threadIdx.x; k < B.ncl; k += BT)

__device__ __forceinline__ unsigned long long dbits(double x) {
    return (unsigned long long)__double_as_longlong(x);
}
__device__ __forceinline__ double bitsd(unsigned long long b) { return __longlong_as_double((long long)b); }
__device__ __forceinline__ int dhi(double x) { return __double2hiint(x); }
// a < b, min for doubles >= +0: by their bits (the FP64 pipe's comparison
// costs an FP64 instruction)
__device__ __forceinline__ bool plt(double a, double b) { return dbits(a) < dbits(b); }
__device__ __forceinline__ double pmin(double a, double b) { return plt(b, a) ? b : a; }
// +0 for a zero of either sign: the sum +0 + x
__device__ __forceinline__ double from_zero(double x) { return (dbits(x) << 1) == 0ULL ? 0. : x; }
// a normal power of two whose products with it are exact
__device__ __forceinline__ bool is_pow2(double x) {
    const unsigned h = (unsigned)dhi(x);
    return __double2loint(x) == 0 && (h & 0x800fffffu) == 0u && h - 0x10000000u < 0x60000000u;
}

// the minimum over the warp, a word after the other
__device__ __forceinline__ unsigned long long warp_min64(unsigned long long v) {
    const unsigned h = __reduce_min_sync(0xffffffffu, (unsigned)(v >> 32));
    const unsigned l = __reduce_min_sync(0xffffffffu, (unsigned)(v >> 32) == h ? (unsigned)v : ~0u);
    return ((unsigned long long)h << 32) | l;
}

template <int BCAP>
__device__ __forceinline__ V3 bld(const BundleSmem<BCAP> &B, int f, int p) {
    return v3(B.d[f][p], B.d[f + 1][p], B.d[f + 2][p]);
}
template <int BCAP>
__device__ __forceinline__ void bst(BundleSmem<BCAP> &B, int f, int p, V3 v) {
    B.d[f][p] = v.x;
    B.d[f + 1][p] = v.y;
    B.d[f + 2][p] = v.z;
}

// exclusive block-wide prefix sum of v over NT threads; all threads must call
template <int NT>
__device__ __forceinline__ int bscan(int v, int *ws, int &total) {
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
    for (int k = 0; k < NT / 32; k++) {
        const int c = ws[k];
        off += (k < w) ? c : 0;
        tot += c;
    }
    __syncthreads();
    total = tot;
    return off + x - v;
}

// FP32 copy of component c of a position relative to the cluster origin, with
// the bound check
template <int BCAP>
__device__ __forceinline__ void st32b(BundleSmem<BCAP> &B, int c, int p, double x, int k) {
    const float u = (float)(x - B.c_ref[c][k]);
    B.x32[c][p] = u;
    if (!(fabsf(u) < B.c_E32[k])) atomicOr(&B.c_flags[k], CF_EXACT);
}
template <int BCAP>
__device__ __forceinline__ float bd2_32(const BundleSmem<BCAP> &B, int s, int t) {
    const float dx = B.x32[0][s] - B.x32[0][t], dy = B.x32[1][s] - B.x32[1][t], dz = B.x32[2][s] - B.x32[2][t];
    return dx * dx + dy * dy + dz * dz;
}

// ---- targets and live pairs -------------------------------------------------
// ordered list of the occupied slots whose flag has `bit`, and the prefix of
// their partner counts (pfx; pfx[count] = total); returns the count
template <int BCAP>
__device__ __forceinline__ int bundle_targets(BundleSmem<BCAP> &B, unsigned char bit) {
    constexpr int BT = BundleSmem<BCAP>::NT, PER = BCAP / BT;
    const int base = threadIdx.x * PER;
    int v = 0;  // partner count << 10 | targets
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int p = base + j;
        if (p < B.used && (B.flag[p] & bit)) v += (B.c_n[B.cl[p]] << 10) | 1;
    }
    int tot;
    int off = bscan<BT>(v, B.ws, tot);
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int p = base + j;
        if (p < B.used && (B.flag[p] & bit)) {
            B.tgt[off & 1023] = (short)p;
            B.pfx[off & 1023] = off >> 10;
            off += (B.c_n[B.cl[p]] << 10) | 1;
        }
    }
    if (threadIdx.x == 0) B.pfx[tot & 1023] = tot >> 10;
    __syncthreads();
    return tot & 1023;
}

// the FP64 test of a pair (rarely run, and kept out of line like the other
// rare paths: what a block step executes should stay in the instruction cache)
template <int BCAP>
__device__ __noinline__ int pair_live_exact(double eps2, int mode, int s, int t) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    const V3 dr = bld(B, mode == 0 ? F_POS : F_XP, t) - bld(B, mode == 1 ? F_XP : F_POS, s);
    double dr2 = dot(dr, dr);
    dr2 += eps2;
    const double r = pmin(B.d[F_ROI][s], B.d[F_ROI][t]);
    return !(dr2 * r * r > (mode == 1 ? 1.033 : 1.000001));
}
// whether target s's pair with t (both of cluster k) is listed
template <int BCAP>
__device__ __forceinline__ int pair_live(const HardArgs &A, const BundleSmem<BCAP> &B, int mode, bool exact, int s,
                                         int t, int k) {
    if (B.eqc[s] == B.eqc[t]) return 0;
    if (!exact && !(B.c_flags[k] & CF_EXACT)) {
        const float rf = fminf(B.roi32[s], B.roi32[t]);
        // (1 + 1/64)^2 and the product's rounding
        return bd2_32(B, s, t) * (rf * rf) <= B.c_thrf[k] * (mode == 0 ? 1.f : 1.033f);
    }
    return pair_live_exact<BCAP>(A.P.eps2, mode, s, t);
}

// Targets and pair list of a bundle of at most 32 slots by warp 0, without
// barriers (seven in the general form; for the chains of clusters that run
// alone).  More than 128 items: the targets only.
template <int BCAP>
__device__ __forceinline__ void bundle_lists_small(const HardArgs &A, BundleSmem<BCAP> &B) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x;
    auto prefix = [&](int v) {  // inclusive
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(ALL, v, o);
            if (lane >= o) v += y;
        }
        return v;
    };
    {
        const bool tg = lane < B.used && (B.flag[lane] & MF_TGT);
        const unsigned m = __ballot_sync(ALL, tg);
        const int cn = tg ? B.c_n[B.cl[lane]] : 0, at = __popc(m & ((1u << lane) - 1u)), nt = __popc(m);
        const int end = prefix(cn), total = __shfl_sync(ALL, end, 31);
        if (tg) {
            B.tgt[at] = (short)lane;
            B.pfx[at] = end - cn;
            B.segb[at] = B.sege[at] = 0;
        }
        if (lane == 0) B.pfx[nt] = total;
        __syncwarp();
        int n = 0;
        if (total <= 4 * 32) {
            const int per = total <= 32 ? 1 : 4, f0 = per * lane, f1 = min(f0 + per, total);
            unsigned lv = 0u;
            int lo = 0;
            if (f0 < total) {
                while (B.pfx[lo + 1] <= f0) lo++;
                int l = lo;
#pragma unroll 1
                for (int f = f0; f < f1; f++) {
                    while (B.pfx[l + 1] <= f) l++;
                    const int s = B.tgt[l], k = B.cl[s];
                    lv |= (unsigned)pair_live(A, B, 1, false, s, B.c_off[k] + (f - B.pfx[l]), k) << (f - f0);
                }
            }
            __syncwarp();
            const int nl = __popc(lv), stop = prefix(nl);
            int off = stop - nl;
            n = __shfl_sync(ALL, stop, 31);
            for (; lv; lv &= lv - 1u) {
                const int f = f0 + __ffs((int)lv) - 1;
                while (B.pfx[lo + 1] <= f) lo++;
                B.list[off++] = ((unsigned)lo << 16) | (unsigned)(B.c_off[B.cl[B.tgt[lo]]] + (f - B.pfx[lo]));
            }
            __syncwarp();
            for (int q = lane; q < n; q += 32) {
                const int ti = B.list[q] >> 16;
                const int tp = q > 0 ? (int)(B.list[q - 1] >> 16) : -1;
                if (ti != tp) {
                    B.segb[ti] = (short)q;
                    if (tp >= 0) B.sege[tp] = (short)q;
                }
                if (q == n - 1) B.sege[ti] = (short)n;
            }
        }
        if (lane == 0) {
            B.ln = n;
            B.nt = nt;
        }
    }
}

// The live pairs from item `base` of the targets' (target, partner) items on,
// until the items end or the list is full: B.list[0..B.ln).  Returns the next
// item.  mode 0: full (pos of both); 1: predicted i and j; 2: corrected i,
// predicted j.  exact: FP64 tests for every cluster.  Ends with the targets' runs
// (segb, sege) being written: the caller's next barrier comes before they are read.
template <int BCAP>
__device__ __forceinline__ int bundle_build(const HardArgs &A, BundleSmem<BCAP> &B, int mode, int nt, int base, bool exact) {
    constexpr int BT = BundleSmem<BCAP>::NT;
    const int tid = threadIdx.x, total = B.pfx[nt];
#pragma unroll 1
    for (int i = tid; i < nt; i += BT) B.segb[i] = B.sege[i] = 0;
    int n = 0;
    while (base < total && n + BPT * BT <= BundleSmem<BCAP>::LC) {
        const int per = (total - base <= BT) ? 1 : BPT;  // few items: one a thread
        const int f0 = base + per * tid, f1 = min(f0 + per, total);
        unsigned lv = 0u;
        int lo = 0;
        if (f0 < total) {
            int hi = nt - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (B.pfx[mid] <= f0) lo = mid;
                else hi = mid - 1;
            }
            int l = lo;
#pragma unroll 1
            for (int f = f0; f < f1; f++) {
                while (B.pfx[l + 1] <= f) l++;
                const int s = B.tgt[l], k = B.cl[s];
                lv |= (unsigned)pair_live(A, B, mode, exact, s, B.c_off[k] + (f - B.pfx[l]), k) << (f - f0);
            }
        }
        int cnt;
        int off = n + bscan<BT>(__popc(lv), B.ws, cnt);
        for (; lv; lv &= lv - 1u) {  // the live ones, in order
            const int f = f0 + __ffs((int)lv) - 1;
            while (B.pfx[lo + 1] <= f) lo++;
            B.list[off++] = ((unsigned)lo << 16) | (unsigned)(B.c_off[B.cl[B.tgt[lo]]] + (f - B.pfx[lo]));
        }
        n += cnt;
        base += per * BT;
    }
    if (tid == 0) B.ln = n;
    __syncthreads();
    // each target's run of the list
#pragma unroll 1
    for (int q = tid; q < n; q += BT) {
        const int ti = B.list[q] >> 16;
        const int tp = q > 0 ? (int)(B.list[q - 1] >> 16) : -1;
        if (ti != tp) {
            B.segb[ti] = (short)q;
            if (tp >= 0) B.sege[tp] = (short)q;
        }
        if (q == n - 1) B.sege[ti] = (short)n;
    }
    return base;
}

// ---- pair terms ---------------------------------------------------------------
// where a pair sits in the cutoff function's range: x = (gamma - y) /
// (gamma - 1) < 0 inside gamma r_out (K = 0), >= 1 beyond r_out (K = 1)
__device__ __forceinline__ bool kx_near(double x) { return dhi(x) < 0 && (dbits(x) << 1) != 0ULL; }
__device__ __forceinline__ bool kx_far(double x) { return dhi(x) >= 0x3ff00000; }

// 1 - K and the bracket 140 x^3 (x-1)^3 r_out_inv / (1 - gamma) of dK/dt for a
// pair that is not near; the operand order of cut_Kx and cut_dKdt
__device__ __forceinline__ void kx_mid(const Params &P, double x, double r_out_inv, double &Kc, double &dKdr) {
    const double x2 = x * x, x_1 = x - 1.;
    const bool near = kx_near(x), far = kx_far(x);
    const double K = (((-20. * x + 70.) * x - 84.) * x + 35.) * x2 * x2;
    const double D = 140. * x * x * x * x_1 * x_1 * x_1 * r_out_inv * P.g_1_inv;
    Kc = near ? 1. : (far ? 0. : 1. - K);
    dKdr = (near || far) ? 0. : D;
}

// the seven terms (acc_d xyz, jerk_d xyz, phi_d) of target s from partner t:
// the arithmetic of hard_force for one pair.  Near pairs (K = 0, 1 - K = 1,
// dK/dt = 0) need 37 FP64 operations, the others 63.
template <int BCAP>
__device__ __forceinline__ void pair_terms(const HardArgs &A, const BundleSmem<BCAP> &B, int fi, int fj, bool phi,
                                           int s, int t, bool mine, double *o, int st) {
    const Params &P = A.P;
    const V3 dr = bld(B, fj, t) - bld(B, fi, s);
    double dr2 = dot(dr, dr);
    if (!(A.plain & PL_EPS2)) dr2 += P.eps2;
    const double r_out_inv = pmin(B.d[F_ROI][s], B.d[F_ROI][t]);
    const V3 dv = bld(B, fj + 3, t) - bld(B, fi + 3, s);
    const double rij = sqrt_rn(dr2);
    const double rinv = rcp_rn(rij);
    const double r2inv = rinv * rinv;
    const double mj = B.d[F_MASS][t];
    const double mr3 = mj * (r2inv * rinv);
    const double alpha = dot(dr, dv) * r2inv;
    if (phi && mine) {
        const double Wc = 1. - cut_W(P, rij, r_out_inv);
        o[6 * st] = mj * rinv * Wc;
    }
    const double x = (P.gamma - rij * r_out_inv) * P.g_1_inv;
    double b = 3. * alpha, mk = mr3;
    V3 kv = dv;
    if (!__all_sync(0xffffffffu, kx_near(x))) {
        double Kc, dKdr;
        kx_mid(P, x, r_out_inv, Kc, dKdr);
        b = 3. * (alpha * Kc) + alpha * rij * dKdr;
        kv = Kc * dv;
        mk = mr3 * Kc;
    }
    if (!mine) return;
    o[0] = mk * dr.x; o[st] = mk * dr.y; o[2 * st] = mk * dr.z;
    o[3 * st] = mr3 * (kv.x - b * dr.x);
    o[4 * st] = mr3 * (kv.y - b * dr.y);
    o[5 * st] = mr3 * (kv.z - b * dr.z);
}

// sun_force (p3t_phys.cuh) of target s into its running forces
template <int BCAP>
__device__ __forceinline__ void sun_terms(const HardArgs &A, BundleSmem<BCAP> &B, int fi, bool phi, int s) {
    const Params &P = A.P;
    const V3 x = bld(B, fi, s), v = bld(B, fi + 3, s);
    double r2 = dot(x, x);
    if (!(A.plain & PL_EPS2_SUN)) r2 += P.eps2_sun;
    const double r2inv = rcp_rn(r2);
    const double rinv = sqrt_rn(r2inv);
    double mr3 = rinv * r2inv;
    if (!(A.plain & PL_M_SUN)) mr3 = P.m_sun * mr3;
    const double alpha = dot(x, v) * r2inv;
    if (phi) B.d[F_PHS][s] = -P.m_sun * rinv;
    const V3 dr = v3(-x.x, -x.y, -x.z), dv = v3(-v.x, -v.y, -v.z);
    bst(B, F_NAS, s, mr3 * dr);
    bst(B, F_NJS, s, mr3 * (dv - 3. * alpha * dr));
}

// terms of list[q0..q1) and, with sun, the targets' sun force: one lane an item
template <int BCAP>
__device__ __forceinline__ void bundle_terms(const HardArgs &A, BundleSmem<BCAP> &B, int fi, int fj, bool phi, int q0,
                                             int np, int ns, int st) {
    constexpr int BT = BundleSmem<BCAP>::NT;
    const int np32 = (np + 31) & ~31;  // pairs and sun forces in different warps
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int w0 = threadIdx.x - lane; w0 < np32 + ns; w0 += BT) {  // whole warps
        const int it = w0 + lane;
        if (w0 < np32) {
            const unsigned e = B.list[q0 + min(it, np - 1)];
            pair_terms(A, B, fi, fj, phi, B.tgt[e >> 16], e & 0xffffu, it < np, B.term + it, st);
        } else if (it < np32 + ns) {
            sun_terms(A, B, fi, phi, B.tgt[it - np32]);
        }
    }
}

// The same with the components of an item in three lanes of four (at most
// NT / 4 items): each lane computes its component's differences and products,
// the sums of three are gathered by shuffles in the order of dot().
template <int BCAP>
__device__ __forceinline__ void bundle_terms_split(const HardArgs &A, BundleSmem<BCAP> &B, int fi, int fj, int q0,
                                                   int np, int ns, int st) {
    const Params &P = A.P;
    const int np8 = (np + 7) & ~7;
    const int it = threadIdx.x >> 2, c = min((int)(threadIdx.x & 3), 2);
    const int w8 = it & ~7;  // the warp's first item
    if (w8 >= np8 + ns) return;
    constexpr unsigned ALL = 0xffffffffu;
    const bool sun = w8 >= np8;
    const bool mine = (threadIdx.x & 3) < 3 && (sun ? it < np8 + ns : it < np);
    auto dot3 = [&](double p) {
        const double a = __shfl_sync(ALL, p, 0, 4), b = __shfl_sync(ALL, p, 1, 4), d = __shfl_sync(ALL, p, 2, 4);
        return a + b + d;
    };
    if (!sun) {
        const unsigned e = B.list[q0 + min(it, np - 1)];
        const int s = B.tgt[e >> 16], t = e & 0xffffu;
        const double dr = B.d[fj + c][t] - B.d[fi + c][s];
        double dr2 = dot3(dr * dr);
        if (!(A.plain & PL_EPS2)) dr2 += P.eps2;
        const double r_out_inv = pmin(B.d[F_ROI][s], B.d[F_ROI][t]);
        const double dv = B.d[fj + 3 + c][t] - B.d[fi + 3 + c][s];
        const double rv = dot3(dr * dv);
        const double rij = sqrt_rn(dr2);
        const double rinv = rcp_rn(rij);
        const double r2inv = rinv * rinv;
        const double mr3 = B.d[F_MASS][t] * (r2inv * rinv);
        const double alpha = rv * r2inv;
        const double x = (P.gamma - rij * r_out_inv) * P.g_1_inv;
        double b = 3. * alpha, kv = dv, mk = mr3;
        if (!__all_sync(ALL, kx_near(x))) {
            double Kc, dKdr;
            kx_mid(P, x, r_out_inv, Kc, dKdr);
            b = 3. * (alpha * Kc) + alpha * rij * dKdr;
            kv = Kc * dv;
            mk = mr3 * Kc;
        }
        const double a = mk * dr, j = mr3 * (kv - b * dr);
        if (mine) {
            B.term[c * st + it] = a;
            B.term[(3 + c) * st + it] = j;
        }
    } else {
        const int s = B.tgt[min(it - np8, ns - 1)];
        const double x = B.d[fi + c][s], v = B.d[fi + 3 + c][s];
        double r2 = dot3(x * x);
        const double xv = dot3(x * v);
        if (!(A.plain & PL_EPS2_SUN)) r2 += P.eps2_sun;
        const double r2inv = rcp_rn(r2);
        const double rinv = sqrt_rn(r2inv);
        double mr3 = rinv * r2inv;
        if (!(A.plain & PL_M_SUN)) mr3 = P.m_sun * mr3;
        const double alpha = xv * r2inv;
        const double a = mr3 * -x, j = mr3 * (-v - 3. * alpha * -x);
        if (mine) {
            B.d[F_NAS + c][s] = a;
            B.d[F_NJS + c][s] = j;
        }
    }
}

// A pass of at most 8 pairs and 8 targets, the longest chains' block steps: its
// time is the dependent FP64 operations of one pair, so the independent parts
// of a pair go to different warps -- 1 - K to warp 0, the bracket of dK/dt to
// warp 1, dv, the powers of 1/r and the result to warp 2, the sun force to
// warp 3 -- each with a component per lane (four lanes a pair); the fourth lane
// takes the scalars of the last products.  26 instead of 46 dependent FP64
// instructions.  Contains a barrier: every thread of the CTA calls it.
template <int BCAP>
__device__ __forceinline__ void bundle_terms_small(const HardArgs &A, BundleSmem<BCAP> &B, int fi, int fj, int q0,
                                                   int np, int ns, int st) {
    const Params &P = A.P;
    constexpr unsigned ALL = 0xffffffffu;
    const int w = threadIdx.x >> 5, it = (threadIdx.x & 31) >> 2, c4 = threadIdx.x & 3, c = min(c4, 2);
    auto dot3 = [&](double p) {
        const double a = __shfl_sync(ALL, p, 0, 4), b = __shfl_sync(ALL, p, 1, 4), d = __shfl_sync(ALL, p, 2, 4);
        return a + b + d;
    };
    double dr = 0., dv = 0., mr3 = 0., alpha = 0., t1 = 0.;
    if (w < 3 && np > 0) {
        const unsigned e = B.list[q0 + min(it, np - 1)];
        const int s = B.tgt[e >> 16], t = e & 0xffffu;
        dr = B.d[fj + c][t] - B.d[fi + c][s];
        double dr2 = dot3(dr * dr);
        if (!(A.plain & PL_EPS2)) dr2 += P.eps2;
        const double rij = sqrt_rn(dr2);
        if (w < 2) {
            const double r_out_inv = pmin(B.d[F_ROI][s], B.d[F_ROI][t]);
            const double x = (P.gamma - rij * r_out_inv) * P.g_1_inv;
            const bool near = kx_near(x), far = kx_far(x);
            double v = w == 0 ? 1. : 0.;  // near: 1 - K = 1, dK/dr = 0
            if (!__all_sync(ALL, near)) {
                if (w == 0) {
                    const double x2 = x * x;
                    const double K = (((-20. * x + 70.) * x - 84.) * x + 35.) * x2 * x2;
                    v = near ? 1. : (far ? 0. : 1. - K);
                } else {
                    const double x_1 = x - 1.;
                    const double D = 140. * x * x * x * x_1 * x_1 * x_1 * r_out_inv * P.g_1_inv;
                    v = (near || far) ? 0. : D;
                }
            }
            if (c4 == 0) (w == 0 ? B.q_Kc : B.q_D)[it] = v;
        } else {
            dv = B.d[fj + 3 + c][t] - B.d[fi + 3 + c][s];
            const double rv = dot3(dr * dv);
            const double rinv = rcp_rn(rij);
            const double r2inv = rinv * rinv;
            mr3 = B.d[F_MASS][t] * (r2inv * rinv);
            alpha = rv * r2inv;
            t1 = alpha * rij;
        }
    } else if (w == 3 && ns > 0) {
        const int s = B.tgt[min(it, ns - 1)];
        const double x = B.d[fi + c][s], v = B.d[fi + 3 + c][s];
        double r2 = dot3(x * x);
        const double xv = dot3(x * v);
        if (!(A.plain & PL_EPS2_SUN)) r2 += P.eps2_sun;
        const double r2inv = rcp_rn(r2);
        const double rinv = sqrt_rn(r2inv);
        double m3 = rinv * r2inv;
        if (!(A.plain & PL_M_SUN)) m3 = P.m_sun * m3;
        const double al = xv * r2inv;
        const double a = m3 * -x, j = m3 * (-v - 3. * al * -x);
        if (it < ns && c4 < 3) {
            B.d[F_NAS + c][s] = a;
            B.d[F_NJS + c][s] = j;
        }
    }
    __syncthreads();
    if (w == 2 && np > 0) {
        const double Kc = B.q_Kc[it], D = B.q_D[it];
        const bool sc = c4 == 3;  // the lane of the scalars
        // lanes 0-2: 1 - K times dv, times m/r^3, times dr; lane 3: dK/dt, 1 - K times alpha, times 3
        const double p1 = (sc ? t1 : Kc) * (sc ? D : dv);
        const double p2 = (sc ? alpha : mr3) * Kc;
        const double p3 = p2 * (sc ? 3. : dr);
        const double b = __shfl_sync(ALL, p3 + p1, 3, 4);
        const double j = mr3 * (p1 - b * dr);
        if (it < np && !sc) {
            B.term[c * st + it] = p3;
            B.term[(3 + c) * st + it] = j;
        }
    }
}

// ---- sums and corrector ---------------------------------------------------------
// 1 / Dt: recip_pow2_or_div (p3t_phys.cuh) with the division out of line
__device__ __forceinline__ double recip_dt(double x) {
    return is_pow2(x) ? bitsd(0x7FE0000000000000ULL - dbits(x)) : ex_outside(1., x, 1);
}

// component c of FPHard::correct (src/particle.h:1208-1274) for target slot s:
// correct()'s roundings with 2 J0, -2 Am and, for a power-of-two Dt, the
// products by Dt fused where they are exact.  last: also a2 and a3, over the
// step's starting acc and jerk (which nothing reads after it).
template <int BCAP>
__device__ __forceinline__ void correct_comp(BundleSmem<BCAP> &B, int s, int c, double as, double js, double ad,
                                             double jd, bool last) {
    const double Dt = B.d[F_TE][s];
    const double J0_s = Dt * B.d[F_JS + c][s], J1_s = Dt * js, Am_s = as - B.d[F_AS + c][s];
    const double A2_s = 3. * Am_s - fma(2., J0_s, J1_s);
    const double A3_s = fma(-2., Am_s, J1_s + J0_s);
    const double J0_d = B.d[F_JD + c][s] * Dt, J1_d = jd * Dt, Am_d = ad - B.d[F_AD + c][s];
    const double A2_d = 3. * Am_d - fma(2., J0_d, J1_d);
    const double A3_d = fma(-2., Am_d, J1_d + J0_d);
    const double A2 = A2_s + A2_d, A3 = A3_s + A3_d;
    const double dx = 1.6666666666666667e-2 * (Dt * Dt) * (5. * A2 + 3. * 1.1666666666666667e-3 * A3);
    const double dv = 8.3333333333333333e-2 * Dt * fma(4., A2, 3. * A3);
    B.d[F_POS + c][s] = B.d[F_XP + c][s] + dx;
    B.d[F_VEL + c][s] = B.d[F_VP + c][s] + dv;
    if ((dhi(dx) & 0x7fffffff) >= B.hmov[s]) B.moved = 1;
    if (last) {
        const double Di = recip_dt(Dt), Di2 = Di * Di, Di3 = Di2 * Di;
        const double t2 = 2. * Di2, t3 = 6. * Di3;
        B.d[F_AS + c][s] = t2 * (A2_s + 3. * A3_s);
        B.d[F_JS + c][s] = t3 * A3_s;
        B.d[F_AD + c][s] = (2. * (A2_d + 3. * A3_d)) * Di2;
        B.d[F_JD + c][s] = (6. * A3_d) * Di3;
    }
}

// a power of two to the n-th, and c times 2^e, by the exponent (no range checks)
__device__ __forceinline__ int pow2_exp(double x) { return ((dhi(x) >> 20) & 0x7ff) - 1023; }
__device__ __forceinline__ double scale2(double c, int e) {
    return __hiloint2double(dhi(c) + (e << 20), __double2loint(c));
}

// 2 x, by the exponent where x is normal and stays so
__device__ __forceinline__ double twice(double x) {
    const unsigned e = ((unsigned)dhi(x) >> 20) & 0x7ffu;
    return e - 1u < 2045u ? __hiloint2double(dhi(x) + (1 << 20), __double2loint(x)) : x + x;
}

// The sums and the correction of at most NT / 6 targets with the sun's and the
// planets' halves of a component in a pair of lanes (their operations are the
// same up to the operands), then position and velocity: 13 and 17 dependent
// FP64 instructions where one lane a component takes 30 and 42.  The roundings
// are correct_comp's.
template <int BCAP>
__device__ __forceinline__ void sum_correct_split(BundleSmem<BCAP> &B, int nt, int q0, int np, int st, bool last) {
    constexpr unsigned ALL = 0xffffffffu;
    const int it = min((int)threadIdx.x, 6 * nt - 1);
    if ((int)(threadIdx.x & ~31u) >= 6 * nt) return;  // no target in this warp
    const bool mine = threadIdx.x < 6 * nt;
    const int h = it & 1, t = (it >> 1) / 3, c = (it >> 1) - 3 * t, s = B.tgt[t];
    double acc, jerk;
    if (h == 0) {
        acc = B.d[F_NAS + c][s];
        jerk = B.d[F_NJS + c][s];
    } else {
        acc = jerk = 0.;
        int q = B.segb[t] - q0;
        const int qe = B.sege[t] - q0;
        if (q < qe) {
            acc = from_zero(B.term[c * st + q]);
            jerk = from_zero(B.term[(3 + c) * st + q]);
#pragma unroll 1
            for (q++; q < qe; q++) {
                acc += B.term[c * st + q];
                jerk += B.term[(3 + c) * st + q];
            }
        }
        if (mine) {
            B.d[F_NAD + c][s] = acc;
            B.d[F_NJD + c][s] = jerk;
        }
    }
    const int f0 = (h ? F_AD : F_AS) + c, f1 = (h ? F_JD : F_JS) + c;
    const double Dt = B.d[F_TE][s], j0 = B.d[f1][s], Am = acc - B.d[f0][s];
    const int ex = pow2_exp(Dt);
    const bool p2 = is_pow2(Dt) && ex > -256 && ex < 256;  // (the scaled factors stay normal)
    double A2, A3;
    if (__all_sync(ALL, p2)) {
        // products by Dt are exact and commute with the rounding of a sum
        A2 = fma(-Dt, fma(2., j0, jerk), 3. * Am);
        A3 = fma(Dt, jerk + j0, -twice(Am));
    } else {
        const double J0 = Dt * j0, J1 = Dt * jerk;
        A2 = 3. * Am - fma(2., J0, J1);
        A3 = fma(-2., Am, J1 + J0);
    }
    const double A2t = A2 + __shfl_xor_sync(ALL, A2, 1), A3t = A3 + __shfl_xor_sync(ALL, A3, 1);
    // even lane: the position, odd lane: the velocity
    const double sum = (h ? 4. : 5.) * A2t + (h ? 3. : 3. * 1.1666666666666667e-3) * A3t;
    double cf;
    if (p2) cf = scale2(h ? 8.3333333333333333e-2 : 1.6666666666666667e-2, h ? ex : 2 * ex);
    else cf = h ? 8.3333333333333333e-2 * Dt : 1.6666666666666667e-2 * (Dt * Dt);
    const double d = cf * sum;
    const double r = B.d[(h ? F_VP : F_XP) + c][s] + d;
    if (!mine) return;
    B.d[(h ? F_VEL : F_POS) + c][s] = r;
    if (!h && (dhi(d) & 0x7fffffff) >= B.hmov[s]) B.moved = 1;
    if (last) {
        const double S = A2 + 3. * A3;
        double a2, a3;
        if (p2) {
            a2 = scale2(2., -2 * ex) * S;
            a3 = scale2(6., -3 * ex) * A3;
        } else {
            const double Di = recip_dt(Dt), Di2 = Di * Di, Di3 = Di2 * Di;
            a2 = h ? (2. * S) * Di2 : (2. * Di2) * S;
            a3 = h ? (6. * A3) * Di3 : (6. * Di3) * A3;
        }
        B.d[f0][s] = a2;
        B.d[f1][s] = a3;
    }
}

// mergeAccJerk (src/hermite.h:36-83) of merged target s: twins in insertion order
template <int BCAP>
__device__ __noinline__ void bundle_merge(int s) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    V3 a = B.d[F_MASS][s] * bld(B, F_NAD, s), j = B.d[F_MASS][s] * bld(B, F_NJD, s);
    double m = B.d[F_MASS][s];
    for (int k = B.twh[s], g = 0; k >= 0 && g < BCAP; k = B.twn[k], g++) {
        addto(a, B.d[F_MASS][k] * bld(B, F_NAD, k));
        addto(j, B.d[F_MASS][k] * bld(B, F_NJD, k));
        m += B.d[F_MASS][k];
    }
    const double mi = 1. / m;
    a = a * mi;
    j = j * mi;
    bst(B, F_NAD, s, a);
    bst(B, F_NJD, s, j);
    for (int k = B.twh[s], g = 0; k >= 0 && g < BCAP; k = B.twn[k], g++) {
        bst(B, F_NAD, k, a);
        bst(B, F_NJD, k, j);
    }
}

// The pass's listed pairs where few targets have long runs of them (a cluster of a
// hundred members or more, all close): terms and in-order sums into the targets'
// running forces.  A target's sum is a chain of one FP64 addition per pair and
// component, 64 cycles each, so a drain that holds one target's pairs leaves all but six
// lanes waiting; here the list is drained in D parts that each hold a D-th of every
// target's run, and the chains run side by side.  Lone clusters whose pairs are all live,
// us per block step: 300 members 1665 -> 949, 500 members 5156 -> 2560, 100 members (in
// 128 threads) 274 -> 248.  Shorter runs lose more to the extra barriers than the chains
// gain (64 members, runs of 17: 33.1 -> 35.7), and more targets leave too little of a run
// to a drain.
constexpr int DENSE_M = 32, DENSE_RUN = 20;  // targets of such a list at most, pairs a target at least
template <int BCAP>
__device__ __forceinline__ bool dense_list(const BundleSmem<BCAP> &B, int n) {
    const int m = (int)(B.list[n - 1] >> 16) - (int)(B.list[0] >> 16) + 1;
    return m <= DENSE_M && n >= DENSE_RUN * m;
}
template <int BCAP>
__device__ __noinline__ void bundle_dense(const HardArgs &A, int fi, int fj, bool phi, int nt, bool first) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT, TC = BundleSmem<BCAP>::TC, PER = TC / BT;
    constexpr unsigned ALL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31;
    const int st = phi ? (6 * TC) / 7 : TC, nc = phi ? 7 : 6;  // components: acc, jerk, phi
    const int n = B.ln, t0 = B.list[0] >> 16, m = (int)(B.list[n - 1] >> 16) - t0 + 1;
    const int D = (n + st - m - 1) / (st - m);  // the sum of the runs' D-ths, rounded up, is at most st
    if (first) {
#pragma unroll 1
        for (int i = tid; i < nc * nt; i += BT) {
            const int c = i / nt;
            B.d[c < 6 ? F_NAD + c : F_PHD][B.tgt[i - c * nt]] = 0.;
        }
        bundle_terms(A, B, fi, fj, phi, 0, 0, nt, st);  // the sun's
    }
    __syncthreads();  // (segb and sege)
    // target t0 + t: its run's D-th, and where that starts among the terms
    if (tid < 32) {
        const int w = lane < m ? (B.sege[t0 + lane] - B.segb[t0 + lane] + D - 1) / D : 0;
        int x = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(ALL, x, o);
            if (lane >= o) x += y;
        }
        B.dn_w[lane] = (short)w;
        B.dn_b[lane] = (short)(x - w);
        if (lane == 31) B.dn_b[32] = (short)x;
    }
    __syncthreads();
    const int total = B.dn_b[32];
    // this thread's places among the terms: next list entry, end of its run, step
    int q[PER], qe[PER], dq[PER];
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int it = tid + u * BT;
        int t = 0;
        for (int h = 16; h > 0; h >>= 1)
            if (t + h < m && B.dn_b[t + h] <= it) t += h;
        dq[u] = B.dn_w[t];
        q[u] = B.segb[t0 + t] + it - B.dn_b[t];
        qe[u] = it < total ? B.sege[t0 + t] : 0;
    }
#pragma unroll 1
    for (int d = 0; d < D; d++) {
#pragma unroll 1
        for (int u = 0; u < PER; u++) {
            const int qu = u == 0 ? q[0] : q[PER - 1], qeu = u == 0 ? qe[0] : qe[PER - 1], du = u == 0 ? dq[0] : dq[PER - 1];
            const int at = qu + d * du;
            const bool mine = at < qeu;
            if (!__any_sync(ALL, mine)) continue;
            const unsigned e = B.list[mine ? at : 0];
            pair_terms(A, B, fi, fj, phi, B.tgt[e >> 16], e & 0xffffu, mine, B.term + tid + u * BT, st);
        }
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < nc * m; i += BT) {
            const int c = i / m, t = i - c * m, w = B.dn_w[t];
            const int k = min(w, B.sege[t0 + t] - B.segb[t0 + t] - d * w);
            double *const sum = &B.d[c < 6 ? F_NAD + c : F_PHD][B.tgt[t0 + t]];
            const double *const p = B.term + c * st + B.dn_b[t];
            double a = *sum;
            if (c < 6) {
#pragma unroll 4
                for (int u = 0; u < k; u++) a += p[u];
            } else {
                for (int u = 0; u < k; u++) a -= p[u];
            }
            *sum = a;
        }
        __syncthreads();
    }
}

// One force pass over the nt targets: list, terms, in-order sums into the
// targets' running forces, mergeAccJerk for merged targets (in a full pass
// those with twins).  corr 1, 2: then the first or second correction.  phi: the
// potentials too (a full pass at a cluster's end).  Ends with a barrier.
template <int BCAP, bool FULL>
__device__ __forceinline__ void bundle_pass(const HardArgs &A, BundleSmem<BCAP> &B, int mode, int nt, bool want_phi,
                                            int corr, bool &listed) {
    constexpr int BT = BundleSmem<BCAP>::NT, TC = BundleSmem<BCAP>::TC;
    // items a pass takes with a component a lane: all four lanes' worth of 128 threads; of
    // 256 less (8 members, 56 pairs and 8 targets, 17.0 -> 16.2 us per block step)
    constexpr int SPLIT = BT == 128 ? 32 : 48;
    const int tid = threadIdx.x;
    const bool phi = FULL && want_phi;
    const int fi = mode == 1 ? F_XP : F_POS, fj = FULL ? F_POS : F_XP;
    const int st = phi ? (6 * TC) / 7 : TC;  // terms held at once
    const bool merge = B.any_dead != 0;
    const bool exact = mode == 2 && B.moved != 0;
    if (exact) listed = false;
    int base = 0;
    bool first = true, more = true;
    while (more) {
        if (!listed) {
            base = bundle_build(A, B, mode, nt, base, exact);
            more = base < B.pfx[nt];
            listed = first && !more && !exact;
        } else {
            more = false;
        }
        const int n = B.ln;
        if (tid == 0) B.live[mode == 0 ? 1 : 0] += n;
        int q0 = 0;
        do {
            int np = min(n - q0, st);
            const int ns = first ? nt : 0;
            if (!FULL && np <= 8 && ns <= 8) bundle_terms_small(A, B, fi, fj, q0, np, ns, st);
            else if (!phi && ((np + 7) & ~7) + ns <= SPLIT) bundle_terms_split(A, B, fi, fj, q0, np, ns, st);
            else if (q0 == 0 && n > st && dense_list(B, n)) {  // terms and sums of the whole list
                bundle_dense<BCAP>(A, fi, fj, phi, nt, first);
                first = false;
                q0 = n;
                np = 0;
            } else bundle_terms(A, B, fi, fj, phi, q0, np, ns, st);
            __syncthreads();
            HP_MARK(HP_PAIRS);
            const bool end = q0 + np >= n && !more;
            const bool fuse = corr && end && !merge;
            if (!FULL && fuse && first && 6 * nt <= BT) sum_correct_split(B, nt, q0, np, st, corr == 2);
            else
#pragma unroll 1
                for (int it = tid; it < 3 * nt; it += BT) {
                const int t = it / 3, c = it - 3 * t, s = B.tgt[t];
                double ad = first ? 0. : B.d[F_NAD + c][s], jd = first ? 0. : B.d[F_NJD + c][s];
                int k = max((int)B.segb[t], q0) - q0;
                const int ke = min((int)B.sege[t], q0 + np) - q0;
                if (first && k < ke) {
                    ad = from_zero(B.term[c * st + k]);
                    jd = from_zero(B.term[(3 + c) * st + k]);
                    k++;
                }
#pragma unroll 1
                for (; k < ke; k++) {
                    ad += B.term[c * st + k];
                    jd += B.term[(3 + c) * st + k];
                }
                B.d[F_NAD + c][s] = ad;
                B.d[F_NJD + c][s] = jd;
                if (fuse) correct_comp(B, s, c, B.d[F_NAS + c][s], B.d[F_NJS + c][s], ad, jd, corr == 2);
            }
            if (phi)
#pragma unroll 1
                for (int t = tid; t < nt; t += BT) {
                    const int s = B.tgt[t];
                    double ph = first ? 0. : B.d[F_PHD][s];
                    const int ke = min((int)B.sege[t], q0 + np) - q0;
                    for (int k = max((int)B.segb[t], q0) - q0; k < ke; k++) ph -= B.term[6 * st + k];
                    B.d[F_PHD][s] = ph;
                }
            __syncthreads();
            first = false;
            q0 += np;
        } while (q0 < n);
    }
    if (merge) {
#pragma unroll 1
        for (int t = tid; t < nt; t += BT) {
            const int s = B.tgt[t];
            if (mode == 0 ? (B.merged[s] && B.twh[s] >= 0) : (!B.dead[s] && B.merged[s])) bundle_merge<BCAP>(s);
        }
        __syncthreads();
        if (corr) {
#pragma unroll 1
            for (int it = tid; it < 3 * nt; it += BT) {
                const int t = it / 3, c = it - 3 * t, s = B.tgt[t];
                correct_comp(B, s, c, B.d[F_NAS + c][s], B.d[F_NJS + c][s], B.d[F_NAD + c][s], B.d[F_NJD + c][s],
                             corr == 2);
            }
            __syncthreads();
        }
    }
    HP_MARK(HP_CORRECT);
}

// a full pass over the flagged slots' targets: FP32 copies of their clusters'
// positions, then the pass
template <int BCAP>
__device__ __noinline__ int bundle_full(const HardArgs &A, bool phi) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT;
#pragma unroll 1
    FOR_SLOTS(p) {
        if (!(B.flag[p] & MF_TGT)) continue;
        const int k = B.cl[p];
#pragma unroll 1
        for (int c = 0; c < 3; c++) st32b(B, c, p, B.d[F_POS + c][p], k);
    }
    const int nt = bundle_targets(B, MF_TGT);
    bool listed = false;
    bundle_pass<BCAP, true>(A, B, 0, nt, phi, 0, listed);
    return nt;
}

// the running forces of the targets become their state
template <int BCAP>
__device__ __forceinline__ void bundle_take(BundleSmem<BCAP> &B, int nt) {
    constexpr int BT = BundleSmem<BCAP>::NT;
#pragma unroll 1
    for (int it = threadIdx.x; it < 12 * nt; it += BT) {
        const int t = it / 12, f = it - 12 * t, s = B.tgt[t];
        B.d[F_AS + f][s] = B.d[F_NAS + f][s];
    }
    __syncthreads();
}

// ---- collision detection ------------------------------------------------------
// unordered pairs {a, b} of each cluster, balanced over members: member a
// takes b = a + d (mod n) for d = 1..n/2 (the pair at distance n/2 once)
template <int BCAP>
__device__ __forceinline__ void bundle_detect(const HardArgs &A, BundleSmem<BCAP> &B, bool second, int p0) {
    constexpr int BT = BundleSmem<BCAP>::NT;
#pragma unroll 1
    for (int p = p0; p < B.used; p += BT) {
        if (B.dead[p]) continue;
        const int k = B.cl[p];
        const int o = B.c_off[k], n = B.c_n[k], a = p - o;
        const bool exact = (B.c_flags[k] & CF_EXACT) != 0;
        const float thr = B.c_thrc[k], fr = B.fr32[p];
#pragma unroll 1
        for (int d = 1; 2 * d <= n; d++) {
            if (2 * d == n && a >= d) break;
            int b = a + d;
            if (b >= n) b -= n;
            const int q = o + b;
            if (!exact) {
                const float rs = fr + B.fr32[q];
                if (bd2_32(B, p, q) > thr * (rs * rs)) continue;
            }
            if (B.dead[q]) continue;
            const int lo = (a < b) ? a : b, hi = (a < b) ? b : a;
            const int gl = B.gslot[o + lo], gh = B.gslot[o + hi];
            const V3 dr = bld(B, F_XP, o + lo) - bld(B, F_XP, o + hi);
            const double d2 = dot(dr, dr);
            const double r2 = A.H.f[gl] * A.H.r_planet[gl] + A.H.f[gh] * A.H.r_planet[gh];
            if (d2 > r2 * r2 * 1.000001) continue;
            const double R = sqrt(d2) / r2;
            if (!(R < 1.)) continue;
            const long long pp = (long long)lo * n + hi;
            if (!second) {
                atomicMin(&B.c_R[k], dbits(R));
                const int i = atomicAdd(&B.n_sv, 1);
                if (i < BSURV) {
                    B.sv_k[i] = k;
                    B.sv_R[i] = R;
                    B.sv_p[i] = pp;
                }
            } else if (dbits(R) == B.c_R[k]) {
                atomicMin((unsigned long long *)&B.c_pb[k], (unsigned long long)pp);
            }
        }
    }
}

// the colliding pair of each cluster that has one (the smallest R, then the
// first ordered pair), and the block step of its alive members
template <int BCAP>
__device__ __noinline__ void bundle_collisions_found(const HardArgs &A) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT;
    if (B.n_sv <= BSURV) {
#pragma unroll 1
        for (int i = threadIdx.x; i < B.n_sv; i += BT)
            if (dbits(B.sv_R[i]) == B.c_R[B.sv_k[i]])
                atomicMin((unsigned long long *)&B.c_pb[B.sv_k[i]], (unsigned long long)B.sv_p[i]);
    } else {
        bundle_detect(A, B, true, threadIdx.x);
    }
    __syncthreads();
#pragma unroll 1
    FOR_CLUSTERS(k) {
        if (B.c_R[k] < dbits(1.)) {
            B.c_flags[k] |= CF_COL;
            const int o = B.c_off[k], n = B.c_n[k];
            const int a = (int)(B.c_pb[k] / n), b = (int)(B.c_pb[k] % n);
            if (B.d[F_MASS][o + a] < B.d[F_MASS][o + b]) { B.c_imp[k] = o + a; B.c_tar[k] = o + b; }
            else { B.c_imp[k] = o + b; B.c_tar[k] = o + a; }
            B.c_act[k] = 0;
        }
    }
    __syncthreads();
#pragma unroll 1
    FOR_SLOTS(p) {
        const int k = B.cl[p];
        if (!(B.c_flags[k] & CF_COL)) continue;
        B.d[F_DT][p] = B.d[F_TE][p] = B.c_ts[k] - B.d[F_TH][p];
        B.flag[p] = B.dead[p] ? 0 : (MF_ACT | MF_TGT);
        if (!B.dead[p]) atomicAdd(&B.c_act[k], 1);
    }
    __syncthreads();
}

// ---- bundle lifecycle ---------------------------------------------------------------
// warp 0: claim clusters from the queue and admit them while they fit (lane
// 0 decides, the decisions are broadcast so the warp's control flow stays
// uniform).  Phase 0: the heavy clusters (the first n_tier[3] of tier 1:
// predicted long chains of block steps), one at a time and alone in the
// bundle, so their iterations stay short; phase 1: the rest, packed.
template <int BCAP>
__device__ __noinline__ void bundle_refill(const HardArgs &A) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    const int lane = threadIdx.x & 31;
    const int n_heavy = A.n_tier[3];
    // (with few clusters no CTA holds some back that others could take)
    const int n_claim = max(1, min(BCLAIM, (A.n_tier[1] - n_heavy) / (int)gridDim.x));
    if (threadIdx.x < 32) {
        int lone = 0;
        if (lane == 0 && B.phase == 0) {
            if (B.ncl > 0) {
                lone = 1;  // a heavy cluster is running: nothing joins it
            } else {
                const int q = atomicAdd(&A.queue[2], 1);
                if (q < n_heavy) {
                    const int c = A.order[A.n_tier[0] + q];
                    const int k = B.ncl++;
                    B.c_idx[k] = c;
                    B.c_off[k] = 0;
                    B.c_n[k] = A.cnt[c];
                    B.c_flags[k] = 0;
                    B.used = B.c_n[k];
                    lone = 1;
                } else {
                    B.phase = 1;
                }
            }
        }
        lone = __shfl_sync(0xffffffffu, lone, 0);
        __syncwarp();
        for (int guard = 0; !lone && guard < (1 << 20); guard++) {
            int stop = 0, claim = 0;
            if (lane == 0 && B.i_pend >= B.n_pend) {
                if (B.exhausted) stop = 1;
                else claim = 1;
            }
            stop = __shfl_sync(0xffffffffu, stop, 0);
            claim = __shfl_sync(0xffffffffu, claim, 0);
            if (stop) break;
            if (claim) {
                int q = 0;
                if (lane == 0) q = atomicAdd(&A.queue[1], n_claim);
                q = __shfl_sync(0xffffffffu, q, 0);
                const int qi = q + lane;
                const bool ok = lane < n_claim && qi < A.n_tier[1] - n_heavy;
                const unsigned m = __ballot_sync(0xffffffffu, ok);
                if (ok) {
                    const int c = A.order[A.n_tier[0] + n_heavy + qi];
                    B.pend_c[lane] = c;
                    B.pend_n[lane] = A.cnt[c];
                }
                __syncwarp();
                if (lane == 0) {
                    B.n_pend = __popc(m);
                    B.i_pend = 0;
                    if (__popc(m) < n_claim) B.exhausted = 1;
                }
                __syncwarp();
                if (m == 0u) break;
            }
            // admit in queue order
            int full = 0;
            if (lane == 0) {
                while (B.i_pend < B.n_pend) {
                    const int c = B.pend_c[B.i_pend], n = B.pend_n[B.i_pend];
                    // with fragmentation, keep room for the fragments of a collision
                    const int room = (A.frag.a_frag > 0.) ? 2 * A.frag.n_frag_max : 0;
                    if (B.used + n + room > BCAP || B.ncl >= bmaxcl(BCAP)) break;
                    const int k = B.ncl++;
                    B.c_idx[k] = c;
                    B.c_off[k] = B.used;
                    B.c_n[k] = n;
                    B.c_flags[k] = 0;
                    B.used += n;
                    B.i_pend++;
                }
                full = B.i_pend < B.n_pend;
            }
            full = __shfl_sync(0xffffffffu, full, 0);
            __syncwarp();
            if (full) break;  // the next claimed cluster waits for space
        }
    }
    __syncthreads();
}

// the start of a block step for the clusters from k0 on: the step's time and
// the collision keys
template <int BCAP>
__device__ __forceinline__ void bundle_open(BundleSmem<BCAP> &B, int k) {
    B.c_ts[k] = bitsd(B.c_key[k]);
    B.c_R[k] = dbits(1.);
    B.c_pb[k] = 0x7fffffffffffffffLL;
    B.c_flags[k] &= ~CF_COL;
    B.c_act[k] = 0;
    B.c_steps[k]++;
}

// load the fresh clusters (bundle indices fresh_k..ncl-1, slots
// fresh_p..used-1), their first full force and the time of their first step
template <int BCAP>
__device__ __noinline__ void bundle_load(const HardArgs &A) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT;
    const Hard &H = A.H;
    const int tid = threadIdx.x;
    const int k0 = B.fresh_k, k1 = B.ncl, p0 = B.fresh_p, p1 = B.used;
#pragma unroll 1
    for (int k = k0 + tid; k < k1; k += BT) {
        const int c = B.c_idx[k];
        const int goff = A.off[c];
        B.c_goff[k] = goff;
        const V3 r0 = ld3(A.S.pos, A.members[goff]);
        B.c_ref[0][k] = r0.x; B.c_ref[1][k] = r0.y; B.c_ref[2][k] = r0.z;
        B.c_steps[k] = 0; B.c_work[k] = 0;
        B.c_n0[k] = B.c_n[k];
        B.c_addn[k] = 0;
        ClusterRec &R = A.crec[c];
        R.t0 = A.times ? global_ns() : 0;
        R.ed = R.edd = 0.;
        R.n_frag = 0;
        R.n_col = 0;
        // maxima of |x - ref| and |v| components and of r_out_inv, minimum of f r_planet
        B.c_key[k] = 0ULL;
        B.c_tm[k] = 0ULL;
        B.c_R[k] = 0ULL;
        B.c_pb[k] = (long long)dbits(1.e300);
    }
    __syncthreads();
#pragma unroll 1
    for (int p = p0 + tid; p < p1; p += BT) {
        int lo = k0, hi = k1 - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (B.c_off[mid] <= p) lo = mid;
            else hi = mid - 1;
        }
        const int k = lo, g = B.c_goff[k] + (p - B.c_off[k]), i = A.members[g];
        // FPHard(const FPGrav&), src/particle.h:1096-1116 (the forces come
        // from the first full pass)
        const V3 x = ld3(A.S.pos, i), v = ld3(A.S.vel, i);
        const double mass = A.S.mass[i], rp = A.S.r_planet[i], f = A.S.f[i], roi = A.S.r_out_inv[i], dt = A.S.dt[i];
        const double acc0 = A.S.acc0[i], tc = A.S.time[i];
        const int64_t id = A.S.id[i];
        bst(B, F_POS, p, x);
        bst(B, F_VEL, p, v);
        B.d[F_MASS][p] = mass;
        B.d[F_ROI][p] = roi;
        B.d[F_TH][p] = 0.;
        B.d[F_DT][p] = dt;
        B.d[F_TE][p] = 0. + dt;
        B.d[F_A02][p] = A.P.alpha2 * acc0 * acc0;
        H.mass[g] = mass; H.r_planet[g] = rp; H.f[g] = f; H.r_out_inv[g] = roi;
        H.time_c[g] = tc; H.acc0[g] = acc0; H.id[g] = id;
        H.dead[g] = 0; H.merged[g] = 0;
        H.tw_head[g] = H.tw_tail[g] = H.tw_next[g] = -1;
        const double fr = f * rp;
        B.fr32[p] = (float)fr;
        B.roi32[p] = (float)roi;
        // the high word of a double just below r_out / 128
        B.hmov[p] = (int)(__float_as_uint(0.0078f / B.roi32[p]) >> 3) + (896 << 20);
        B.gslot[p] = g;
        B.cl[p] = (short)k;
        B.eqc[p] = (short)p;
        B.owner[p] = B.twh[p] = B.twn[p] = -1;
        B.dead[p] = B.merged[p] = 0;
        const double ext = dmax(fabs(x.x - B.c_ref[0][k]), dmax(fabs(x.y - B.c_ref[1][k]), fabs(x.z - B.c_ref[2][k])));
        const double vm = dmax(fabs(v.x), dmax(fabs(v.y), fabs(v.z)));
        atomicMax(&B.c_key[k], dbits(ext));
        atomicMax(&B.c_tm[k], dbits(vm));
        atomicMax(&B.c_R[k], dbits(roi));
        atomicMin((unsigned long long *)&B.c_pb[k], dbits(fr));
    }
    __syncthreads();
#pragma unroll 1
    for (int k = k0 + tid; k < k1; k += BT) {
        // coordinate bound, then the prefilter thresholds (see the header)
        const double E = (bitsd(B.c_key[k]) + 2. * bitsd(B.c_tm[k]) * A.t_end) * 1.0001 + 1.e-30;
        const double err = 3.e-7 * E;
        const double rmax = bitsd(B.c_R[k]), frmin = bitsd((unsigned long long)B.c_pb[k]);
        const double tf = 1.000001 + 1.0001 * err * rmax;
        const double tc = 1.000001 + 1.0001 * err / (2. * frmin);
        B.c_thrf[k] = __double2float_ru(tf * tf * 1.000001);
        B.c_thrc[k] = (frmin > 0.) ? __double2float_ru(tc * tc * 1.000001) : __int_as_float(0x7f800000);
        B.c_E32[k] = __double2float_rd(E);
        B.c_key[k] = dbits(1.e10);
    }
#pragma unroll 1
    for (int p = tid; p < p1; p += BT) B.flag[p] = p < p0 ? 0 : MF_TGT;
    __syncthreads();
#pragma unroll 1
    for (int p = p0 + tid; p < p1; p += BT) atomicMin(&B.c_key[B.cl[p]], dbits(B.d[F_TE][p]));
    const int nt = bundle_full<BCAP>(A, false);
    bundle_take(B, nt);
#pragma unroll 1
    for (int k = k0 + tid; k < k1; k += BT) bundle_open(B, k);
    if (tid == 0) B.n_sv = B.moved = 0;
    __syncthreads();
}

// every field of slot p from the state of record (global slot g), after a collision
template <int BCAP>
__device__ __forceinline__ void bundle_reload(const HardArgs &A, BundleSmem<BCAP> &B, int p, int g, int k) {
    const Hard &H = A.H;
    bst(B, F_POS, p, ld3(H.pos, g));
    bst(B, F_VEL, p, ld3(H.vel, g));
    B.d[F_MASS][p] = H.mass[g];
    B.d[F_ROI][p] = H.r_out_inv[g];
    B.d[F_TH][p] = H.th[g];
    B.d[F_DT][p] = H.dt[g];
    B.d[F_TE][p] = 0.;
    B.d[F_A02][p] = A.P.alpha2 * H.acc0[g] * H.acc0[g];
    B.fr32[p] = (float)(H.f[g] * H.r_planet[g]);
    B.roi32[p] = (float)H.r_out_inv[g];
    B.hmov[p] = (int)(__float_as_uint(0.0078f / B.roi32[p]) >> 3) + (896 << 20);
    B.dead[p] = (unsigned char)H.dead[g];
    B.merged[p] = (unsigned char)H.merged[g];
    B.gslot[p] = g;
    B.cl[p] = (short)k;
    for (int f = F_AS; f < F_MASS; f++) B.d[f][p] = 0.;
}

// Slot p's new place: its persistent fields move to slot q (>= 0) with the
// cluster index k and its cluster's shift dp; every thread calls it, PER slots each.
template <int BCAP>
__device__ __forceinline__ void bundle_move(BundleSmem<BCAP> &B, const int *mv_new, const int *mv_k, const int *mv_d) {
    constexpr int BT = BundleSmem<BCAP>::NT, PER = BCAP / BT;
    const int tid = threadIdx.x;
#pragma unroll 1
    for (int f = 0; f < F_KEEP; f += 8) {
        double v[PER][8];
#pragma unroll
        for (int j = 0; j < PER; j++)
            if (mv_new[j] >= 0)
#pragma unroll
                for (int u = 0; u < 8; u++) v[j][u] = B.d[f + u][tid + j * BT];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < PER; j++)
            if (mv_new[j] >= 0)
#pragma unroll
                for (int u = 0; u < 8; u++) B.d[f + u][mv_new[j]] = v[j][u];
    }
    float r32[PER], f32[PER];
    int gs[PER], hm[PER], lk[PER][4], dm[PER];
#pragma unroll
    for (int j = 0; j < PER; j++)
        if (mv_new[j] >= 0) {
            const int p = tid + j * BT;
            auto sh = [&](int x) { return x >= 0 ? x + mv_d[j] : -1; };
            r32[j] = B.roi32[p]; f32[j] = B.fr32[p];
            gs[j] = B.gslot[p]; hm[j] = B.hmov[p];
            lk[j][0] = sh(B.owner[p]); lk[j][1] = sh(B.eqc[p]); lk[j][2] = sh(B.twh[p]); lk[j][3] = sh(B.twn[p]);
            dm[j] = B.dead[p] | (B.merged[p] << 8);
        }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; j++)
        if (mv_new[j] >= 0) {
            const int q = mv_new[j];
            B.roi32[q] = r32[j]; B.fr32[q] = f32[j];
            B.gslot[q] = gs[j]; B.hmov[q] = hm[j];
            B.cl[q] = (short)mv_k[j];
            B.owner[q] = (short)lk[j][0]; B.eqc[q] = (short)lk[j][1]; B.twh[q] = (short)lk[j][2];
            B.twn[q] = (short)lk[j][3];
            B.dead[q] = (unsigned char)(dm[j] & 0xff);
            B.merged[q] = (unsigned char)(dm[j] >> 8);
        }
    __syncthreads();
}

// Clusters made fragments (KOMINAMI): their member ranges grow by them and the
// clusters after them move up.  Where the bundle has no room for all, the growing
// clusters leave it; k_hard_wide takes them up after the launch, from the state of
// record that their collision has just written, in a bundle of BCAP_WIDE slots each.
template <int BCAP>
__device__ __noinline__ void bundle_grow(const HardArgs &A) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT, PER = BCAP / BT;
    const int tid = threadIdx.x;
    static_assert(bmaxcl(BCAP) <= BT, "one thread per bundle cluster");
    const int add = (tid < B.ncl) ? B.c_addn[tid] : 0;
    const int my_n = (tid < B.ncl) ? B.c_n[tid] : 0;
    int tot;
    const int noff = bscan<BT>(my_n + add, B.ws, tot);
    if (tot > BCAP) {
        if (BCAP == BCAP_WIDE) {  // one cluster: no form has more slots
            if (tid == 0) atomicOr(A.status, ST_CLUSTER_TOO_BIG);
        } else if (add > 0) {
            ClusterRec &R = A.crec[B.c_idx[tid]];
            R.steps = B.c_steps[tid];
            R.work = B.c_work[tid];
            A.left[atomicAdd(&A.queue[4], 1)] = B.c_idx[tid];
            B.c_flags[tid] = (B.c_flags[tid] & ~CF_COL) | CF_GONE;
        }
        __syncthreads();
        return;
    }
    if (tid < B.ncl) B.c_key[tid] = (unsigned long long)(unsigned)noff;  // new offsets, by cluster
    __syncthreads();
    int mv_new[PER], mv_k[PER], mv_d[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int p = tid + j * BT;
        mv_new[j] = -1;
        if (p < B.used) {
            const int k = B.cl[p];
            mv_k[j] = k;
            mv_d[j] = (int)B.c_key[k] - B.c_off[k];
            mv_new[j] = p + mv_d[j];
        }
    }
    __syncthreads();
    bundle_move(B, mv_new, mv_k, mv_d);
    if (tid < B.ncl) {
        B.c_off[tid] = noff;
        B.c_n[tid] = my_n + add;
        // fragments are smaller than the members the prefilter margins were
        // set for: exact FP64 tests for this cluster from here on
        if (add > 0) B.c_flags[tid] |= CF_EXACT;
        for (int i = 0; i < add; i++) {
            const int q = noff + my_n + i;
            bundle_reload(A, B, q, B.c_addg[tid] + i, tid);
            B.eqc[q] = (short)q;
            B.owner[q] = B.twh[q] = B.twn[q] = -1;
        }
    }
    if (tid == 0) B.used = tot;
    __syncthreads();
}

// slot p of cluster k from the state of record, with its merge lists as slots:
// twins, their owner, equal ids (every slot's gslot is set)
template <int BCAP>
__device__ __forceinline__ void bundle_rejoin(const HardArgs &A, BundleSmem<BCAP> &B, int p, int k) {
    const Hard &H = A.H;
    const int g = B.gslot[p], o = B.c_off[k], n = B.c_n[k];
    bundle_reload(A, B, p, g, k);
    auto slot_of = [&](int t) {
        if (t >= 0)
            for (int q = 0; q < n; q++)
                if (B.gslot[o + q] == t) return o + q;
        return -1;
    };
    B.twh[p] = (short)slot_of(H.tw_head[g]);
    B.twn[p] = (short)slot_of(H.tw_next[g]);
    const int64_t id = H.id[g];
    int own = -1, eq = p;
    for (int q = n - 1; q >= 0; q--) {
        const int gj = B.gslot[o + q];
        if (H.id[gj] == id) eq = o + q;
        if (H.merged[gj])
            for (int t = H.tw_head[gj], gg = 0; t >= 0 && gg < 4096; t = H.tw_next[t], gg++)
                if (t == g) own = o + q;
    }
    B.owner[p] = (short)own;
    B.eqc[p] = (short)eq;
    if (B.dead[p]) B.any_dead = 1;
}

// the clusters of a collision, their members back from the state of record: a
// full force and first time steps
template <int BCAP>
__device__ __noinline__ void bundle_restart(const HardArgs &A) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT;
    const Params &P = A.P;
    const Hard &H = A.H;
#pragma unroll 1
    FOR_SLOTS(p) B.flag[p] = (B.c_flags[B.cl[p]] & CF_COL) ? MF_TGT : 0;
    __syncthreads();
    const int nc = bundle_full<BCAP>(A, false);
    bundle_take(B, nc);
#pragma unroll 1
    for (int i = threadIdx.x; i < nc; i += BT) {
        const int s = B.tgt[i];
        if (B.dead[s]) continue;
        B.d[F_DT][s] = dt_initial(P, B.d[F_TH][s], B.d[F_DT][s], H.acc0[B.gslot[s]], bld(B, F_AD, s), bld(B, F_JD, s),
                                  bld(B, F_AS, s), bld(B, F_JS, s));
    }
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < nc; i += BT) {
        const int s = B.tgt[i];
        if (B.merged[s])
            for (int t = B.twh[s], gg = 0; t >= 0 && gg < BCAP; t = B.twn[t], gg++) B.d[F_DT][t] = B.d[F_DT][s];
    }
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < nc; i += BT) {
        const int s = B.tgt[i];
        B.d[F_TE][s] = B.d[F_TH][s] + B.d[F_DT][s];
    }
    __syncthreads();
}

// the collisions of the block step: the colliding clusters' state goes to
// the state of record, one thread per cluster resolves the collision on it,
// and their members come back with a full force and first time steps
template <int BCAP>
__device__ __noinline__ void bundle_collide(const HardArgs &A) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT;
    const Params &P = A.P;
    const Hard &H = A.H;
#pragma unroll 1
    FOR_SLOTS(p) {
        if (!(B.c_flags[B.cl[p]] & CF_COL)) continue;
        const int g = B.gslot[p];
        st3(H.pos, g, bld(B, F_POS, p));
        st3(H.vel, g, bld(B, F_VEL, p));
        H.th[g] = B.d[F_TH][p];
        H.dt[g] = B.d[F_DT][p];
        H.phi_d[g] = 0.;
        H.phi_s[g] = 0.;
    }
    if (threadIdx.x == 0) B.grew = 0;
    __syncthreads();
#pragma unroll 1
    FOR_CLUSTERS(k) {
        B.c_addn[k] = 0;
        if (!(B.c_flags[k] & CF_COL)) continue;
        ColRec rec;
        double e1 = 0., e2 = 0.;
        const int o = B.c_off[k], n = B.c_n[k], c = B.c_idx[k];
        ClusterRec &R = A.crec[c];
        int fs[32];
        FragCtx X{&A, &B.gslot[o], n, c, A.S.id_cluster[A.members[B.c_goff[k]]], &R.n_frag, fs};
        const int nf = collide(P, H, B.gslot[B.c_imp[k]], B.gslot[B.c_tar[k]], e1, e2, rec, &X);
        R.ed += e1;
        R.edd += e2;
        rec.cluster = c;
        rec.seq = R.n_col++;
        rec.n = B.c_n0[k];
        const int slot = atomicAdd(A.n_cols, 1);
        if (slot < A.col_cap) A.cols[slot] = rec;
        else atomicOr(A.status, ST_QUEUE_OVERFLOW);
        if (nf > 0) {
            B.c_addn[k] = nf;
            B.c_addg[k] = fs[0];  // a collision's fragments have consecutive slots
            B.grew = 1;
            for (int i = 0; i < nf; i++) A.frags[fs[i] - A.frag_base].n0 = B.c_n0[k];
        }
    }
    __threadfence_block();
    __syncthreads();
#pragma unroll 1
    FOR_SLOTS(p) {
        const int k = B.cl[p];
        B.flag[p] = 0;
        if (!(B.c_flags[k] & CF_COL)) continue;
        bundle_rejoin(A, B, p, k);
    }
    __syncthreads();
    if (B.grew) bundle_grow<BCAP>(A);
    bundle_restart<BCAP>(A);
}

__device__ __noinline__ double dt_next_general(const HardArgs &A, double time, double dt, double dt_1) {
    return dt_next_hermite(A.P, time, dt, dt_1);
}
// dt_next_hermite by the exponents: its halvings of a power of two against
// the time's lowest set bit and the criterion's exponent
__device__ __forceinline__ double dt_next_bits(const HardArgs &A, double time, double dt, double dt_1) {
    const Params &P = A.P;
    const double dmax_ = 0.5 * P.dt_tree;
    if (!is_pow2(dt) || !is_pow2(dmax_) || !(dhi(time) >= 0 && dhi(time) < 0x7fe00000) || dhi(dt_1) < 0)
        return dt_next_general(A, time, dt, dt_1);
    const int ed = dhi(dt) >> 20;
    int e = min(ed + 1, dhi(dmax_) >> 20);
    const unsigned long long b = dbits(time), m = (b & ((1ULL << 52) - 1)) | (1ULL << 52);
    if (b != 0ULL) {  // time a multiple of 2^e: e at most its lowest set bit's exponent
        const int et = (int)(b >> 52);
        if (et == 0) return dt_next_general(A, time, dt, dt_1);
        e = min(e, et - 52 + (__ffsll((long long)m) - 1));
    }
    if (e < 64) return dt_next_general(A, time, dt, dt_1);
    const int e1 = dhi(dt_1) >> 20;
    while (e1 < e && ed - 1 < e) e--;  // dt_1 < 2^e: its exponent is smaller
    const double next = __hiloint2double(e << 20, 0);
    return plt(next, 2. * P.dt_min) ? P.dt_min : next;
}

// dmin of two criteria: by their bits unless one is NaN or negative
__device__ __forceinline__ double dmin_crit(double a, double b) {
    const unsigned long long inf = 0x7ff0000000000000ULL;
    return dbits(a) <= inf && dbits(b) <= inf ? pmin(a, b) : dmin(a, b);
}

// time and calcDeltat (src/particle.h:1276-1314) of the targets, and their
// running forces into the state.  The two criteria (planets, sun) of a target
// in a pair of lanes; when there are few targets, the four norms of each in
// lanes of their own.
template <int BCAP>
__device__ __forceinline__ void bundle_dt(const HardArgs &A, BundleSmem<BCAP> &B, int nt) {
    constexpr int BT = BundleSmem<BCAP>::NT;
    constexpr unsigned ALL = 0xffffffffu;
    const Params &P = A.P;
    const bool wide = 8 * nt <= BT;
    const int sh = wide ? 3 : 1, L = 1 << sh;  // lanes a target
#pragma unroll 1
    for (int base = 0; base < L * nt; base += BT) {
        const int i = base + threadIdx.x;
        if (i - (i & 31) >= L * nt) break;  // no target in this warp
        const int t = min(i >> sh, nt - 1), r = i & (L - 1);
        const bool act = i < L * nt;
        const int s = B.tgt[t], k = B.cl[s];
        double num, den, Jerk;  // dt4th (p3t_phys.cuh): eta sqrt((Acc Snap + Jerk^2) / (Jerk Crac + Snap^2))
        const int sun = wide ? r >> 2 : r;
        if (wide) {
            const int w = r & 3;
            // acc and jerk as the last pass left them, snap and crackle as the corrector did
            const int f = (w < 2) ? (sun ? F_NAS : F_NAD) + 3 * w : (sun ? F_AS : F_AD) + 3 * (w - 2);
            const V3 v = bld(B, f, s);
            const double n2 = dot(v, v) + (w == 0 && !sun ? B.d[F_A02][s] : 0.);
            const double nn = sqrt_rn(n2);
            // even lanes: Acc Snap + Jerk^2, odd lanes: Jerk Crac + Snap^2
            const double m1 = __shfl_sync(ALL, nn, w & 1, 4), m2 = __shfl_sync(ALL, nn, 2 + (w & 1), 4);
            const double q2 = __shfl_sync(ALL, n2, 1 + (w & 1), 4);
            Jerk = __shfl_sync(ALL, nn, 1, 4);
            const double nd = m1 * m2 + q2;
            num = __shfl_sync(ALL, nd, 0, 4);
            den = __shfl_sync(ALL, nd, 1, 4);
        } else {
            // a norm after the other
            double n2[4];
#pragma unroll
            for (int w = 0; w < 4; w++) {
                const V3 v = bld(B, (w < 2) ? (sun ? F_NAS : F_NAD) + 3 * w : (sun ? F_AS : F_AD) + 3 * (w - 2), s);
                n2[w] = dot(v, v);
            }
            n2[0] = n2[0] + (sun ? 0. : B.d[F_A02][s]);
            double nn[4];
#pragma unroll 1
            for (int w = 0; w < 4; w++) nn[w] = sqrt_rn(n2[w]);
            num = nn[0] * nn[2] + n2[1];
            den = nn[1] * nn[3] + n2[2];
            Jerk = nn[1];
        }
        const double crit = (dbits(Jerk) << 1) != 0ULL ? (sun ? P.eta_sun : P.eta) * sqrt_rn(div_rn(num, den))
                                                       : 1.7976931348623157e308;
        const double other = __shfl_xor_sync(ALL, crit, L / 2);
        if (act) {
            for (int f = r; f < 12; f += L) B.d[F_AS + f][s] = B.d[F_NAS + f][s];
            if (r == 0) {
                const double th = B.d[F_TH][s] + B.d[F_TE][s];
                B.d[F_TH][s] = th;
                double dt = B.d[F_DT][s];
                if (!(B.c_flags[k] & CF_COL) && !B.dead[s]) {
                    dt = dt_next_bits(A, th, dt, dmin_crit(crit, other));
                    B.d[F_DT][s] = dt;
                }
                B.d[F_TE][s] = th + dt;
            }
        }
    }
    __syncthreads();
    if (B.any_dead) {  // a twin's block step is its target's
#pragma unroll 1
        for (int i = threadIdx.x; i < nt; i += BT) {
            const int s = B.tgt[i], k = B.cl[s];
            if (B.dead[s] && B.owner[s] >= 0 && !(B.c_flags[k] & CF_COL)) B.d[F_DT][s] = B.d[F_DT][B.owner[s]];
        }
        __syncthreads();
    }
}

// the end of a block step (col: with collisions): each cluster's next step is opened,
// or the cluster is finished (or gone), which sets any
template <int BCAP>
__device__ __forceinline__ void bundle_advance(const HardArgs &A, BundleSmem<BCAP> &B, int used, bool col) {
    constexpr int BT = BundleSmem<BCAP>::NT;
    // getSystemTime (src/hermite.h:25-35) and makeActiveList's next time
    // (src/hermite.h:4-24): the minima of th and th + dt over the alive members
    if (threadIdx.x == 0) B.any = B.n_sv = B.moved = 0;
    if (col) {
#pragma unroll 1
        FOR_CLUSTERS(k) B.c_key[k] = B.c_tm[k] = dbits(1.e10);
        __syncthreads();
    }
    if (used <= 32 && B.ncl == 1 && !col) {  // one cluster: by a warp
        if (threadIdx.x < 32) {
            const int p = threadIdx.x;
            const bool in = p < used && !B.dead[p];
            const unsigned long long th = warp_min64(in ? dbits(B.d[F_TH][p]) : ~0ULL),
                                     te = warp_min64(in ? dbits(B.d[F_TE][p]) : ~0ULL);
            if (p == 0) {
                B.c_tm[0] = min(th, dbits(1.e10));
                B.c_key[0] = min(te, dbits(1.e10));
            }
        }
    } else {
#pragma unroll 1
        FOR_SLOTS(p) {
            if (B.dead[p]) continue;
            const int k = B.cl[p];
            atomicMin(&B.c_tm[k], dbits(B.d[F_TH][p]));
            atomicMin(&B.c_key[k], dbits(B.d[F_TE][p]));
        }
    }
    __syncthreads();
#pragma unroll 1
    FOR_CLUSTERS(k) {
        const bool going = B.c_tm[k] < dbits(A.t_end) && !(B.c_flags[k] & CF_GONE);
        if (going && B.c_steps[k] < A.max_steps) {
            bundle_open(B, k);
        } else {
            if (going) atomicOr(A.status, ST_ITER_CAP);
            B.c_flags[k] |= CF_FIN;
            B.any = 1;
        }
    }
    __syncthreads();
    HP_MARK(HP_TIME);
}

// one block step of every cluster in the bundle (timeIntegrate_multi body,
// src/hermite.h:224-479), whose time bundle_open has set
template <int BCAP>
__device__ __forceinline__ void bundle_step(const HardArgs &A, BundleSmem<BCAP> &B) {
    constexpr int BT = BundleSmem<BCAP>::NT;
    // FPHard::predict (src/particle.h:1183-1206), one lane per (member,
    // component): predict()'s roundings, the products by a power-of-two Dt
    // fused where they are exact.  The active set: the alive members whose
    // step ends now.
    const int used = B.used, lane = threadIdx.x & 31;
#pragma unroll 1
    for (int w0 = threadIdx.x - lane; w0 < 3 * used; w0 += BT) {  // whole warps
        const int it = min(w0 + lane, 3 * used - 1);
        const int c = it >= 2 * used ? 2 : (it >= used ? 1 : 0), p = it - c * used, k = B.cl[p];
        const double ts = B.c_ts[k], Dt = ts - B.d[F_TH][p];
        const double x = B.d[F_POS + c][p], v = B.d[F_VEL + c][p];
        const double a = B.d[F_AS + c][p] + B.d[F_AD + c][p], j = B.d[F_JS + c][p] + B.d[F_JD + c][p];
        const double hD = Dt * 0.5, u = fma(0.5, a, 1.6666666666666667e-1 * Dt * j);
        double xp, vp;
        if (__all_sync(0xffffffffu, is_pow2(Dt))) {
            xp = fma(Dt, fma(Dt, u, v), x);
            vp = fma(Dt, fma(hD, j, a), v);
        } else {
            xp = x + Dt * (v + Dt * u);
            vp = v + Dt * (a + hD * j);
        }
        if (w0 + lane >= 3 * used) continue;
        B.d[F_XP + c][p] = xp;
        B.d[F_VP + c][p] = vp;
        st32b(B, c, p, xp, k);
        if (c == 0) {
            const bool act = !B.dead[p] && dbits(B.d[F_TE][p]) == dbits(ts);
            B.flag[p] = act ? (MF_ACT | MF_TGT) : 0;
            if (act) {
                B.d[F_TE][p] = Dt;
                atomicAdd(&B.c_act[k], 1);
            }
        }
    }
    __syncthreads();
    HP_MARK(HP_PREDICT);
    // collisionDetermination, src/hermite.h:98-196
    // beside it, in warp 0, the lists of a small bundle (made again if there is a
    // collision, whose targets are others)
    bool listed = false;
    const bool small = used <= 32 && !B.any_dead;
    if (!small) bundle_detect(A, B, false, threadIdx.x);
    else if (threadIdx.x >= 32) bundle_detect(A, B, false, threadIdx.x - 32);
    else bundle_lists_small(A, B);
    __syncthreads();
    const bool col = B.n_sv > 0;
    if (col) bundle_collisions_found<BCAP>(A);
    HP_MARK(HP_DETECT);
    if (B.any_dead) {  // the twins of active merged members
#pragma unroll 1
        FOR_SLOTS(p) {
            const int ow = B.owner[p];
            if (B.dead[p] && ow >= 0 && (B.flag[ow] & MF_ACT)) {
                B.flag[p] |= MF_TGT;
                B.d[F_TE][p] = B.c_ts[B.cl[p]] - B.d[F_TH][p];
            }
        }
        __syncthreads();
    }
    int nt;
    if (small && !col) {
        nt = B.nt;
        listed = B.pfx[nt] <= 4 * 32;
    } else {
        nt = bundle_targets(B, MF_TGT);
    }
    HP_MARK(HP_ACTIVE);
    // predicted forces and first correction, corrected forces and second
    // correction, corrected forces
#pragma unroll 1
    for (int ps = 0; ps < 3; ps++) bundle_pass<BCAP, false>(A, B, ps == 0 ? 1 : 2, nt, false, (ps + 1) % 3, listed);
#pragma unroll 1
    FOR_CLUSTERS(k) {
        B.c_work[k] += (long long)B.c_act[k] * B.c_n[k];
        B.c_key[k] = B.c_tm[k] = dbits(1.e10);
    }
    bundle_dt(A, B, nt);
    HP_MARK(HP_DT);
    if (col) bundle_collide<BCAP>(A);
    HP_MARK(HP_COLLIDE);
    bundle_advance(A, B, used, col);
}

// final forces, write-back and removal of the finished clusters (those that are gone
// are only removed)
template <int BCAP>
__device__ __noinline__ void bundle_retire(const HardArgs &A) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT, PER = BCAP / BT;
    const Hard &H = A.H;
    const int tid = threadIdx.x;
#pragma unroll 1
    FOR_SLOTS(p) B.flag[p] = (B.c_flags[B.cl[p]] & (CF_FIN | CF_GONE)) == CF_FIN ? MF_TGT : 0;
    __syncthreads();
    const int nt = bundle_full<BCAP>(A, true);
    // write back to FPGrav, with resetTime (src/hard.h:768-787)
#pragma unroll 1
    for (int i = tid; i < nt; i += BT) {
        const int s = B.tgt[i], g = B.gslot[s], k = B.cl[s];
        const double th = B.d[F_TH][s], dt = B.d[F_DT][s];
        const V3 x = bld(B, F_POS, s), v = bld(B, F_VEL, s), as = bld(B, F_NAS, s), js = bld(B, F_NJS, s),
                 ad = bld(B, F_NAD, s), jd = bld(B, F_NJD, s);
        const double phd = B.d[F_PHD][s], phs = B.d[F_PHS][s];
        if (g >= A.frag_base) {  // a fragment: joins the system after the launch
            A.frags[g - A.frag_base].n_cl = B.c_n[k];
            st3(H.pos, g, x); st3(H.vel, g, v); st3(H.acc_s, g, as); st3(H.jerk_s, g, js);
            st3(H.acc_d, g, ad); st3(H.jerk_d, g, jd);
            H.phi_d[g] = phd; H.phi_s[g] = phs; H.th[g] = th; H.dt[g] = dt;
            continue;
        }
        const int idx = A.members[g];
        st3(A.S.pos, idx, x); st3(A.S.vel, idx, v);
        st3(A.S.acc_s, idx, as); st3(A.S.jerk_s, idx, js);
        st3(A.S.acc_d, idx, ad); st3(A.S.jerk_d, idx, jd);
        A.S.phi_d[idx] = phd; A.S.phi_s[idx] = phs;
        A.S.mass[idx] = B.d[F_MASS][s]; A.S.r_planet[idx] = H.r_planet[g];
        A.S.time[idx] = H.time_c[g] + th; A.S.dt[idx] = dt;
        A.S.id[idx] = H.id[g];
        A.S.dead[idx] = B.dead[s]; A.S.merged[idx] = B.merged[s];
        A.S.n_cluster[idx] = B.c_n[k];
    }
#pragma unroll 1
    FOR_CLUSTERS(k) {
        if ((B.c_flags[k] & (CF_FIN | CF_GONE)) != CF_FIN) continue;
        const int c = B.c_idx[k];
        const ClusterRec &R = A.crec[c];
        A.cl_edisp[2 * c] = (R.n_col > 0) ? R.ed : 0.;
        A.cl_edisp[2 * c + 1] = (R.n_col > 0) ? R.edd : 0.;
        if (A.cost) {
            A.cost[2 * c] = B.c_steps[k];
            A.cost[2 * c + 1] = B.c_work[k];
        }
        if (A.times) {
            A.times[2 * c] = R.t0;
            A.times[2 * c + 1] = global_ns();
        }
    }
    // compaction: kept clusters move down, in order
    int keep = 0, nk = 0, nkeep = 0, noff = 0, tot = 0;
    int t_idx = 0, t_n = 0, t_goff = 0, t_steps = 0, t_flags = 0, t_n0 = 0;
    double t_ts = 0., t_ref0 = 0., t_ref1 = 0., t_ref2 = 0.;
    long long t_work = 0;
    float t_thrf = 0.f, t_thrc = 0.f, t_E = 0.f;
    if (tid < B.ncl) {
        keep = !(B.c_flags[tid] & CF_FIN);
        t_idx = B.c_idx[tid]; t_n = B.c_n[tid]; t_goff = B.c_goff[tid];
        t_steps = B.c_steps[tid]; t_flags = B.c_flags[tid]; t_n0 = B.c_n0[tid];
        t_ts = B.c_ts[tid]; t_ref0 = B.c_ref[0][tid]; t_ref1 = B.c_ref[1][tid]; t_ref2 = B.c_ref[2][tid];
        t_work = B.c_work[tid];
        t_thrf = B.c_thrf[tid]; t_thrc = B.c_thrc[tid]; t_E = B.c_E32[tid];
    }
    static_assert(bmaxcl(BCAP) <= BT, "one thread per bundle cluster");
    noff = bscan<BT>(keep ? (t_n << 10) | 1 : 0, B.ws, tot);
    nk = noff & 1023;
    noff >>= 10;
    nkeep = tot & 1023;
    tot >>= 10;
    // old -> new offset and index per kept cluster, through c_key (free here)
    if (tid < B.ncl)
        B.c_key[tid] = keep ? ((unsigned long long)(unsigned)noff | ((unsigned long long)(unsigned)nk << 32)) : ~0ULL;
    __syncthreads();
    int mv_new[PER], mv_k[PER], mv_d[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int p = tid + j * BT;
        mv_new[j] = -1;
        if (p < B.used) {
            const int k = B.cl[p];
            const unsigned long long key = B.c_key[k];
            if (key != ~0ULL) {
                mv_k[j] = (int)(key >> 32);
                mv_d[j] = (int)(key & 0xffffffffULL) - B.c_off[k];
                mv_new[j] = p + mv_d[j];
            }
        }
    }
    __syncthreads();
    if (nkeep > 0) bundle_move(B, mv_new, mv_k, mv_d);
    if (keep) {
        B.c_idx[nk] = t_idx; B.c_off[nk] = noff; B.c_n[nk] = t_n; B.c_goff[nk] = t_goff;
        B.c_steps[nk] = t_steps; B.c_flags[nk] = t_flags; B.c_n0[nk] = t_n0;
        B.c_ts[nk] = t_ts; B.c_ref[0][nk] = t_ref0; B.c_ref[1][nk] = t_ref1; B.c_ref[2][nk] = t_ref2;
        B.c_work[nk] = t_work;
        B.c_thrf[nk] = t_thrf; B.c_thrc[nk] = t_thrc; B.c_E32[nk] = t_E;
        B.c_R[nk] = dbits(1.);
        B.c_pb[nk] = 0x7fffffffffffffffLL;
        B.c_act[nk] = 0;
        B.c_addn[nk] = 0;
    }
    if (tid == 0) {
        B.ncl = nkeep;
        B.used = tot;
        B.any_dead = 0;
    }
    __syncthreads();
#pragma unroll 1
    FOR_SLOTS(p) {
        if (B.dead[p]) B.any_dead = 1;
    }
    __syncthreads();
}

template <int BCAP>
__device__ __forceinline__ void bundle_init(BundleSmem<BCAP> &B) {
    if (threadIdx.x == 0) {
        B.used = B.ncl = B.n_pend = B.i_pend = B.exhausted = B.phase = 0;
        B.n_sv = B.moved = B.any = B.any_dead = 0;
        B.live[0] = B.live[1] = 0ULL;
        for (int k = 0; k < HP_N; k++) B.ph_acc[k] = 0;
        B.ph_t = clock64();
    }
}
template <int BCAP>
__device__ __forceinline__ void bundle_close(const HardArgs &A, BundleSmem<BCAP> &B) {
    if (threadIdx.x == 0 && A.live) {
        atomicAdd(&A.live[0], B.live[0]);
        atomicAdd(&A.live[1], B.live[1]);
    }
    if (A.phase_cycles && threadIdx.x == 0)
        for (int k = 0; k < HP_N; k++) atomicAdd(&A.phase_cycles[k], (unsigned long long)B.ph_acc[k]);
}

// Cluster c, which a bundle left in bundle_grow, in a wide bundle of its own: members
// and, in the order they were made, fragments from the state of record, then the rest of
// that block step.  The bundle's prefilter bounds are not kept: every pair gets its
// exact test.  False: too many for the wide bundle.
template <int BCAP>
__device__ __noinline__ bool bundle_resume(const HardArgs &A, int c) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    constexpr int BT = BundleSmem<BCAP>::NT;
    const ClusterRec &R = A.crec[c];
    const int tid = threadIdx.x, n0 = A.cnt[c], n = n0 + (int)R.n_frag, goff = A.off[c];
    if (n > BCAP) {
        if (tid == 0) atomicOr(A.status, ST_CLUSTER_TOO_BIG);
        return false;
    }
    if (tid == 0) {
        B.ncl = 1;
        B.used = n;
        B.any_dead = B.n_sv = B.moved = 0;
        B.c_idx[0] = c;
        B.c_off[0] = 0;
        B.c_n[0] = n;
        B.c_n0[0] = n0;
        B.c_goff[0] = goff;
        B.c_addn[0] = 0;
        B.c_steps[0] = R.steps;
        B.c_work[0] = R.work;
        B.c_flags[0] = CF_COL | CF_EXACT;
        B.c_thrf[0] = B.c_thrc[0] = B.c_E32[0] = 0.f;
        const V3 r0 = ld3(A.H.pos, goff);
        B.c_ref[0][0] = r0.x; B.c_ref[1][0] = r0.y; B.c_ref[2][0] = r0.z;
    }
#pragma unroll 1
    for (int p = tid; p < n0; p += BT) B.gslot[p] = goff + p;
    const int nf = min(*A.n_frags, A.frag_cap);
#pragma unroll 1
    for (int k = tid; k < nf; k += BT) {
        const FragRec &F = A.frags[k];
        if (F.cluster == c && F.seq >= 0 && n0 + F.seq < n) B.gslot[n0 + F.seq] = F.gslot;
    }
    __syncthreads();
#pragma unroll 1
    FOR_SLOTS(p) bundle_rejoin(A, B, p, 0);
    __syncthreads();
    bundle_restart<BCAP>(A);
    bundle_advance(A, B, n, true);
    return true;
}

// The clusters above a bundle's slots (the queue's tier 0), concurrently with
// k_hard_bundles: one CTA takes one at a time as a lone wide bundle, up to A.wide_cap
// bodies.  resume: after k_hard_bundles, the clusters whose fragments outgrew their
// bundle.  Same arithmetic, bit for bit, as every other form.
constexpr int WT = bundle_threads(BCAP_WIDE);  // threads of a wide CTA (it holds its SM)
__global__ void __launch_bounds__(WT, 1) k_hard_wide(const __grid_constant__ HardArgs A, int resume) {
    constexpr int BCAP = BCAP_WIDE;
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    __shared__ int q_sh;
    const int tid = threadIdx.x;
    const int todo = resume ? A.queue[4] : A.n_tier[0];
    bundle_init(B);
    for (int guard = 0; guard < (1 << 30); guard++) {
        if (tid == 0) q_sh = atomicAdd(&A.queue[resume ? 5 : 0], 1);
        __syncthreads();
        const int q = q_sh;
        __syncthreads();
        if (q >= todo) break;
        const int c = resume ? A.left[q] : A.order[q];
        const int n = A.cnt[c];
        if (resume) {
            if (!bundle_resume<BCAP>(A, c)) continue;
            if (B.any) bundle_retire<BCAP>(A);
        } else if (n > A.wide_cap) {  // k_hard_team's
            continue;
        } else {
            if (tid == 0) {
                B.ncl = 1;
                B.c_idx[0] = c;
                B.c_off[0] = 0;
                B.c_n[0] = n;
                B.c_flags[0] = 0;
                B.used = n;
                B.fresh_k = B.fresh_p = 0;
                B.any_dead = 0;
            }
            __syncthreads();
            bundle_load<BCAP>(A);
        }
        // bundle_step advances the cluster by one block step; it retires when done
        for (int it = 0; it < A.max_steps + 8 && B.ncl > 0; it++) {
            bundle_step(A, B);
            if (B.any) bundle_retire<BCAP>(A);
        }
        __syncthreads();
    }
    bundle_close(A, B);
}

// The clusters above A.wide_cap (in tier 0, with k_hard_wide's): one CTA takes one at a
// time in the one-cluster-per-CTA form.  Its pair loops are a thread a target, so it has
// 512 threads: 600 members 8.76 ms per block step in 256, 6.58 in 512.
constexpr int TEAM_T = 512;
__global__ void __launch_bounds__(TEAM_T, 1) k_hard_team(const __grid_constant__ HardArgs A) {
    __shared__ double red_d[TEAM_T / 32];
    __shared__ long long red_l[TEAM_T / 32];
    __shared__ int q_sh;
    const Team<TEAM_T> tm{(int)threadIdx.x, red_d, red_l};
    for (int guard = 0; guard < (1 << 30); guard++) {
        if (threadIdx.x == 0) q_sh = atomicAdd(&A.queue[6], 1);
        __syncthreads();
        const int q = q_sh;
        __syncthreads();
        if (q >= A.n_tier[0]) break;
        const int c = A.order[q];
        if (A.cnt[c] > A.wide_cap) run_cluster<TEAM_T>(A, c, tm);
    }
}

// bundles of BCAP member slots until the queue is empty; OCC CTAs per SM
template <int BCAP, int OCC>
__global__ void __launch_bounds__(bundle_threads(BCAP), OCC) k_hard_bundles(const __grid_constant__ HardArgs A) {
    BundleSmem<BCAP> &B = bundle_smem<BCAP>();
    bundle_init(B);
    __syncthreads();
    for (int guard = 0; guard < (1 << 30); guard++) {
        if (guard == 0 || B.any) {  // clusters have left (or none has come yet)
            if (threadIdx.x == 0) {
                B.fresh_k = B.ncl;
                B.fresh_p = B.used;
            }
            __syncthreads();
            bundle_refill<BCAP>(A);
            if (B.ncl == 0) break;
            if (B.fresh_k < B.ncl) bundle_load<BCAP>(A);
        }
        HP_MARK(HP_ADMIT);
        bundle_step(A, B);
        if (B.any) bundle_retire<BCAP>(A);
        HP_MARK(HP_RETIRE);
    }
    bundle_close(A, B);
}

#undef FOR_SLOTS
#undef FOR_CLUSTERS

}  // namespace p3t
