// Entropically smoothed F2M dual bound and its adjoint, for batches of
// instances (no counterpart in the reference, which solves the LP only).
//
// Graph: the union over points of each point's N nearest neighbours by FP32
// Euclidean distance c = sqrt(dx*dx + dy*dy) (round-to-nearest, no FMA), ties
// by index; node lists ascending in neighbour index.
//
// Bound: with z_e = (u_a + u_b - c_e)/tau and sigma the logistic function,
//   L(u) = 2 sum_v u_v - tau sum_e softplus(z_e),
// the dual of the entropy-smoothed fractional 2-matching LP, so L(u) bounds
// that LP from below for every u.  Forward: T damped Jacobi coordinate-ascent
// steps from u = 0 (s_v = root of sum_{e=(v,w)} sigma((s + u_w - c_e)/tau) = 2,
// u_v <- (1 - omega) u_v + omega s_v), then L(u^T).  Backward: the exact
// adjoint of those steps (implicit function theorem at each root), with the
// iterates recomputed from checkpoints every K steps instead of stored, then
// chained through c_e = |p_a - p_b| to the coordinates.  All dual arithmetic
// is FP64; coordinates and costs are FP32.
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "f2m_device.cuh"
#include "f2m_internal.h"

namespace f2m {

constexpr int kST = 512;  // threads of a solver CTA (one instance at a time)

__device__ __forceinline__ float sdist(float x0, float y0, float x1, float y1) {
    const float dx = __fsub_rn(x0, x1), dy = __fsub_rn(y0, y1);
    return __fsqrt_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)));
}

__device__ __forceinline__ int find_inst(const int64_t* offs, int n_inst, int64_t g) {
    int lo = 0, hi = n_inst - 1;  // last b with offs[b] <= g
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (offs[mid] <= g) lo = mid; else hi = mid - 1;
    }
    return lo;
}

/* ---------------- kNN: warp per point, brute force over its instance ---- */
// Sorts 64 keys ascending, elements l (a) and 32 + l (b) in lane l.
template <class T>
__device__ __forceinline__ void warp_sort64(T& a, T& b) {
    const int l = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 64; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j == 32) {
                if (b < a) { const T t = a; a = b; b = t; }
            } else {
                const T pa = __shfl_xor_sync(0xffffffffu, a, j), pb = __shfl_xor_sync(0xffffffffu, b, j);
                const bool low = (l & j) == 0;
                // (element 32 + l differs from l in bit 5 only, which decides the direction at k = 32)
                const bool ua = (l & k) == 0 || k == 64, ub = k == 32 ? false : ua;
                a = ((low == ua) == (pa < a)) ? pa : a;
                b = ((low == ub) == (pb < b)) ? pb : b;
            }
        }
    }
}
// Each warp finds its point's N smallest keys (cost bits << 32 | local index;
// the cost is non-negative, so the unsigned order is (cost, index)).
//
// N <= 32: a first scan keeps the two smallest costs of every lane; the N-th
// smallest of those 64 bounds the N-th smallest cost (a few ranks above it,
// as a lane seldom holds three of the first N), and a second scan collects
// what lies at or below it -- one sort instead of an insertion for each of the
// N ln(V / N) improvements (19 ms of insertions for 1,024 instances of 1,100
// points on average, N = 24).  More than 64 collected (ties), or fewer than N
// (NaN), take the insertion, as N > 32 does.
constexpr int kKnnBuf = 64;
__global__ void __launch_bounds__(256) k_sknn(SmoothBatch S) {
    __shared__ unsigned long long s_key[8][kKnnBuf];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t g = (int64_t)blockIdx.x * 8 + wid;
    if (g >= S.n_total) return;
    const int b = find_inst(S.offs, S.n_inst, g);
    const int64_t base = S.offs[b];
    const int V = (int)(S.offs[b + 1] - base);
    const int N = min(S.N, V - 1);
    const int i = (int)(g - base);
    const float xi = S.x[g], yi = S.y[g];
    const float* px = S.x + base;
    const float* py = S.y + base;
    unsigned long long A = ~0ull, Bk = ~0ull;
    bool insert = N > 32;
    if (!insert) {
        float m0 = INFINITY, m1 = INFINITY;
#pragma unroll 4
        for (int j = lane; j < V; j += 32) {
            const float c = j != i ? sdist(xi, yi, px[j], py[j]) : INFINITY;
            m1 = fminf(m1, fmaxf(m0, c));
            m0 = fminf(m0, c);
        }
        warp_sort64(m0, m1);
        const float bound = __shfl_sync(0xffffffffu, m0, N - 1);
        int cnt = 0;
        for (int j0 = 0; j0 < V; j0 += 32) {
            const int j = j0 + lane;
            const float c = j < V && j != i ? sdist(xi, yi, px[j], py[j]) : NAN;
            const unsigned m = __ballot_sync(0xffffffffu, c <= bound);
            const int at = cnt + __popc(m & ((1u << lane) - 1u));
            if (c <= bound && at < kKnnBuf) s_key[wid][at] = ((unsigned long long)__float_as_uint(c) << 32) | (unsigned)j;
            cnt += __popc(m);
        }
        __syncwarp();
        insert = cnt < N || cnt > kKnnBuf;
        if (!insert) {
            A = lane < cnt ? s_key[wid][lane] : ~0ull;
            Bk = 32 + lane < cnt ? s_key[wid][32 + lane] : ~0ull;
            warp_sort64(A, Bk);
        }
    }
    // insertion into a sorted list spread over two registers per lane
    // (elements l and 32 + l)
    unsigned long long thr = ~0ull;  // element N-1
    for (int j0 = 0; insert && j0 < V; j0 += 32) {
        const int j = j0 + lane;
        unsigned long long key = ~0ull;
        if (j < V && j != i) {
            const float c = sdist(xi, yi, px[j], py[j]);
            key = ((unsigned long long)__float_as_uint(c) << 32) | (unsigned)j;
        }
        unsigned m = __ballot_sync(0xffffffffu, key < thr);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const unsigned long long k = __shfl_sync(0xffffffffu, key, src);
            if (k >= thr) continue;
            const int pos = __popc(__ballot_sync(0xffffffffu, A < k)) +
                            __popc(__ballot_sync(0xffffffffu, Bk < k));
            const unsigned long long pa = __shfl_up_sync(0xffffffffu, A, 1);
            const unsigned long long pb = __shfl_up_sync(0xffffffffu, Bk, 1);
            const unsigned long long a31 = __shfl_sync(0xffffffffu, A, 31);
            const unsigned long long nA = lane < pos ? A : (lane == pos ? k : pa);
            const int hb = 32 + lane;
            const unsigned long long nB = hb < pos ? Bk : (hb == pos ? k : (lane == 0 ? a31 : pb));
            A = nA;
            Bk = nB;
            thr = (N - 1 < 32) ? __shfl_sync(0xffffffffu, A, N - 1) : __shfl_sync(0xffffffffu, Bk, N - 33);
        }
    }
    unsigned long long* out = S.top + g * S.N;
    if (lane < S.N) out[lane] = lane < N ? A : ~0ull;
    if (32 + lane < S.N) out[32 + lane] = 32 + lane < N ? Bk : ~0ull;
}

// reverse counts: rdeg[w] = number of points that keep w
__global__ void k_srdeg(SmoothBatch S) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= S.n_total * S.N) return;
    const unsigned long long k = S.top[t];
    if (k == ~0ull) return;
    const int64_t g = t / S.N;
    const int b = find_inst(S.offs, S.n_inst, g);
    atomicAdd(&S.rdeg[S.offs[b] + (unsigned)(k & 0xffffffffu)], 1);
}

__global__ void k_stcap(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= S.n_total) return;
    S.deg[g] = S.N + S.rdeg[g];
    S.tcur[g] = 0;
}

__global__ void k_sfill(SmoothBatch S) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= S.n_total * S.N) return;
    const int64_t g = t / S.N;
    const int k = (int)(t % S.N);
    const unsigned long long key = S.top[t];
    int32_t w = -1;
    if (key != ~0ull) w = (int32_t)(key & 0xffffffffu);
    S.tnbr[S.tcap[g] + k] = w;  // own list (-1 = none)
    if (w < 0) return;
    const int b = find_inst(S.offs, S.n_inst, g);
    const int64_t gw = S.offs[b] + w;
    const int p = atomicAdd(&S.tcur[gw], 1);
    S.tnbr[S.tcap[gw] + S.N + p] = (int32_t)(g - S.offs[b]);
}

// Sort each temporary list by neighbour, drop repeats and the -1 fillers, a warp
// a list: up to 64 entries in registers, longer ones in place by the same
// network with every comparison ascending (each merge starts with the mirrored
// partner), where the missing entries up to a power of two would stay put.  (500
// points, N = 48: 499 us with a thread a list in place, 627 through local memory,
// 20 so.)
__global__ void __launch_bounds__(128) k_ssort(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (g >= S.n_total) return;
    const int lane = threadIdx.x & 31;
    const unsigned before = (1u << lane) - 1u;
    int32_t* a = S.tnbr + S.tcap[g];
    const int n = S.N + S.rdeg[g];
    int m = 0, last = -1;  // entries kept, largest value so far
    auto pack = [&](int32_t v) {  // 32 sorted values
        int32_t prev = __shfl_up_sync(0xffffffffu, v, 1);
        if (lane == 0) prev = last;
        const bool keep = v != prev && v != INT_MAX;
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        if (keep) a[m + __popc(kept & before)] = v;
        m += __popc(kept);
        last = __shfl_sync(0xffffffffu, v, 31);
    };
    if (n <= 64) {
        int32_t v = lane < n ? a[lane] : INT_MAX, w = 32 + lane < n ? a[32 + lane] : INT_MAX;
        __syncwarp();
        warp_sort64(v, w);
        pack(v);
        pack(w);
    } else {
        for (int k = 2; k < 2 * n; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int t = lane; t < n; t += 32) {
                    const int u = j == k >> 1 ? t ^ (k - 1) : t ^ j;
                    if (u <= t || u >= n) continue;
                    const int32_t x = a[t], y = a[u];
                    if (y < x) { a[t] = y; a[u] = x; }
                }
                __syncwarp();
            }
        }
        for (int i = 0; i < n; i += 32) {
            const int32_t v = i + lane < n ? a[i + lane] : INT_MAX;
            __syncwarp();
            pack(v);
            __syncwarp();
        }
    }
    if (lane == 0) S.deg[g] = m;
}

__global__ void k_scopy(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= S.n_total) return;
    const int b = find_inst(S.offs, S.n_inst, g);
    const int64_t base = S.offs[b];
    const int32_t* a = S.tnbr + S.tcap[g];
    const int64_t r0 = S.row[g];
    const int n = (int)(S.row[g + 1] - r0);
    for (int k = 0; k < n; ++k) {
        const int32_t w = a[k];
        S.nbr[r0 + k] = w;
        S.c[r0 + k] = sdist(S.x[g], S.y[g], S.x[base + w], S.y[base + w]);
    }
}

__global__ void k_smirror(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= S.n_total) return;
    const int b = find_inst(S.offs, S.n_inst, g);
    const int64_t base = S.offs[b];
    const int32_t v = (int32_t)(g - base);
    for (int64_t k = S.row[g]; k < S.row[g + 1]; ++k) {
        const int64_t gw = base + S.nbr[k];
        int64_t lo = S.row[gw], hi = S.row[gw + 1] - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (S.nbr[mid] < v) lo = mid + 1; else hi = mid;
        }
        S.mirror[k] = lo;
    }
}

/* ---------------- lists by ascending cost -------------------------------- */
// A node root reads its list in ascending cost and stops early, so each list
// is stored a second time sorted by (cost, neighbour): splace holds each entry's
// place in the CSR row, the entries are the cost bits and the local neighbour.
// The persistent kernel, a lane to a node, reads the first S.W of them from slices
// of 32 nodes (sell), a column with unit stride: from the rows its reads touched
// a sector a lane (132 ms against 55 for the bound and gradient of 1,024 lattice
// instances).  An instance's last slice is as wide as its nodes, rounded up to
// whole sectors (sbase counts such places).  With four lanes or more to a node,
// the per-step kernels, the rows (sent) are sectors.
//
// A warp a node sorts up to 64 entries in registers; the few longer lists rank
// each entry among the others.  (500 points, N = 48: 170 us with a thread a list,
// 8 so.)
__global__ void __launch_bounds__(128) k_ssorted(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (g >= S.n_total) return;
    const int lane = threadIdx.x & 31;
    const int64_t r0 = S.row[g];
    const int n = (int)(S.row[g + 1] - r0);
    auto key_of = [&](int k) { return ((unsigned long long)__float_as_uint(S.c[r0 + k]) << 32) | (unsigned)k; };
    auto put = [&](int k, unsigned long long key) { S.splace[r0 + k] = (int)(unsigned)key; };
    // entries within reach of the first root (u = 0)
    auto reach_of = [&](unsigned third) { return __uint_as_float(third) + (float)(kReach * S.tau); };
    auto count = [&](int in) {
        if (lane != 0) return;
        unsigned long long* at = S.reach + blockIdx.x % kReachCounters;
        atomicAdd(at, (unsigned long long)in);
        if (in > 4 * kStepScratch) atomicAdd(at + kReachCounters, 1ull);
    };
    if (n <= 64) {
        unsigned long long a = lane < n ? key_of(lane) : ~0ull, b = 32 + lane < n ? key_of(32 + lane) : ~0ull;
        warp_sort64(a, b);
        if (lane < n) put(lane, a);
        if (32 + lane < n) put(32 + lane, b);
        if (S.reach) {
            const float lim = reach_of(__shfl_sync(0xffffffffu, (unsigned)(a >> 32), 2));
            auto in = [&](int k, unsigned long long key) {
                return __ballot_sync(0xffffffffu, k < n && __uint_as_float((unsigned)(key >> 32)) <= lim);
            };
            count(__popc(in(lane, a)) + __popc(in(32 + lane, b)));
        }
        return;
    }
    for (int k = lane; k < n; k += 32) {
        const unsigned long long x = key_of(k);
        int rank = 0;
        for (int j = 0; j < n; ++j) rank += key_of(j) < x;
        put(rank, x);
    }
    if (S.reach) {
        __syncwarp();
        const float lim = reach_of(__float_as_uint(S.c[r0 + S.splace[r0 + 2]]));
        int in = 0;
        for (int k = lane; k < n; k += 32) in += S.c[r0 + k] <= lim;
        count(__reduce_add_sync(0xffffffffu, in));
    }
}

// entry j of the list at r0 in ascending cost
__device__ __forceinline__ uint2 sorted_entry(const SmoothBatch& S, int64_t r0, int j) {
    const int64_t k = r0 + S.splace[r0 + j];
    return make_uint2(__float_as_uint(S.c[k]), (unsigned)S.nbr[k]);
}
// Where node v of an instance of V nodes, at place `base` of sbase, has its column
// of a slice, and the distance between its entries.
__device__ __forceinline__ int64_t slice_column(const SmoothBatch& S, int64_t base, int V, int v, int& stride) {
    const int s0 = v & ~31;
    stride = min(32, (V - s0 + 3) & ~3);
    return (base + s0) * S.W + (v - s0);
}
__global__ void __launch_bounds__(128) k_ssell(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= S.n_total) return;
    const int b = find_inst(S.offs, S.n_inst, g);
    int stride;
    uint2* out = S.sell + slice_column(S, S.sbase[b], (int)(S.offs[b + 1] - S.offs[b]), (int)(g - S.offs[b]), stride);
    const int64_t r0 = S.row[g];
    const int n = min(S.W, (int)(S.row[g + 1] - r0));
    for (int j = 0; j < n; ++j) out[(int64_t)stride * j] = sorted_entry(S, r0, j);
}
// the rows of the per-step kernels
__global__ void __launch_bounds__(128) k_ssent(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (g >= S.n_total) return;
    const int64_t r0 = S.row[g];
    const int n = (int)(S.row[g + 1] - r0);
    for (int j = threadIdx.x & 31; j < n; j += 32) S.sent[r0 + j] = sorted_entry(S, r0, j);
}

/* ---------------- node roots over the entries within reach --------------- */
__device__ __forceinline__ double sigm(double z) {
    if (z >= 0) return 1.0 / (1.0 + exp(-z));
    const double e = exp(z);
    return e / (1.0 + e);
}
__device__ __forceinline__ double softplus(double z) { return fmax(z, 0.0) + log1p(exp(-fabs(z))); }
// sigma(z) (1 - sigma(z)) without cancellation
__device__ __forceinline__ double dsig(double z) {
    const double e = exp(-fabs(z)), big = 1.0 / (1.0 + e);
    return e * big * big;
}

// sum_k sigma(z_k) - 2 without cancellation: each term splits into its
// rounding to 0 or 1 (counted exactly) and the remainder m = min(sigma,
// 1 - sigma) = e/(1+e), e = exp(-|z|), so the tiny residuals that place a
// root between two well-separated costs keep their relative precision.
struct LogitAcc {
    double cnt = 0, tail = 0, scale = 0, slope = 0;
    __device__ __forceinline__ void add(double z) {
        const double e = exp(-fabs(z));
        const double big = 1.0 / (1.0 + e), m = e * big;
        if (z >= 0) { cnt += 1.0; tail -= m; } else { tail += m; }
        scale += m;
        slope += m * big;
    }
};

// Newton's method for the root s of sum_k sigma((s - a_k)/tau) = 2 from the
// LP root (midpoint of the 2nd and 3rd smallest a_k), kept inside the bracket
// [smallest a_k - 40 tau, third smallest + 40 tau] by bisection; stops at a
// relative residual of 1e-14, a step below the resolution of s or a bracket
// of a few ulps.  `step` returns the next point, or NAN to stop.
__device__ __forceinline__ double root_step(const LogitAcc& r, double tau, double s, double& lo,
                                            double& hi) {
    const double g = (r.cnt - 2.0) + r.tail, gp = r.slope / tau;
    if (g > 0) hi = s; else lo = s;
    if (g == 0 || fabs(g) <= 1e-14 * r.scale) return NAN;
    double sn = (gp > 0) ? s - g / gp : 0.5 * (lo + hi);
    if (fabs(sn - s) <= 4e-16 * (1.0 + fabs(s))) return NAN;
    if (!(sn > lo && sn < hi)) sn = 0.5 * (lo + hi);
    if (sn == s || hi - lo <= 4e-16 * (1.0 + fabs(s))) return NAN;
    return sn;
}

// Which entries a root needs.  With m2 the third smallest a_k, the root is at
// most m2 + tau ln 2 (three sigmas of 2/3 there), and a Newton step is at most
// 2 tau long (a remainder's slope is at least half the remainder), so no point
// the sums are taken at lies above m2 + 3 tau.  An entry past m2 + kReach tau
// then adds less than e^-(kReach - 3) of what the third smallest adds to the
// scale of the residual: 64 of them stay below 3e-19 of it, where FP64 rounds
// at 1e-16.  They are left out; with tau at a hundredth of the point spacing
// three to five of some thirty entries remain.  Since a_k >= c_k - max u, the
// scan of the ascending costs ends at the first c_k above that bound.
constexpr int kBuf = kStepScratch;

// A group of G lanes holds a node, lane l its entries l, l + G, ...: the lanes'
// reads of a column fill sectors, their exponentials run side by side, and sums
// and selections take log2 G shuffles.  Every lane of a warp takes part in the
// shuffles; a group without a node has an empty list.
// One lane's part of a list: get(j) its j-th entry, acc(j) where its share of
// dL/dc is summed; n entries.
template <int G>
struct RowPart {
    int n, deg;
    const uint2* ent;
    double* gs;
    __device__ __forceinline__ uint2 get(int j) const { return ent[j * G]; }
    __device__ __forceinline__ double& acc(int j) const { return gs[j * G]; }
};
struct SInst {
    int b, V;
    int64_t base, w0;    // first node, first place of its slices
    const int64_t* row;  // row + base
};
// a node alone (G = 1): its column, and past W its CSR row
struct SlicePart {
    int n, deg, W, stride;
    const uint2* col;
    double* gcol;
    const SmoothBatch* S;
    int64_t r0;
    __device__ __forceinline__ uint2 get(int j) const { return j < W ? col[stride * j] : sorted_entry(*S, r0, j); }
    __device__ __forceinline__ double& acc(int j) const {
        return j < W ? gcol[stride * j] : S->gc[r0 + S->splace[r0 + j]];
    }
};
// of node v of the instance that starts at node `base` (no entries: in = false)
template <int G>
__device__ __forceinline__ RowPart<G> row_part(const SmoothBatch& S, int64_t base, int v, bool in) {
    RowPart<G> p{0, 0, nullptr, nullptr};
    if (in) {
        const int l = threadIdx.x % G;
        const int64_t r0 = S.row[base + v];
        p.deg = (int)(S.row[base + v + 1] - r0);
        p.n = (p.deg - l + G - 1) / G;
        p.ent = S.sent + r0 + l;
        p.gs = S.gs + r0 + l;
    }
    return p;
}
__device__ __forceinline__ SlicePart slice_part(const SmoothBatch& S, const SInst& I, int v, bool in) {
    SlicePart p{0, 0, S.W, 0, nullptr, nullptr, &S, 0};
    if (in) {
        p.r0 = I.row[v];
        p.n = p.deg = (int)(I.row[v + 1] - p.r0);
        const int64_t at = slice_column(S, I.w0, I.V, v, p.stride);
        p.col = S.sell + at;
        p.gcol = S.gsell + at;
    }
    return p;
}
template <int G>
__device__ __forceinline__ double grp_sum(double x) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
// the three smallest of two sorted triples
__device__ __forceinline__ void low3_merge(double& m0, double& m1, double& m2, double p0, double p1, double p2) {
    const double n0 = dmin2(m0, p0);
    const double n1 = dmin2(dmin2(m1, p1), dmax2(m0, p0));
    m2 = dmin2(dmin2(m2, p2), dmin2(dmax2(m1, p0), dmax2(m0, p1)));
    m0 = n0;
    m1 = n1;
}
template <int G>
__device__ __forceinline__ void grp_low3(double& m0, double& m1, double& m2) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)
        low3_merge(m0, m1, m2, __shfl_xor_sync(0xffffffffu, m0, o), __shfl_xor_sync(0xffffffffu, m1, o),
                   __shfl_xor_sync(0xffffffffu, m2, o));
}

// Scratch of one lane: up to cap values and their 16-bit indices, strided so
// that a warp's accesses do not conflict.
struct SBuf {
    double* x;
    uint16_t* i;
    int stride, cap;
    __device__ __forceinline__ void push(int& cnt, double v, int k) const {
        if (cnt < cap) { x[cnt * stride] = v; i[cnt * stride] = (uint16_t)k; }
        ++cnt;
    }
};

// Max of the lanes' x into *slot, as an ordered integer.
__device__ __forceinline__ long long ord_of(double x) {
    const long long i = __double_as_longlong(x);
    return i ^ ((i >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double ord_to(long long i) {
    return __longlong_as_double(i ^ ((i >> 63) & 0x7fffffffffffffffll));
}
constexpr long long kOrdLow = -0x7ff0000000000001ll;  // ord_of(-inf)
__device__ __forceinline__ void warp_ord_max(double x, long long* slot) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
    if ((threadIdx.x & 31) == 0) atomicMax(slot, ord_of(x));
}

// Terms of the sums: list entries they cover, and those taken (an exponential
// each; the others are out of reach).
struct STerms {
    unsigned long long covered = 0, taken = 0;
};
// The root of a node given the potentials u and a bound umax >= every u; *thr
// receives m2 + kReach tau.
template <int G, class List, class UP>
__device__ __forceinline__ double node_root(const SmoothBatch& S, const List& L, UP u, double umax, const SBuf& B,
                                            double* thr, STerms& terms) {
    constexpr int C = G >= 8 ? 2 : 4;  // columns read at once
    const bool lead = threadIdx.x % G == 0;
    const double win = kReach * S.tau;
    auto cost = [&](const uint2& e) { return (double)__uint_as_float(e.x); };
    double m0 = INFINITY, m1 = INFINITY, m2 = INFINITY;  // of this lane's entries so far
    double bound = INFINITY;                             // at least m2 of the node + win
    int cnt = 0, end = 0;
    while (end < L.n) {
        uint2 e[C];
        double a[C];
#pragma unroll
        for (int i = 0; i < C; ++i) e[i] = end + i < L.n ? L.get(end + i) : make_uint2(0x7f800000u, 0u);
#pragma unroll
        for (int i = 0; i < C; ++i) a[i] = cost(e[i]) - u[e[i].y];
#pragma unroll
        for (int i = 0; i < C; ++i) {
            top3_insert(a[i], m0, m1, m2);
            bound = dmin2(bound, m2 + win);
            if (a[i] <= bound && end + i < L.n) B.push(cnt, a[i], end + i);
        }
        end = min(end + C, L.n);
        if (cost(e[C - 1]) - umax > bound) break;
    }
    __syncwarp();
    if (G > 1) grp_low3<G>(m0, m1, m2);
    const double t = m2 + win;
    *thr = t;
    double lo = m0 - 40 * S.tau, hi = m2 + 40 * S.tau;
    double s = 0.5 * (m1 + m2);
    bool go = L.deg > 0;
    for (int it = 0; it < S.newton_max; ++it) {
        LogitAcc r;
        if (go) {
            if (lead) terms.covered += L.deg;
            terms.taken += cnt;
            if (cnt <= B.cap) {
                #pragma unroll 2
                for (int j = 0; j < cnt; ++j) r.add((s - B.x[j * B.stride]) * S.inv_tau);
            } else {
                for (int j = 0; j < end; j += 4) {  // four at a time, their loads and sums side by side
                    double z[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint2 e = j + i < end ? L.get(j + i) : make_uint2(0x7f800000u, 0u);
                        const double a = cost(e) - u[e.y];
                        z[i] = a <= t ? (s - a) * S.inv_tau : -INFINITY;  // adds nothing
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) r.add(z[i]);
                }
            }
        }
        if (G > 1) {
            __syncwarp();
            r.cnt = grp_sum<G>(r.cnt);
            r.tail = grp_sum<G>(r.tail);
            r.scale = grp_sum<G>(r.scale);
            r.slope = grp_sum<G>(r.slope);
        }
        if (go) {
            const double sn = root_step(r, S.tau, s, lo, hi);
            if (sn != sn) go = false;
            else s = sn;
        }
        if (G > 1 ? !__any_sync(0xffffffffu, go) : !go) break;
    }
    return s;
}

// Reverse pass 1 of one step: mu_v = omega lam_v / D_v with D_v = sum p_e over
// the entries within reach (p falls off as the remainders do), and
// q_e = mu_v p_e added to the node's share of dL/dc.
template <int G, class List, class UP>
__device__ __forceinline__ double node_rev1(const SmoothBatch& S, const List& L, UP u, double umax, const SBuf& B,
                                            double s, double thr, double lam, STerms& terms) {
    constexpr int C = G >= 8 ? 2 : 4;
    int cnt = 0, end = 0;
    while (end < L.n) {
        uint2 e[C];
#pragma unroll
        for (int i = 0; i < C; ++i) e[i] = end + i < L.n ? L.get(end + i) : make_uint2(0x7f800000u, 0u);
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const double a = (double)__uint_as_float(e[i].x) - u[e[i].y];
            if (a <= thr && end + i < L.n) B.push(cnt, a, end + i);
        }
        end = min(end + C, L.n);
        if ((double)__uint_as_float(e[C - 1].x) - umax > thr) break;
    }
    if (threadIdx.x % G == 0) terms.covered += L.deg;
    terms.taken += cnt;
    double D = 0.0;
    auto p_of = [&](double a) { return dsig((s - a) * S.inv_tau) * S.inv_tau; };
    auto each = [&](auto f) {  // entries within reach, re-read
        for (int j = 0; j < end; ++j) {
            const uint2 e = L.get(j);
            const double a = (double)__uint_as_float(e.x) - u[e.y];
            if (a <= thr) f(j, a);
        }
    };
    if (cnt <= B.cap) {
        for (int j = 0; j < cnt; ++j) {
            const double p = p_of(B.x[j * B.stride]);
            B.x[j * B.stride] = p;
            D += p;
        }
    } else {
        each([&](int, double a) { D += p_of(a); });
    }
    __syncwarp();
    D = grp_sum<G>(D);
    const double mu = D > 0 ? S.omega * lam / D : 0.0;  // D == 0: all saturated
    if (cnt <= B.cap) {
        for (int j = 0; j < cnt; ++j) L.acc(B.i[j * B.stride]) += mu * B.x[j * B.stride];
    } else {
        each([&](int j, double a) { L.acc(j) += mu * p_of(a); });
    }
    return mu;
}
// Reverse pass 2: what the neighbours v that hold node w within their reach
// (a = c - u_w at most thr_v) take from lam_w: the sum of mu_v p over them, p
// formed from the same operands as in pass 1, so q need not be stored.
template <int G, class List, class TP, class SP, class MP>
__device__ __forceinline__ double node_rev2(const SmoothBatch& S, const List& L, double uw, double thrmax, TP thr,
                                            SP s, MP mu, const SBuf& B, STerms& terms) {
    constexpr int C = G >= 8 ? 2 : 4;
    int cnt = 0, end = 0;
    while (end < L.n) {
        uint2 e[C];
#pragma unroll
        for (int i = 0; i < C; ++i) e[i] = end + i < L.n ? L.get(end + i) : make_uint2(0x7f800000u, 0u);
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const double a = (double)__uint_as_float(e[i].x) - uw;
            if (end + i < L.n && a <= thr[e[i].y]) B.push(cnt, a, (int)e[i].y);
        }
        end = min(end + C, L.n);
        if ((double)__uint_as_float(e[C - 1].x) - uw > thrmax) break;
    }
    terms.taken += cnt;
    double sum = 0.0;
    auto q_of = [&](int v, double a) { return mu[v] * (dsig((s[v] - a) * S.inv_tau) * S.inv_tau); };
    if (cnt <= B.cap) {
        for (int j = 0; j < cnt; ++j) sum += q_of(B.i[j * B.stride], B.x[j * B.stride]);
    } else {
        for (int j = 0; j < end; ++j) {
            const uint2 e = L.get(j);
            const double a = (double)__uint_as_float(e.x) - uw;
            if (a <= thr[e.y]) sum += q_of((int)e.y, a);
        }
    }
    __syncwarp();
    return grp_sum<G>(sum);
}

/* ---------------- the bound and its adjoint: one CTA per instance ------- */

// One damped Jacobi step u -> un; writes the roots and the reach bounds when
// given, and the largest new potential into *umax_next.
__device__ __forceinline__ void sjacobi(const SmoothBatch& S, const SInst& I, const double* u, double* un,
                                        double* s_out, double* t_out, const SBuf& B, double umax,
                                        long long* umax_next, STerms& terms) {
    double mx = -INFINITY;
    const int v1 = (I.V + 31) & ~31;  // whole warps
    for (int v = threadIdx.x; v < v1; v += kST) {
        const auto nd = slice_part(S, I, v, v < I.V);
        double thr;
        const double s = node_root<1>(S, nd, u, umax, B, &thr, terms);
        if (v < I.V) {
            if (s_out) { s_out[v] = s; t_out[v] = thr; }
            const double x = (1.0 - S.omega) * u[v] + S.omega * s;
            un[v] = x;
            mx = fmax(mx, x);
        }
        __syncwarp();
    }
    warp_ord_max(mx, umax_next);
}

__device__ double sbound(const SmoothBatch& S, const SInst& I, const double* u, double* sred,
                         STerms& terms) {
    double su = 0.0, sp = 0.0;
    for (int v = threadIdx.x; v < I.V; v += kST) {
        su += 2.0 * u[v];
        for (int64_t k = I.row[v]; k < I.row[v + 1]; ++k) {
            const int w = S.nbr[k];
            if (w > v) { sp += softplus((u[v] + u[w] - (double)S.c[k]) / S.tau); ++terms.covered; ++terms.taken; }
        }
    }
    su = block_sum<kST>(su, sred);
    sp = block_sum<kST>(sp, sred);
    return su - S.tau * sp;
}

// What bounds it: the scans of the list heads (a column read, a gathered
// potential and the top-3 insertion an entry) and the few exponentials a root
// needs, and for the last instances of a batch the latency of their 300
// dependent passes.  Two 512-thread CTAs an SM: 40.9 ms for 1,024 lattice
// instances of 200-2,000 points (N = 24, tau 1e-3, 100 steps, gradient), 49.7
// with four of 256 threads, 47.1 with one of 1,024; 347 ms with a thread per
// node over the whole CSR row, an exponential and two divisions an entry.
template <bool GRAD>
__global__ void __launch_bounds__(kST, 2) k_sbound(SmoothBatch S, int cap, int max_v) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double sred[kST / 32];
    __shared__ int sitem;
    __shared__ long long smax[3], stmax[2];  // largest potential (three steps), largest reach bound
    double* Ha = reinterpret_cast<double*>(smem_raw);
    double* bx = Ha + 2 * (size_t)max_v;
    const SBuf B{bx + threadIdx.x, reinterpret_cast<uint16_t*>(bx + (size_t)cap * kST) + threadIdx.x, kST, cap};
    // terms of this thread's sums (Newton sums, softplus, sigma,
    // sigma'), added to S.work when the queue is empty
    STerms terms;
    for (;;) {
        if (threadIdx.x == 0) sitem = atomicAdd(S.queue, 1);
        __syncthreads();
        const int item = sitem;
        __syncthreads();
        if (item >= S.n_inst) {
            if (S.work) {
                if (terms.covered) atomicAdd(S.work, terms.covered);
                if (terms.taken) atomicAdd(S.work + 1, terms.taken);
            }
            return;
        }
        SInst I;
        I.b = S.order[item];
        I.base = S.offs[I.b];
        I.V = (int)(S.offs[I.b + 1] - I.base);
        I.row = S.row + I.base;
        I.w0 = S.sbase[I.b];
        const int v1 = (I.V + 31) & ~31;
        double* Hb = Ha + max_v;
        const int T = S.iters, K = S.ckpt;
        double* ck = S.ck + I.base * S.n_ck;
        for (int v = threadIdx.x; v < I.V; v += kST) Ha[v] = 0.0;
        if (threadIdx.x == 0) { smax[0] = ord_of(0.0); smax[1] = smax[2] = kOrdLow; }
        __syncthreads();
        double* u = Ha;
        double* un = Hb;
        for (int t = 0; t < T; ++t) {
            if (GRAD && t % K == 0)
                for (int v = threadIdx.x; v < I.V; v += kST) ck[(t / K) * I.V + v] = u[v];
            if (threadIdx.x == 0) smax[(t + 2) % 3] = kOrdLow;
            sjacobi(S, I, u, un, nullptr, nullptr, B, ord_to(smax[t % 3]), &smax[(t + 1) % 3], terms);
            __syncthreads();
            double* tt = u; u = un; un = tt;
        }
        const double L = sbound(S, I, u, sred, terms);
        if (threadIdx.x == 0) S.L[I.b] = L;
        if (!GRAD) { __syncthreads(); continue; }
        // adjoint of L(u^T) with respect to u^T and (explicitly) c; the
        // explicit sigma_e is split evenly over the edge's two slots
        const double up = S.dL[I.b];
        double* lam = S.lam + I.base;
        double* lam2 = S.lam2 + I.base;
        double* mu = S.mu + I.base;
        for (int v = threadIdx.x; v < I.V; v += kST) {
            LogitAcc r;
            for (int64_t k = I.row[v]; k < I.row[v + 1]; ++k) {
                const double z = (u[v] + u[S.nbr[k]] - (double)S.c[k]) / S.tau;
                r.add(z);
                S.gc[k] = up * (0.5 * sigm(z));
                terms.covered += 2;
                terms.taken += 2;
            }
            lam[v] = up * (-((r.cnt - 2.0) + r.tail));  // 2 - sum sigma
        }
        __syncthreads();
        double* su_ = S.segu + I.base * K;
        double* ss_ = S.segs + I.base * K;
        double* st_ = S.segt + I.base * K;
        double* sm_ = S.segm + (int64_t)I.b * K;  // largest potential of each stored iterate
        const int nseg = (T + K - 1) / K;
        for (int seg = nseg - 1; seg >= 0; --seg) {
            const int t0 = seg * K, t1 = min(T, t0 + K);
            if (threadIdx.x == 0) smax[0] = smax[1] = smax[2] = kOrdLow;
            __syncthreads();
            double mx = -INFINITY;
            for (int v = threadIdx.x; v < I.V; v += kST) {
                const double x = ck[seg * I.V + v];
                Ha[v] = x;
                mx = fmax(mx, x);
            }
            warp_ord_max(mx, &smax[0]);
            __syncthreads();
            u = Ha;
            un = Hb;
            for (int t = t0; t < t1; ++t) {  // recompute the segment's iterates
                const int j = t - t0;
                double* ut = su_ + (int64_t)j * I.V;
                for (int v = threadIdx.x; v < I.V; v += kST) ut[v] = u[v];
                if (threadIdx.x == 0) { smax[(j + 2) % 3] = kOrdLow; sm_[j] = ord_to(smax[j % 3]); }
                sjacobi(S, I, u, un, ss_ + (int64_t)j * I.V, st_ + (int64_t)j * I.V, B, ord_to(smax[j % 3]),
                        &smax[(j + 1) % 3], terms);
                __syncthreads();
                double* tt = u; u = un; un = tt;
            }
            for (int t = t1 - 1; t >= t0; --t) {
                const int j = t - t0;
                const double* ut = su_ + (int64_t)j * I.V;
                const double* st = ss_ + (int64_t)j * I.V;
                const double* tv = st_ + (int64_t)j * I.V;
                if (threadIdx.x == 0) stmax[t & 1] = kOrdLow;
                __syncthreads();
                // the iterate and its reach bounds in shared memory
                double tm = -INFINITY;
                for (int v = threadIdx.x; v < I.V; v += kST) {
                    Ha[v] = ut[v];
                    const double x = tv[v];
                    Hb[v] = x;
                    tm = fmax(tm, x);
                }
                warp_ord_max(tm, &stmax[t & 1]);
                __syncthreads();
                const double umax = sm_[j], thrmax = ord_to(stmax[t & 1]);
                for (int v = threadIdx.x; v < v1; v += kST) {
                    const bool in = v < I.V;
                    const auto nd = slice_part(S, I, v, in);
                    const double m = node_rev1<1>(S, nd, (const double*)Ha, umax, B, in ? st[v] : 0.0,
                                                    in ? Hb[v] : 0.0, in ? lam[v] : 0.0, terms);
                    if (in) mu[v] = m;
                    __syncwarp();
                }
                __syncthreads();
                for (int v = threadIdx.x; v < v1; v += kST) {
                    const bool in = v < I.V;
                    const auto nd = slice_part(S, I, v, in);
                    const double x = node_rev2<1>(S, nd, in ? Ha[v] : 0.0, thrmax, (const double*)Hb, st,
                                                    (const double*)mu, B, terms);
                    if (in) lam2[v] = (1.0 - S.omega) * lam[v] - x;
                    __syncwarp();
                }
                __syncthreads();
                double* tt = lam; lam = lam2; lam2 = tt;
            }
        }
    }
}

/* ---------------- one launch per step, all instances --------------------- */
// G lanes per node, each instance's nodes from a whole warp on (sbase counts
// warps); the potentials stay in global memory.
constexpr int kWT = 128;  // threads of a CTA
template <int kWG>
struct SThread {
    RowPart<kWG> nd;
    int b;
    int64_t g, base;
    bool in, lead;
};
template <int kWG>
__device__ __forceinline__ bool step_thread(const SmoothBatch& S, SThread<kWG>& t) {
    const int64_t w = (int64_t)blockIdx.x * (kWT / 32) + (threadIdx.x >> 5);
    if (w >= S.n_warps) return false;
    t.b = find_inst(S.sbase, S.n_inst, w);
    t.base = S.offs[t.b];
    const int v = (int)(w - S.sbase[t.b]) * (32 / kWG) + (threadIdx.x & 31) / kWG;
    t.g = t.base + v;
    t.in = t.g < S.offs[t.b + 1];
    t.lead = t.in && threadIdx.x % kWG == 0;
    t.nd = row_part<kWG>(S, t.base, v, t.in);
    return true;
}
#define F2M_SBUF                                                         \
    __shared__ double s_bx[kBuf * kWT];                                  \
    __shared__ uint16_t s_bi[kBuf * kWT];                                \
    const SBuf B{s_bx + threadIdx.x, s_bi + threadIdx.x, kWT, kBuf}

// u -> un for every node; stores u (ust), the roots (sst) and the reach bounds
// (tst) when given, and checkpoints u at index ck (>= 0).  umax / umax_next:
// the largest potential of each instance, before and after.
template <int kWG>
__global__ void __launch_bounds__(kWT) k_sw_step(SmoothBatch S, const double* u, double* un, double* ust, double* sst,
                                                 double* tst, int ck, const long long* umax, long long* umax_next) {
    F2M_SBUF;
    SThread<kWG> t;
    if (!step_thread(S, t)) return;
    double mx = -INFINITY, thr;
    STerms terms;
    const double s = node_root<kWG>(S, t.nd, u + t.base, ord_to(umax[t.b]), B, &thr, terms);
    if (t.lead) {
        const int64_t g = t.g;
        const double uv = u[g];
        if (ck >= 0) S.ck[(int64_t)ck * S.n_total + g] = uv;
        if (ust) ust[g] = uv;
        if (sst) { sst[g] = s; tst[g] = thr; }
        mx = (1.0 - S.omega) * uv + S.omega * s;
        un[g] = mx;
    }
    __syncwarp();
    warp_ord_max(mx, umax_next + t.b);
}

// u = 0 (ck < 0) or a checkpoint, and its largest value per instance
template <int kWG>
__global__ void __launch_bounds__(kWT) k_sw_init(SmoothBatch S, double* u, int ck, long long* umax) {
    SThread<kWG> t;
    if (!step_thread(S, t)) return;
    double x = -INFINITY;
    if (t.lead) {
        x = ck < 0 ? 0.0 : S.ck[(int64_t)ck * S.n_total + t.g];
        u[t.g] = x;
    }
    __syncwarp();
    warp_ord_max(x, umax + t.b);
}
// the per-instance maxima of every step, reset
__global__ void k_sw_low(long long* m, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) m[i] = kOrdLow;
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
struct WNode {
    int64_t g, base, r0;
    int n;
};
__device__ __forceinline__ bool warp_node(const SmoothBatch& S, WNode& W) {
    W.g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (W.g >= S.n_total) return false;
    const int b = find_inst(S.offs, S.n_inst, W.g);
    W.base = S.offs[b];
    W.r0 = S.row[W.g];
    W.n = (int)(S.row[W.g + 1] - W.r0);
    return true;
}

// per-node terms of L(u^T) and, for the adjoint, lambda^T and the explicit
// dL/dc (sigma_e split over the edge's two slots)
template <bool GRAD>
__global__ void __launch_bounds__(256) k_sw_final(SmoothBatch S, const double* u) {
    WNode W;
    if (!warp_node(S, W)) return;
    const int lane = threadIdx.x & 31;
    const int b = find_inst(S.offs, S.n_inst, W.g);
    const double up = GRAD ? S.dL[b] : 0.0;
    const int v = (int)(W.g - W.base);
    double sp = 0.0;
    LogitAcc r;
    for (int k = lane; k < W.n; k += 32) {
        const int w = S.nbr[W.r0 + k];
        const double z = (u[W.g] + u[W.base + w] - (double)S.c[W.r0 + k]) / S.tau;
        if (w > v) sp += softplus(z);
        if (GRAD) {
            r.add(z);
            S.gc[W.r0 + k] = up * (0.5 * sigm(z));
        }
    }
    sp = warp_sum(sp);
    if (GRAD) {
        r.cnt = warp_sum(r.cnt);
        r.tail = warp_sum(r.tail);
    }
    if (lane == 0) {
        S.Lp[W.g] = 2.0 * u[W.g] - S.tau * sp;
        if (GRAD) S.lam[W.g] = up * (-((r.cnt - 2.0) + r.tail));  // 2 - sum sigma
    }
}

__global__ void __launch_bounds__(256) k_sw_sumL(SmoothBatch S) {
    __shared__ double sred[8];
    const int b = blockIdx.x;
    double x = 0.0;
    for (int64_t g = S.offs[b] + threadIdx.x; g < S.offs[b + 1]; g += 256) x += S.Lp[g];
    x = block_sum<256>(x, sred);
    if (threadIdx.x == 0) S.L[b] = x;
}

template <int kWG>
__global__ void __launch_bounds__(kWT) k_sw_rev1(SmoothBatch S, const double* ut, const double* st, const double* tv,
                                                 const double* lam, const long long* umax, long long* thrmax) {
    F2M_SBUF;
    SThread<kWG> t;
    if (!step_thread(S, t)) return;
    STerms terms;
    const double thr = t.in ? tv[t.g] : -INFINITY;
    const double mu = node_rev1<kWG>(S, t.nd, ut + t.base, ord_to(umax[t.b]), B, t.in ? st[t.g] : 0.0, thr,
                                     t.in ? lam[t.g] : 0.0, terms);
    if (t.lead) S.mu[t.g] = mu;
    __syncwarp();
    warp_ord_max(thr, thrmax + t.b);
}

template <int kWG>
__global__ void __launch_bounds__(kWT) k_sw_rev2(SmoothBatch S, const double* ut, const double* st, const double* tv,
                                                 const double* lam, double* lam2, const long long* thrmax) {
    F2M_SBUF;
    SThread<kWG> t;
    if (!step_thread(S, t)) return;
    STerms terms;
    const double x = node_rev2<kWG>(S, t.nd, t.in ? ut[t.g] : 0.0, ord_to(thrmax[t.b]), tv + t.base, st + t.base,
                                    (const double*)S.mu + t.base, B, terms);
    if (t.lead) lam2[t.g] = (1.0 - S.omega) * lam[t.g] - x;
}

// the steps' shares of dL/dc added to the slots (the persistent kernel adds those
// past its slices itself)
__global__ void __launch_bounds__(128) k_s_merge(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= S.n_total) return;
    const int64_t r0 = S.row[g];
    const int n = (int)(S.row[g + 1] - r0);
    if (!S.W) {
        for (int k = 0; k < n; ++k) S.gc[r0 + S.splace[r0 + k]] += S.gs[r0 + k];
        return;
    }
    const int b = find_inst(S.offs, S.n_inst, g);
    int stride;
    const double* col =
        S.gsell + slice_column(S, S.sbase[b], (int)(S.offs[b + 1] - S.offs[b]), (int)(g - S.offs[b]), stride);
    for (int k = 0; k < min(n, S.W); ++k) S.gc[r0 + S.splace[r0 + k]] += col[(int64_t)stride * k];
}

__global__ void k_sw_coord(SmoothBatch S) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= S.n_total) return;
    const int b = find_inst(S.offs, S.n_inst, g);
    const int64_t base = S.offs[b];
    const double xv = S.x[g], yv = S.y[g];
    double gx = 0.0, gy = 0.0;
    for (int64_t k = S.row[g]; k < S.row[g + 1]; ++k) {
        const double ce = (double)S.c[k];
        if (ce == 0.0) continue;
        const int64_t gw = base + S.nbr[k];
        const double dc = S.gc[k] + S.gc[S.mirror[k]];
        gx += dc * (xv - (double)S.x[gw]) / ce;
        gy += dc * (yv - (double)S.y[gw]) / ce;
    }
    S.gx[g] = (float)gx;
    S.gy[g] = (float)gy;
}

/* ---------------- host launchers ---------------------------------------- */
static unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

cudaError_t launch_smooth_graph(SmoothBatch& S, int64_t* scan_scratch, cudaStream_t s,
                                int64_t* launches) {
    cudaError_t e;
    const int64_t nN = S.n_total * S.N;
    if ((e = cudaMemsetAsync(S.rdeg, 0, sizeof(int32_t) * S.n_total, s)) != cudaSuccess) return e;
    if (S.reach && (e = cudaMemsetAsync(S.reach, 0, sizeof(unsigned long long) * 2 * kReachCounters, s)) != cudaSuccess) return e;
    k_sknn<<<nblk(S.n_total, 8), 256, 0, s>>>(S);
    k_srdeg<<<nblk(nN, 256), 256, 0, s>>>(S);
    k_stcap<<<nblk(S.n_total, 256), 256, 0, s>>>(S);
    *launches += 3;
    if ((e = launch_scan(S.deg, S.tcap, S.n_total, scan_scratch, s, launches)) != cudaSuccess) return e;
    k_sfill<<<nblk(nN, 256), 256, 0, s>>>(S);
    k_ssort<<<nblk(S.n_total, 4), 128, 0, s>>>(S);
    *launches += 2;
    if ((e = launch_scan(S.deg, S.row, S.n_total, scan_scratch, s, launches)) != cudaSuccess) return e;
    k_scopy<<<nblk(S.n_total, 128), 128, 0, s>>>(S);
    k_ssorted<<<nblk(S.n_total, 4), 128, 0, s>>>(S);
    *launches += 3;
    return cudaGetLastError();
}
// The sorted entries, in slices or rows as the path reads them.
cudaError_t launch_smooth_entries(SmoothBatch& S, cudaStream_t s, int64_t* launches) {
    if (S.W) k_ssell<<<nblk(S.n_total, 128), 128, 0, s>>>(S);
    else k_ssent<<<nblk(S.n_total, 4), 128, 0, s>>>(S);
    ++*launches;
    return cudaGetLastError();
}
// Zeroes the sums of the reverse steps.
static cudaError_t clear_smooth_sums(const SmoothBatch& S, cudaStream_t s) {
    return S.W ? cudaMemsetAsync(S.gsell, 0, sizeof(double) * S.n_warps * S.W, s)
               : cudaMemsetAsync(S.gs, 0, sizeof(double) * S.s_cap, s);
}
// dL/dc of every slot, then the coordinates
static cudaError_t launch_smooth_coord(const SmoothBatch& S, cudaStream_t s, int64_t* launches) {
    k_s_merge<<<nblk(S.n_total, 128), 128, 0, s>>>(S);
    k_smirror<<<nblk(S.n_total, 128), 128, 0, s>>>(S);  // (over the steps' shares, merged now)
    k_sw_coord<<<nblk(S.n_total, 256), 256, 0, s>>>(S);
    *launches += 3;
    return cudaGetLastError();
}

template <int G>
static cudaError_t launch_steps_of(SmoothBatch& S, bool grad, cudaStream_t s, int64_t* launches) {
    const int64_t n = S.n_total;
    const unsigned gw = nblk(n, 8), gs = nblk(S.n_warps, kWT / 32);
    const int T = S.iters, K = S.ckpt;
    double* u = S.ua;
    double* un = S.ub;
    // the largest potentials of each instance: iterate t of the forward pass at
    // t, of a segment's recomputation at T + 1 + t, then the reach bounds
    auto um = [&](int64_t t) { return S.umax + t * S.n_inst; };
    const int64_t rows = (grad ? 3 : 1) * (int64_t)(T + 1) + 1;
    k_sw_low<<<nblk(rows * S.n_inst, 256), 256, 0, s>>>(S.umax, rows * S.n_inst);
    k_sw_init<G><<<gs, kWT, 0, s>>>(S, u, -1, um(0));
    *launches += 2;
    for (int t = 0; t < T; ++t) {
        k_sw_step<G><<<gs, kWT, 0, s>>>(S, u, un, nullptr, nullptr, nullptr, (grad && t % K == 0) ? t / K : -1, um(t),
                                     um(t + 1));
        double* tt = u; u = un; un = tt;
    }
    if (grad) k_sw_final<true><<<gw, 256, 0, s>>>(S, u);
    else k_sw_final<false><<<gw, 256, 0, s>>>(S, u);
    k_sw_sumL<<<S.n_inst, 256, 0, s>>>(S);
    *launches += T + 2;
    if (!grad) return cudaGetLastError();
    cudaError_t e = clear_smooth_sums(S, s);
    if (e != cudaSuccess) return e;
    double* lam = S.lam;
    double* lam2 = S.lam2;
    for (int seg = (T + K - 1) / K - 1; seg >= 0; --seg) {
        const int t0 = seg * K, t1 = min(T, t0 + K);
        u = S.ua;
        un = S.ub;
        k_sw_init<G><<<gs, kWT, 0, s>>>(S, u, seg, um(T + 1 + t0));
        for (int t = t0; t < t1; ++t) {
            // (the last step of a segment has no reader; its maximum goes to the spare row)
            k_sw_step<G><<<gs, kWT, 0, s>>>(S, u, un, S.segu + (int64_t)(t - t0) * n, S.segs + (int64_t)(t - t0) * n,
                                         S.segt + (int64_t)(t - t0) * n, -1, um(T + 1 + t),
                                         t + 1 < t1 ? um(T + 2 + t) : um(3 * (int64_t)(T + 1)));
            double* tt = u; u = un; un = tt;
        }
        for (int t = t1 - 1; t >= t0; --t) {
            const double* ut = S.segu + (int64_t)(t - t0) * n;
            const double* st = S.segs + (int64_t)(t - t0) * n;
            const double* tv = S.segt + (int64_t)(t - t0) * n;
            k_sw_rev1<G><<<gs, kWT, 0, s>>>(S, ut, st, tv, lam, um(T + 1 + t), um(2 * (int64_t)(T + 1) + t));
            k_sw_rev2<G><<<gs, kWT, 0, s>>>(S, ut, st, tv, lam, lam2, um(2 * (int64_t)(T + 1) + t));
            double* tt = lam; lam = lam2; lam2 = tt;
        }
        *launches += 1 + 3 * (t1 - t0);
    }
    return launch_smooth_coord(S, s, launches);
}

// Under two instances an SM a pass of one CTA waits on its own latency, and the
// whole GPU takes each pass instead.  So it does where more than nine list
// entries are within reach of a root on average: a lane of the persistent kernel
// holds a node alone, so its exponentials run one after the other and, past its
// scratch, the list is gathered again for every Newton sum.  Bound and gradient,
// 40 steps, 600 instances of 200-1,500 points, N = 24, persistent / per-step at
// that average: lattice 12.6 / 23.4 ms at 3.4, 17.1 / 29.3 at 6.7, 35.0 / 33.5 at
// 11.7, 58.1 / 37.8 at 25; uniform 23.9 / 32.4 at 6.6, 60.2 / 36.8 at 11.5;
// clustered 30.0 / 33.8 at 6.1, 89.4 / 42.9 at 14.7.
constexpr double kReachPersistent = 9.0;
// Few nodes leave SMs idle, so more lanes share a node's exponentials; many nodes
// fill them, and the shuffles of a wide group are wasted.  100 steps, N = 24, 4 /
// 8 / 16 / 32 lanes: 500 points 4.4 / 3.4 / 2.8 / 2.6 ms, 4,000 points 5.5 / 4.1 /
// 3.6 / 3.8, 10,000 points 6.0 / 5.5 / 5.9 / 7.0, 64 instances of 70,000 points in
// all 8.7 / 10.9 / 16.0 / 22.0.  Four lanes hold 48 entries, and one list of a warp
// past that makes the warp gather its lists again for every Newton sum: eight
// lanes where that is common, at u = 0 or, from an average of about 30 on, as the
// potentials move (40 steps, 4 / 8 lanes: 64 instances of 300-900 points, lattice
// 4.1 / 4.6 ms at 25 entries, 5.4 / 5.1 at 31, clustered with 1% of the nodes past
// 48 8.5 / 5.6 at 30; 600 of 200-1,500, uniform 55.6 / 59.8 at 31, lattice 102 / 77
// at 35, clustered with 1% past 48 62.0 / 59.2 at 30, with 12% 103 / 70 at 39).
constexpr int64_t kStepsMany = 14000, kStepsVeryMany = 150000;
bool smooth_needs_reach(int32_t solver, int32_t n_inst, int64_t n_total, int sms) {
    if (solver == 1) return false;
    return (solver == 0 && n_inst >= 2 * sms) || n_total > kStepsMany;
}
bool smooth_takes_steps(int32_t solver, int32_t n_inst, int sms, const SmoothReach& reach) {
    return solver == 2 || (solver == 0 && (n_inst < 2 * sms || reach.mean > kReachPersistent));
}
int smooth_step_lanes(int64_t n_total, const SmoothReach& reach) {
    if (n_total > kStepsMany)
        return reach.over > 0.005 || reach.mean > (n_total <= kStepsVeryMany ? 28 : 33) ? 8 : 4;
    return n_total <= 3000 ? 32 : (n_total <= 7000 ? 16 : 8);
}

cudaError_t launch_smooth_steps(SmoothBatch& S, bool grad, cudaStream_t s, int64_t* launches) {
    switch (S.lanes) {
        case 4: return launch_steps_of<4>(S, grad, s, launches);
        case 8: return launch_steps_of<8>(S, grad, s, launches);
        case 16: return launch_steps_of<16>(S, grad, s, launches);
        default: return launch_steps_of<32>(S, grad, s, launches);
    }
}

int32_t smooth_max_nodes() {
    int dev = 0, lim = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return (lim - 1024) / 16;
}

// Rate of the logistic term at full occupancy: every thread accumulates four
// independent LogitAcc sums (one exp and one division per term, the unit the
// persistent kernel counts), its arguments moving by a small step each round
// so that nothing is loop-invariant.
constexpr int kLogitProbeThreads = 256;
constexpr int kLogitChains = 4;
__global__ void __launch_bounds__(kLogitProbeThreads) k_logit_rate(double* out, int iters) {
    LogitAcc r[kLogitChains];
    double z[kLogitChains];
#pragma unroll
    for (int c = 0; c < kLogitChains; ++c) z[c] = -3.0 + 0.37 * c + 1e-3 * (threadIdx.x & 31);
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int c = 0; c < kLogitChains; ++c) {
            r[c].add(z[c]);
            z[c] += 1e-4;
        }
    }
    double t = 0.0;
#pragma unroll
    for (int c = 0; c < kLogitChains; ++c) t += r[c].cnt + r[c].tail + r[c].scale + r[c].slope;
    if (t == -1.0) out[blockIdx.x] = t;  // never true: the sums are >= 0; keeps them live
}
double logit_probe_terms(int blocks, int iters) {
    return (double)kLogitChains * (double)iters * (double)blocks * kLogitProbeThreads;
}
cudaError_t launch_logit_probe(int blocks, int iters, double* out, cudaStream_t s) {
    k_logit_rate<<<blocks, kLogitProbeThreads, 0, s>>>(out, iters);
    return cudaGetLastError();
}

cudaError_t launch_smooth_bound(SmoothBatch& S, int32_t max_v, bool grad, cudaStream_t s,
                                int64_t* launches) {
    int dev = 0, sms = 0, per_sm = 0, lim = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // two potential arrays, and a thread's scratch where it fits (an instance
    // near the limit re-reads its lists instead)
    const size_t pot = (size_t)max_v * 16, room = (size_t)lim - 1024;
    const size_t half = room / 2 - 1024;  // of two CTAs on an SM
    const size_t fit = pot + kBuf * kST * 10 <= half ? half : room;
    const int cap = (int)std::min<size_t>(fit == half ? 2 * kBuf : kBuf, (fit - pot) / (kST * 10));
    const size_t dyn = pot + (size_t)cap * kST * 10;
    const void* fn = grad ? (const void*)k_sbound<true> : (const void*)k_sbound<false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kST, dyn);
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    int grid = sms * per_sm;
    if (grid > S.n_inst) grid = S.n_inst;
    if ((e = cudaMemsetAsync(S.queue, 0, sizeof(int32_t), s)) != cudaSuccess) return e;
    if (S.work && (e = cudaMemsetAsync(S.work, 0, 2 * sizeof(unsigned long long), s)) != cudaSuccess) return e;
    if (grad && (e = clear_smooth_sums(S, s)) != cudaSuccess) return e;
    if (grad) k_sbound<true><<<grid, kST, dyn, s>>>(S, cap, max_v);
    else k_sbound<false><<<grid, kST, dyn, s>>>(S, cap, max_v);
    ++*launches;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return grad ? launch_smooth_coord(S, s, launches) : cudaSuccess;
}

}  // namespace f2m
