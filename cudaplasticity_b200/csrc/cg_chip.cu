// Masked (P)CG of one instance held on chip for the whole linear solve.
//
// Same solve as the one-launch-per-iteration form of cg_fused.cu
// (ConjGradCuda::solve, src/ConjGradCuda.cu:185-231, in the Chronopoulos-Gear
// arrangement described there: both inner products of an iteration in one
// reduction), as one launch per linear solve. The nodes are ordered along a
// Hilbert curve through the mesh, so that consecutive ones form compact
// patches, and each CTA owns a run of them, one node per thread:
//   - the node's row of K (the first kRegBlocks 2x2 blocks in registers, the
//     rest of a wider row in shared memory) and its x, r, p, w, kp, u, M w,
//     M kp and M stay on chip for the whole solve;
//   - U, in shared memory, holds u of the CTA's own nodes and of its halo
//     (the other CTAs' nodes its rows refer to), addressed by a 16-bit local
//     index per block that the plan computes once per instance;
//   - an iteration is: u' of the own nodes and of the halo into U, w' = K u'
//     from U, five sums, one exchange, which hands every CTA the records
//     (u, M w, M kp) of its halo nodes and the next step's scalars.
// Two exchanges:
//   cluster (up to 16 CTAs): records stay in their owner's shared memory and
//     are read through distributed shared memory; each CTA stores its sums
//     into the other CTAs' shared memory, where they complete an mbarrier
//     phase (one trip, where a cluster barrier and a read of the sums make
//     two); every CTA adds up all CTAs' sums in the same
//     order, so all hold the same scalars and take the same branches.
//   grid (up to one CTA per SM, a cooperative launch): records and sums go
//     through global memory (L2) in 8-byte words of 32 bits of data and their
//     sequence number, so that a reader polls the data itself: one trip
//     through L2 and no fence. One more CTA, without nodes, adds up the sums
//     and posts the next step's scalars (all CTAs reading all CTAs' sums takes
//     twice as long at 63 CTAs and more beyond: every poll then meets every
//     other on the same lines). Every poll is bounded; a CTA that gives up sets sc->chip_err and
//     returns, and so do the others at their next poll.
// T is the type of K's values and of the recurrences (double, or float in the
// mixed mode); x is FP64 and every sum is accumulated and reduced in FP64.
#include <cstdlib>

#include "cg.h"
#include "common.cuh"
#include "internal.h"

namespace cp {

namespace {

constexpr int kRegBlocks = 9;        // blocks of a row in registers (a 4-node mesh's interior row)
constexpr int kChipWarps = 12;       // slices per CTA: 384 threads of 168 registers
constexpr int kMaxCluster = 16;
constexpr int kSums = 5;
constexpr int kMaxPolls = 8;         // warps that poll the CTAs' sums (grid): up to 256 CTAs
constexpr int kHaloMax = 4096;       // halo nodes per CTA
constexpr size_t kSmemCap = 220 * 1024;
constexpr int kPlanThreads = 256;
constexpr int kOrderThreads = 1024;
constexpr int kCurveBits = 10;       // the curve visits a 1024 x 1024 grid over the mesh
constexpr int kDigitBits = 5, kDigits = 1 << kDigitBits;

// ------------------------------------------------------------------ plan --

// Position along the Hilbert curve of a cell of the 2^kCurveBits grid
// (D. Hilbert, 1891; the usual quadrant-by-quadrant rotation).
__device__ __forceinline__ unsigned int curve(unsigned int x, unsigned int y) {
    unsigned int d = 0;
    for (unsigned int s = 1u << (kCurveBits - 1); s > 0; s >>= 1) {
        const unsigned int rx = (x & s) ? 1u : 0u, ry = (y & s) ? 1u : 0u;
        d = 4u * d + ((3u * rx) ^ ry);
        if (ry == 0u) {
            if (rx == 1u) {
                x = ~x & ((1u << kCurveBits) - 1u);
                y = ~y & ((1u << kCurveBits) - 1u);
            }
            const unsigned int t = x;
            x = y;
            y = t;
        }
    }
    return d;
}

// The nodes in curve order, ties by node number: a stable radix sort in one
// block. order[slot] = node (-1 from n to slots), slot_of[node] = slot.
// scratch: 2 n (key, node) pairs.
__global__ void __launch_bounds__(kOrderThreads) k_chip_order(int n, int slots, const double2* __restrict__ xy,
                                                              uint2* scratch, int* order, int* slot_of) {
    extern __shared__ unsigned int cnt[];  // [kDigits][kOrderThreads]
    __shared__ double box[4][kOrderThreads / 32];
    __shared__ unsigned int wtot[kOrderThreads / 32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    double x0 = 1e300, y0 = 1e300, x1 = -1e300, y1 = -1e300;
    for (int i = t; i < n; i += kOrderThreads) {
        const double2 p = xy[i];
        x0 = fmin(x0, p.x); x1 = fmax(x1, p.x);
        y0 = fmin(y0, p.y); y1 = fmax(y1, p.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x0 = fmin(x0, __shfl_xor_sync(0xffffffffu, x0, o));
        y0 = fmin(y0, __shfl_xor_sync(0xffffffffu, y0, o));
        x1 = fmax(x1, __shfl_xor_sync(0xffffffffu, x1, o));
        y1 = fmax(y1, __shfl_xor_sync(0xffffffffu, y1, o));
    }
    if (lane == 0) { box[0][w] = x0; box[1][w] = y0; box[2][w] = x1; box[3][w] = y1; }
    __syncthreads();
    for (int q = 0; q < kOrderThreads / 32; ++q) {
        x0 = fmin(x0, box[0][q]); y0 = fmin(y0, box[1][q]);
        x1 = fmax(x1, box[2][q]); y1 = fmax(y1, box[3][q]);
    }
    const double ext = fmax(x1 - x0, y1 - y0), cells = (double)((1 << kCurveBits) - 1);
    const double scale = ext > 0.0 ? cells / ext : 0.0;
    const int chunk = (n + kOrderThreads - 1) / kOrderThreads;
    const int i0 = min(t * chunk, n), i1 = min(i0 + chunk, n);
    uint2 *a = scratch, *b = scratch + n;
    for (int i = t; i < n; i += kOrderThreads) {
        const double2 p = xy[i];
        const unsigned int cx = (unsigned int)fmin(fmax((p.x - x0) * scale, 0.0), cells);
        const unsigned int cy = (unsigned int)fmin(fmax((p.y - y0) * scale, 0.0), cells);
        a[i] = make_uint2(curve(cx, cy), (unsigned int)i);
    }
    __syncthreads();
    for (int shift = 0; shift < 2 * kCurveBits; shift += kDigitBits) {
        for (int d = 0; d < kDigits; ++d) cnt[d * kOrderThreads + t] = 0u;
        for (int i = i0; i < i1; ++i) ++cnt[((a[i].x >> shift) & (kDigits - 1)) * kOrderThreads + t];
        __syncthreads();
        // exclusive scan in (digit, thread) order, kDigits entries per thread
        unsigned int sum = 0;
        for (int q = 0; q < kDigits; ++q) sum += cnt[t * kDigits + q];
        unsigned int inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) wtot[w] = inc;
        __syncthreads();
        unsigned int run = inc - sum;
        for (int q = 0; q < w; ++q) run += wtot[q];
        for (int q = 0; q < kDigits; ++q) {
            const unsigned int v = cnt[t * kDigits + q];
            cnt[t * kDigits + q] = run;
            run += v;
        }
        __syncthreads();
        for (int i = i0; i < i1; ++i) {
            const uint2 v = a[i];
            b[cnt[((v.x >> shift) & (kDigits - 1)) * kOrderThreads + t]++] = v;
        }
        __syncthreads();
        uint2* q = a;
        a = b;
        b = q;
    }
    for (int i = t; i < slots; i += kOrderThreads) {
        const int nd = i < n ? (int)a[i].y : -1;
        order[i] = nd;
        if (nd >= 0) slot_of[nd] = i;
    }
}

// One block per CTA of the solve: its halo (ascending slots), the local index
// of every block of its rows, and a mark on every slot that is in another
// CTA's halo.
__global__ void __launch_bounds__(kPlanThreads) k_chip_plan(int slots, int own, int wmax,
                                                            const int* __restrict__ slice_ptr,
                                                            const int* __restrict__ scol,
                                                            const int* __restrict__ order,
                                                            const int* __restrict__ slot_of, unsigned short* lidx,
                                                            int* halo, int* halo_cnt, unsigned char* pub) {
    extern __shared__ unsigned int bits[];  // [words] marks, then [words] counts below
    __shared__ int chunk_sum[kPlanThreads];
    const int words = slots / 32;
    unsigned int* below = bits + words;
    const int rank = blockIdx.x, s0 = rank * own, s1 = s0 + own;
    for (int i = threadIdx.x; i < words; i += blockDim.x) bits[i] = 0u;
    __syncthreads();
    for (int s = s0 + threadIdx.x; s < s1; s += blockDim.x) {
        const int nd = order[s];
        if (nd < 0) continue;
        const int base = slice_ptr[nd >> 5], wd = (slice_ptr[(nd >> 5) + 1] - base) >> 5;
        for (int k = 0; k < wd; ++k) {
            const int c = slot_of[scol[base + 32 * k + (nd & 31)]];
            if (c < s0 || c >= s1) atomicOr(&bits[c >> 5], 1u << (c & 31));
        }
    }
    __syncthreads();
    const int chunk = (words + blockDim.x - 1) / blockDim.x;
    const int w0 = min((int)threadIdx.x * chunk, words), w1 = min(w0 + chunk, words);
    int cnt = 0;
    for (int i = w0; i < w1; ++i) cnt += __popc(bits[i]);
    chunk_sum[threadIdx.x] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int t = 0; t < (int)blockDim.x; ++t) {
            const int v = chunk_sum[t];
            chunk_sum[t] = run;
            run += v;
        }
        halo_cnt[rank] = run;
    }
    __syncthreads();
    int at = chunk_sum[threadIdx.x];
    for (int i = w0; i < w1; ++i) {
        below[i] = (unsigned int)at;
        for (unsigned int m = bits[i]; m; m &= m - 1) {
            const int slot = 32 * i + __ffs(m) - 1;
            if (at < kHaloMax) halo[(size_t)rank * kHaloMax + at] = slot;
            pub[slot] = 1;
            ++at;
        }
    }
    __syncthreads();
    for (int s = s0 + threadIdx.x; s < s1; s += blockDim.x) {
        const int nd = order[s];
        if (nd < 0) continue;
        const int base = slice_ptr[nd >> 5], wd = (slice_ptr[(nd >> 5) + 1] - base) >> 5;
        for (int k = 0; k < wd; ++k) {
            const int c = slot_of[scol[base + 32 * k + (nd & 31)]];
            int l = c - s0;
            if (c < s0 || c >= s1)
                l = own + (int)(below[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31)) - 1u)));
            lidx[((size_t)(s >> 5) * wmax + k) * 32 + (s & 31)] = (unsigned short)l;
        }
    }
}

// --------------------------------------------------------------- helpers --

__device__ __forceinline__ unsigned int smem_addr(const void* p) {
    return (unsigned int)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned int mapa(unsigned int addr, int rank) {
    unsigned int r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void ld_cluster(unsigned int a, double2& v) {
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_cluster(unsigned int a, float2& v) {
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
}
// Two doubles into another CTA's shared memory; they count 16 bytes towards
// the phase of the mbarrier there.
__device__ __forceinline__ void st_async(unsigned int a, unsigned int bar, double x, double y) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(a),
                 "l"(__double_as_longlong(x)), "l"(__double_as_longlong(y)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bar_init(unsigned int bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned int bar, unsigned int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned int bar, unsigned int phase) {
    unsigned int ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(bar), "r"(phase)
        : "memory");
    return ok != 0;
}
// Shared-memory reads of U by byte address.
__device__ __forceinline__ void ld_u(unsigned int a, double2& v) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_u(unsigned int a, float2& v) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
}
__device__ __forceinline__ void cluster_arrive_release() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Two words of (32 bits of data, sequence number).
__device__ __forceinline__ uint4 ld_words(const uint4* p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ void st_words(uint4* p, unsigned int lo, unsigned int hi, unsigned int seq) {
    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(lo), "r"(seq), "r"(hi), "r"(seq)
                 : "memory");
}
__device__ __forceinline__ void post(uint4* p, double v, unsigned int seq) {
    st_words(p, __double2loint(v), __double2hiint(v), seq);
}
__device__ __forceinline__ void post(uint4* p, float2 v, unsigned int seq) {
    st_words(p, __float_as_uint(v.x), __float_as_uint(v.y), seq);
}
__device__ __forceinline__ double word_value(const uint4& q) { return __hiloint2double(q.z, q.x); }

// Polls N word pairs per lane until those of every lane of the warp carry seq;
// false after `limit` rounds. The whole warp takes part, with valid addresses
// in every lane: left to diverge, a warp of which some lanes polled and some
// did not took 3700 cycles to come together again.
template <int N>
__device__ __forceinline__ bool poll(const uint4* p, size_t stride, unsigned int seq, unsigned int limit, uint4* c) {
    for (unsigned int round = 0; round < limit; ++round) {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < N; ++i) c[i] = ld_words(p + i * stride);
#pragma unroll
        for (int i = 0; i < N; ++i) ok = ok && c[i].y == seq && c[i].w == seq;
        if (__all_sync(0xffffffffu, ok)) return true;
    }
    return false;
}

// A record (u, M w, M kp): pair i at p[i * stride].
template <typename T>
struct Record;
template <>
struct Record<double> {
    static constexpr int n = 6;
    __device__ static void put(uint4* p, size_t stride, double2 u, double2 mw, double2 mk, unsigned int seq) {
        post(p, u.x, seq);
        post(p + stride, u.y, seq);
        post(p + 2 * stride, mw.x, seq);
        post(p + 3 * stride, mw.y, seq);
        post(p + 4 * stride, mk.x, seq);
        post(p + 5 * stride, mk.y, seq);
    }
    __device__ static void get(const uint4* c, double2* r) {
#pragma unroll
        for (int i = 0; i < 3; ++i) r[i] = make_double2(word_value(c[2 * i]), word_value(c[2 * i + 1]));
    }
};
template <>
struct Record<float> {
    static constexpr int n = 3;
    __device__ static void put(uint4* p, size_t stride, float2 u, float2 mw, float2 mk, unsigned int seq) {
        post(p, u, seq);
        post(p + stride, mw, seq);
        post(p + 2 * stride, mk, seq);
    }
    __device__ static void get(const uint4* c, float2* r) {
#pragma unroll
        for (int i = 0; i < 3; ++i) r[i] = make_float2(__uint_as_float(c[i].x), __uint_as_float(c[i].z));
    }
};
constexpr int kStepWords = 3;  // alpha, beta, go

template <typename V2>
__device__ __forceinline__ V2 make2(decltype(V2::x) x, decltype(V2::x) y) {
    V2 v;
    v.x = x;
    v.y = y;
    return v;
}

// Sums of the five values over the warp in 8 shuffles instead of 25 (the
// shuffle unit takes one warp per cycle and SM): each step folds two values
// into one register per half of the lanes. Lanes 0..3 end with v0, 4..7 with
// v2, 8..15 with v1, 16..23 with v3, 24..31 with v4; every fourth lane stores
// (slot lane / 4 of 8), and sum_slot(i) is a slot that holds value i. (A
// store from the one lane of each value, picked by comparing the lane with
// five constants, compiled to a branch table: 600 cycles more.)
__device__ __forceinline__ double warp_sum5(const double* v, int lane) {
    const unsigned int full = 0xffffffffu;
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
    double a = h16 ? v[3] : v[0], b = h16 ? v[4] : v[1], c = h16 ? 0.0 : v[2];
    a += __shfl_xor_sync(full, h16 ? v[0] : v[3], 16);
    b += __shfl_xor_sync(full, h16 ? v[1] : v[4], 16);
    {
        const double t = __shfl_xor_sync(full, h16 ? v[2] : 0.0, 16);
        c += h16 ? 0.0 : t;
    }
    double d = h8 ? b : a;
    d += __shfl_xor_sync(full, h8 ? a : b, 8);
    c += __shfl_xor_sync(full, c, 8);
    // lanes 0..7: d = v0 sums, c = v2 sums: one of them per half of the lanes
    const bool two = lane < 8;
    double e = (two && h4) ? c : d;
    e += __shfl_xor_sync(full, (two && !h4) ? c : d, 4);
    e += __shfl_xor_sync(full, e, 2);
    e += __shfl_xor_sync(full, e, 1);
    return e;
}
__device__ __forceinline__ constexpr int sum_slot(int i) { return i == 0 ? 0 : i == 1 ? 2 : i == 2 ? 1 : 2 * i - 2; }

// What the exchange decides: the next step's scalars, go = 0 at the end.
struct Step {
    double alpha, beta;
    int go;
};

// ---------------------------------------------------------------- kernel --

template <typename T, bool GRID>
__global__ void __launch_bounds__(kChipWarps * 32, 1) k_chip(ChipArgs<T> a) {
    using V2 = typename Vec2<T>::type;
    using V4 = typename Vec4<T>::type;
    constexpr int W = kRegBlocks, NR = Record<T>::n;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double wsum[16][8];  // per warp: its sums (unused warps stay zero)
    __shared__ double gsum[kMaxPolls][8];  // grid, the adding CTA: the same of the CTAs' sums
    __shared__ __align__(16) double part[2][kMaxCluster][6];  // cluster: every CTA's sums (0, 2, 1, -, 3, 4), by parity
    __shared__ __align__(8) unsigned long long bar[2];  // cluster: they have arrived
    __shared__ Step step;
    const ChipPlan& P = a.plan;
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, w = tid >> 5;
    const int rank = blockIdx.x, ctas = P.ctas, own = P.spc * 32;
    const size_t slots = (size_t)ctas * own;
    const int slot = rank * own + tid, n = GRID && rank == ctas ? -1 : P.order[slot];
    const bool act = n >= 0;
    // shared memory: U [own + halo], then (cluster) records [2][3][own], then
    // the blocks beyond W: values, local indexes
    V2* U = reinterpret_cast<V2*>(smem_raw);
    V2* rec = U + own + P.halo_cap;
    const int extra = P.wmax > W ? P.wmax - W : 0;
    V4* kval = reinterpret_cast<V4*>(rec + (GRID ? 0 : 6 * own));
    unsigned short* kidx = reinterpret_cast<unsigned short*>(kval + (size_t)own * extra);
    const unsigned int u_base = smem_addr(U);

    for (int i = tid; i < 128; i += nthr) (&wsum[0][0])[i] = 0.0;
    for (int i = tid; i < kMaxPolls * 8; i += nthr) (&gsum[0][0])[i] = 0.0;
    for (int i = tid; i < 2 * kMaxCluster * 6; i += nthr) (&part[0][0][0])[i] = 0.0;
    // ---- rows, r = m.(b - K x), M
    V4 kr[W];
    unsigned int li[W];  // byte addresses in U
#pragma unroll
    for (int k = 0; k < W; ++k) {
        kr[k].x = kr[k].y = kr[k].z = kr[k].w = (T)0;
        li[k] = u_base + tid * (unsigned int)sizeof(V2);
    }
    int wd = 0;
    double2 x = make_double2(0.0, 0.0);
    uchar2 m = make_uchar2(0, 0);
    V2 r = make2<V2>(0, 0), p = r, kp = r, wv = r, u = r;
    T mi0 = (T)0, mi1 = (T)0, mi2 = (T)0;  // M, symmetric as K is: m00, m01 = m10, m11
    bool publish = false;
    double v[kSums] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (act) {
        const int base = a.slice_ptr[n >> 5] + (n & 31);
        wd = (a.slice_ptr[(n >> 5) + 1] - base + 31) >> 5;
        m = a.mask[n];
        x = a.x[n];
        publish = P.pub[slot] != 0;
        const unsigned short* lx = P.lidx + (size_t)(slot >> 5) * P.wmax * 32 + lane;
        double k0 = 0.0, k1 = 0.0;
        double4 diag = make_double4(0.0, 0.0, 0.0, 0.0);
        auto residual = [&](int k) {  // FP64, also in the mixed mode
            const long long bi = base + 32LL * k;
            const double2* vp = reinterpret_cast<const double2*>(a.val64 + 4 * bi);
            const double2 lo = __ldg(vp), hi = __ldg(vp + 1);
            const double2 xc = a.x[__ldg(a.scol + bi)];
            k0 += lo.x * xc.x + lo.y * xc.y;
            k1 += hi.x * xc.x + hi.y * xc.y;
            if (k == 0) diag = make_double4(lo.x, lo.y, hi.x, hi.y);
            V4 q;
            q.x = (T)lo.x; q.y = (T)lo.y; q.z = (T)hi.x; q.w = (T)hi.y;
            return q;
        };
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (k < wd) {
                kr[k] = residual(k);
                li[k] = u_base + lx[32 * k] * (unsigned int)sizeof(V2);
            }
        for (int k = W; k < wd; ++k) {
            const size_t q = (size_t)(k - W) * own + tid;
            kval[q] = residual(k);
            kidx[q] = lx[32 * k];
        }
        const double2 bb = a.b[n];
        const double r0 = m.x ? bb.x - k0 : 0.0, r1 = m.y ? bb.y - k1 : 0.0;
        r = make2<V2>((T)r0, (T)r1);
        if (a.precond) {  // inverse of the diagonal block on the free DOFs
            if (m.x && m.y) {
                const double det = diag.x * diag.w - diag.y * diag.z;
                mi0 = (T)(diag.w / det);
                mi1 = (T)(-diag.y / det);
                mi2 = (T)(diag.x / det);
            } else if (m.x) {
                mi0 = (T)(1.0 / diag.x);
            } else if (m.y) {
                mi2 = (T)(1.0 / diag.w);
            }
        } else {
            mi0 = (T)(m.x ? 1 : 0);
            mi2 = (T)(m.y ? 1 : 0);
        }
        u = make2<V2>(mi0 * r.x + mi1 * r.y, mi1 * r.x + mi2 * r.y);
        v[0] = (double)r.x * (double)r.x + (double)r.y * (double)r.y;
        v[1] = bb.x * bb.x + bb.y * bb.y;
        v[2] = r0 * r0 + r1 * r1;
    }
    wd -= W;  // blocks beyond the registers
    // ---- halo: thread nthr - 1 - tid takes the first halo nodes, so that the
    // warps that wait for the sums have few of them
    const int hc = GRID && rank == ctas ? 0 : P.halo_cnt[rank], h0 = nthr - 1 - tid;
    const int* hl = P.halo + (size_t)rank * kHaloMax;
    const unsigned int rec_base = smem_addr(rec);
    // where the record of halo slot s is read: cluster address, or the slot (grid)
    auto halo_at = [&](int s) -> unsigned int {
        if (GRID) return (unsigned int)s;
        const int cr = s / own;
        return mapa(rec_base + (unsigned int)((s - cr * own) * sizeof(V2)), cr);
    };
    // the first halo record of this thread (past the last one: the last one,
    // so that whole warps read), and the smallest h0 of the warp
    const unsigned int ha = hc > 0 ? halo_at(hl[min(h0, hc - 1)]) : 0u;
    const int h_min = nthr - 32 * (w + 1);
    unsigned int seq = GRID ? *a.seq : 0u;
    const int np = (ctas + 31) >> 5;  // grid: warps of CTA 0 that poll the CTAs' sums
    int par = 1;                      // parity of the last exchange
    bool failed = false;
    V2 hr[3];
    // ---- the scalars of the solve: warp 0 (grid: of CTA 0)
    double rr = 0.0, rho = 0.0, rho_inv = 0.0, bnorm2 = 0.0, res64 = 0.0, normB_inv = 0.0;
    int status = 0, converged = 0, lin_done = 0;
    int iter = 0;
    const int max_iter = (int)(a.max_iter < 0x7fffffffLL ? a.max_iter : 0x7fffffffLL);
    unsigned int phase = 0;  // of the mbarriers' next wait
    if (!GRID && tid == 0) {
        bar_init(smem_addr(&bar[0]));
        bar_init(smem_addr(&bar[1]));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bar_expect(smem_addr(&bar[0]), 48u * ctas);
        bar_expect(smem_addr(&bar[1]), 48u * ctas);
    }
    if constexpr (!GRID) {
        cluster_arrive_release();
        cluster_wait();
    } else {
        __syncthreads();
    }

    auto apply_m = [&](V2 q) { return make2<V2>(mi0 * q.x + mi1 * q.y, mi1 * q.x + mi2 * q.y); };
    auto read_halo = [&](unsigned int at, V2* q) {
        if constexpr (GRID) {
            uint4 c[NR];
            if (!poll<NR>(a.ll_rec + (size_t)par * NR * slots + at, slots, seq, a.poll_limit, c)) failed = true;
            Record<T>::get(c, q);
        } else {
            const unsigned int s = at + (unsigned int)(par * 3 * own * sizeof(V2));
#pragma unroll
            for (int i = 0; i < 3; ++i) ld_cluster(s + (unsigned int)(i * own * sizeof(V2)), q[i]);
        }
    };
    // The next step from the sums of an iteration (see cg_fused.cu for the
    // recurrences). Straight-line: one warp runs it while all others wait, and
    // its branches cost more than its arithmetic; why the solve ended is
    // worked out by finish().
    auto decide = [&](const double* tot) -> Step {
        const double g = tot[0], b2 = g * rho_inv;
        const double den = tot[1] + b2 * tot[3] + b2 * b2 * tot[4];
        const double an = g * __drcp_rn(den);
        rr = tot[2];
        rho = g;
        rho_inv = den;  // the loop top replaces it
        iter += 1;
        const int go = (int)(rr * normB_inv > a.eps2) & (int)(iter < max_iter) & (int)(den > 0.0) & (int)(g > 0.0);
        return {an, b2, go};
    };
    auto decide_first = [&](const double* tot) -> Step {
        rho = tot[0];
        const double an = tot[0] / tot[1];
        rho_inv = tot[1];
        if (!(tot[1] > 0.0) || !(an == an)) status = CP_ERR_BREAKDOWN;
        return {an, 0.0, status == 0};
    };
    auto decide_init = [&](const double* tot) -> Step {
        rr = tot[0];
        bnorm2 = tot[1];
        res64 = tot[2];
        normB_inv = a.relative_to_r0 ? (rr > 0.0 ? 1.0 / rr : 0.0) : (bnorm2 > 0.0 ? 1.0 / bnorm2 : 0.0);
        lin_done = a.outer_eps2 >= 0.0 && res64 <= a.outer_eps2 * bnorm2 ? 1 : 0;
        converged = (lin_done || rr == 0.0 || rr * normB_inv <= a.eps2) ? 1 : 0;
        if (!(rr == rr) || !(bnorm2 == bnorm2)) status = CP_ERR_BREAKDOWN;
        return {0.0, 0.0, !converged && !status};
    };
    // The solve's scalars for the host (thread 0 of the CTA that decides).
    auto finish = [&]() {
        if (tid != 0) return;
        CgScalars* sc = a.sc;
        if (failed) {
            atomicExch(&sc->chip_err, 1);
            return;
        }
        if (iter > 0) {  // rho_inv holds the last step's denominator
            if (rr * normB_inv <= a.eps2) converged = 1;
            else if (iter >= max_iter) status = CP_ERR_NOT_CONVERGED;
            else if (!(rho_inv > 0.0) || !(rho > 0.0)) {
                // in FP32 the step may degenerate before the residual does: the
                // solve ends there and the caller takes the FP64 residual
                status = sizeof(T) == 4 ? CP_ERR_DEGENERATE : CP_ERR_BREAKDOWN;
            }
            if (!(rr == rr)) status = CP_ERR_BREAKDOWN;
        }
        sc->rr = rr;
        sc->bb = bnorm2;
        sc->res64 = res64;
        sc->normB_inv = normB_inv;
        sc->eps2 = a.eps2;
        sc->iter = iter;
        sc->max_iter = a.max_iter;
        sc->converged = converged;
        sc->status = status;
        sc->lin_done = lin_done;
        sc->alpha = step.alpha;
        sc->beta = step.beta;
        sc->rho = rho;
        sc->ticket = 0;
        if (GRID) *a.seq = seq;  // every CTA has read the old value: all have taken part in an exchange
    };
    // Posts the own record and the sums v; receives the first halo record (hr)
    // and the next step. Every thread returns with `step` readable.
    auto exchange = [&](auto decide_now) {
        par ^= 1;
        if constexpr (GRID) {
            seq += 1;
            if (publish)
                Record<T>::put(a.ll_rec + (size_t)par * NR * slots + slot, slots, u, apply_m(wv), apply_m(kp),
                               seq + a.seq_skew);
        } else {
            if (publish) {
                V2* own_rec = rec + (size_t)par * 3 * own + tid;
                own_rec[0] = u;
                own_rec[own] = apply_m(wv);
                own_rec[2 * own] = apply_m(kp);
            }
        }
        {
            const double s = warp_sum5(v, lane);
            if ((lane & 3) == 0) wsum[w][lane >> 2] = s;
        }
        __syncthreads();
        // lane (g, j): slot j of the warps g, g + 4, ..; then over g
        const int j = lane & 7, g = lane >> 3;
        double s = 0.0;
        if (w == 0) {
            s = (wsum[g][j] + wsum[g + 4][j]) + wsum[g + 8][j];
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 16);
        }
        if constexpr (GRID) {
            uint4* pp = a.ll_part + (size_t)par * 8 * ctas;
            uint4* rp = a.ll_step + par * 4;
            // slots 0, 1, 2, 4, 6 hold the values 0, 2, 1, 3, 4
            const int val = lane == 1 ? 2 : lane == 2 ? 1 : lane > 2 ? lane / 2 + 1 : 0;
            if (w == 0 && (lane < 3 || lane == 4 || lane == 6))
                post(pp + (size_t)val * ctas + rank, s, seq + a.seq_skew);
            if (w == 0) {
                uint4 c[1];
                if (!poll<1>(rp + min(lane, kStepWords - 1), 1, seq, a.poll_limit, c)) failed = true;
                const double q = word_value(c[0]);
                if (lane == 0) step.alpha = q;
                if (lane == 1) step.beta = q;
                if (lane == 2) step.go = q != 0.0;
            }
            if (h_min < hc) read_halo(ha, hr);
            failed = __syncthreads_or(failed ? 1 : 0) != 0;
        } else {
            if (w == 0) {
                // sums (0, 2), (1, 1), (3, 4) to every CTA, with the records of
                // all warps written before the block barrier above
                const double s2 = __shfl_sync(0xffffffffu, s, j == 4 ? 6 : j + 1);
                if (!(j & 1) && j < 6) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (g + 4 * i < ctas)
                            st_async(mapa(smem_addr(&part[par][rank][j]), g + 4 * i),
                                     mapa(smem_addr(&bar[par]), g + 4 * i), s, s2);
                }
            }
            {
                const unsigned int ba = smem_addr(&bar[par]);
                unsigned int round = 0;
                while (!bar_try(ba, phase)) {
                    if (++round > a.poll_limit) {
                        failed = true;
                        break;
                    }
                }
            }
            if (par) phase ^= 1u;
            if (h_min < hc) read_halo(ha, hr);
            if (w == 0) {
                if (lane == 0) bar_expect(smem_addr(&bar[par]), 48u * ctas);  // its next use
                // lane (g, j): value j of the CTAs g, g + 4, ..; then over g
                const int e = j < 6 ? j : 0;
                s = (part[par][g][e] + part[par][g + 4][e]) + (part[par][g + 8][e] + part[par][g + 12][e]);
                s += __shfl_xor_sync(0xffffffffu, s, 8);
                s += __shfl_xor_sync(0xffffffffu, s, 16);
                double tot[kSums];
#pragma unroll
                for (int i = 0; i < kSums; ++i)
                    tot[i] = __shfl_sync(0xffffffffu, s, i == 0 ? 0 : i == 1 ? 2 : i == 2 ? 1 : i + 1);
                const Step st = decide_now(tot);
                if (lane == 0) step = st;
            }
            failed = __syncthreads_or(failed ? 1 : 0) != 0;
        }
    };
    // U of the own node and of the halo at step (al, bt).
    auto fill_u = [&](T al, T bt) {
        U[tid] = u;
        if (h0 < hc)
            U[own + h0] = make2<V2>(hr[0].x - al * (hr[1].x + bt * hr[2].x), hr[0].y - al * (hr[1].y + bt * hr[2].y));
        if (hc > nthr) {
            for (int b = nthr; h_min + b < hc; b += nthr) {
                const int h = h0 + b;
                read_halo(halo_at(hl[min(h, hc - 1)]), hr);
                if (h < hc)
                    U[own + h] = make2<V2>(hr[0].x - al * (hr[1].x + bt * hr[2].x),
                                           hr[0].y - al * (hr[1].y + bt * hr[2].y));
            }
            if (GRID) failed = __syncthreads_or(failed ? 1 : 0) != 0;
        }
        __syncthreads();
    };
    auto gather = [&]() {
        T k0 = (T)0, k1 = (T)0;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            V2 c;
            ld_u(li[k], c);
            k0 += kr[k].x * c.x + kr[k].y * c.y;
            k1 += kr[k].z * c.x + kr[k].w * c.y;
        }
        for (int k = 0; k < wd; ++k) {
            const size_t q = (size_t)k * own + tid;
            const V4 kv = kval[q];
            const V2 c = U[kidx[q]];
            k0 += kv.x * c.x + kv.y * c.y;
            k1 += kv.z * c.x + kv.w * c.y;
        }
        return make2<V2>(k0, k1);
    };
    if (GRID && rank == ctas) {
        // the CTA without nodes: adds up all CTAs' sums and posts the steps
        auto lead = [&](auto decide_now) {
            par ^= 1;
            seq += 1;
            const uint4* pp = a.ll_part + (size_t)par * 8 * ctas;
            for (int q = w; q < np; q += nthr >> 5) {
                double t[kSums];
                uint4 ch[kSums];
                const int c = 32 * q + lane;
                if (!poll<kSums>(pp + min(c, ctas - 1), ctas, seq, a.poll_limit, ch)) failed = true;
#pragma unroll
                for (int i = 0; i < kSums; ++i) t[i] = c < ctas ? word_value(ch[i]) : 0.0;
                const double r5 = warp_sum5(t, lane);
                if ((lane & 3) == 0) gsum[q][lane >> 2] = r5;
            }
            failed = __syncthreads_or(failed ? 1 : 0) != 0;
            if (w == 0) {
                double t = 0.0;
#pragma unroll
                for (int q = 0; q < kMaxPolls; ++q) t += gsum[q][lane & 7];
                double tot[kSums];
#pragma unroll
                for (int i = 0; i < kSums; ++i) tot[i] = __shfl_sync(0xffffffffu, t, sum_slot(i));
                const Step st = decide_now(tot);
                if (lane < kStepWords)
                    post(a.ll_step + par * 4 + lane, lane == 0 ? st.alpha : lane == 1 ? st.beta : (double)st.go,
                         seq + a.seq_skew);
                if (lane == 0) step = st;
            }
            __syncthreads();
            return step.go != 0 && !failed;
        };
        if (lead(decide_init) && lead(decide_first)) {
            do {
                rho_inv = __drcp_rn(rho);
            } while (lead(decide));
        }
        finish();
        return;
    }
    // ---- (r, r), (b, b), and u to the neighbours
    exchange(decide_init);
    fill_u((T)0, (T)0);
    bool go = step.go != 0 && !failed;
    if (go) {
        // ---- first step: w = K u; gamma = (r, u), delta = (w, u)
        wv = gather();
        v[0] = (double)r.x * (double)u.x + (double)r.y * (double)u.y;
        v[1] = (double)wv.x * (double)u.x + (double)wv.y * (double)u.y;
        v[2] = 0.0;
        exchange(decide_first);
        go = step.go != 0 && !failed;
    }
    // ---- iterations
    while (go) {
        const double alpha = step.alpha;
        if (!GRID) rho_inv = __drcp_rn(rho);  // for the next decision, off its path
        const T al = (T)alpha, bt = (T)step.beta;
        const V2 u0 = u;
        const V2 mw = apply_m(wv), mk = apply_m(kp);
        u = make2<V2>(u0.x - al * (mw.x + bt * mk.x), u0.y - al * (mw.y + bt * mk.y));
        fill_u(al, bt);
        p = make2<V2>(u0.x + bt * p.x, u0.y + bt * p.y);
        kp = make2<V2>(wv.x + bt * kp.x, wv.y + bt * kp.y);
        x.x += alpha * (double)p.x;
        x.y += alpha * (double)p.y;
        if (m.x) r.x -= al * kp.x;
        if (m.y) r.y -= al * kp.y;
        wv = gather();
        v[0] = (double)r.x * (double)u.x + (double)r.y * (double)u.y;
        v[1] = (double)wv.x * (double)u.x + (double)wv.y * (double)u.y;
        v[2] = (double)r.x * (double)r.x + (double)r.y * (double)r.y;
        v[3] = ((double)wv.x * (double)p.x + (double)wv.y * (double)p.y) +
               ((double)kp.x * (double)u.x + (double)kp.y * (double)u.y);
        v[4] = (double)kp.x * (double)p.x + (double)kp.y * (double)p.y;
        exchange(decide);
        go = step.go != 0 && !failed;
    }
    if constexpr (!GRID) {  // the others have read this CTA's memory for the last time
        cluster_arrive_release();
        cluster_wait();
    }
    if (failed) {
        if (tid == 0) atomicExch(&a.sc->chip_err, 1);
        return;
    }
    if (act) a.x[n] = x;
    if (!GRID && rank == 0) finish();
}

// Dynamic shared memory per CTA.
size_t chip_smem(bool grid, int spc, int wmax, int halo, size_t st) {
    const size_t own = (size_t)spc * 32, extra = wmax > kRegBlocks ? wmax - kRegBlocks : 0;
    size_t b = (own + halo) * 2 * st;
    if (!grid) b += 6 * own * 2 * st;
    b += own * extra * (4 * st + 2);
    return (b + 15) / 16 * 16;
}

template <typename K>
cudaLaunchConfig_t chip_config(K, const ChipPlan& p, size_t smem, cudaLaunchAttribute* attr, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.ctas + (p.grid ? 1 : 0));  // the grid form's last CTA adds up the sums
    cfg.blockDim = dim3(32 * p.spc);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    if (p.grid) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    } else {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = p.ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// The attributes of kernel k (per function: the cap, not one instance's size).
template <typename K>
bool chip_attributes(K k, bool grid) {
    bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap) == cudaSuccess;
    if (ok && !grid) ok = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok;
}

template <typename T>
bool chip_schedulable(const ChipPlan& p, int sm_count) {
    const size_t smem = chip_smem(p.grid, p.spc, p.wmax, p.halo_cap, sizeof(T));
    if (smem > kSmemCap) return false;
    if (p.grid) {
        int per_sm = 0;
        if (!chip_attributes(k_chip<T, true>, true) ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_chip<T, true>, 32 * p.spc, smem) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return (long long)per_sm * sm_count >= p.ctas + 1;
    }
    if (!chip_attributes(k_chip<T, false>, false)) return false;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = chip_config(k_chip<T, false>, p, smem, attr, nullptr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_chip<T, false>, &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        return false;
    }
    return true;
}

}  // namespace

// The shape of the cluster (grid = false) or grid form for n nodes; ctas = 0
// when it does not hold them.
//   cluster: about 13 CTAs, of at least 4 slices. 1024 nodes: 8 CTAs of 4
//     slices 1.70 us per iteration, 16 of 2 2.10, 3 of 12 1.92; 4160 nodes: 13
//     of 10 1.93, 11 of 12 1.93 (the whole solve in one cluster with every
//     record read through distributed shared memory: 4.9 and 5.7).
//   grid: about 128 CTAs, of at least 8 slices. 16104 nodes: 63 CTAs of 8
//     slices 3.40 us, 126 of 4 3.82, 42 of 12 3.54 (one launch per iteration,
//     cg_fused.cu: 10.2); 40200 nodes: 126 of 10 3.67, 105 of 12 3.83 (11.3).
//     At sizes that both hold the cluster is the faster one (4160 nodes: 3.13
//     as a grid).
ChipShape chip_shape(int n, int wmax, int sm_count, bool grid) {
    const int n_slices = (n + 31) / 32;
    ChipShape s;
    s.wmax = wmax;
    s.grid = grid;
    s.spc = grid ? std::max((n_slices + 127) / 128, 8) : std::max((n_slices + 12) / 13, 4);
    if (const char* e = std::getenv("CUPLAST_CHIP_FORM")) {  // c<slices per CTA> or g<slices per CTA> (measurements)
        const int v = std::atoi(e + 1);
        if ((e[0] == 'c' || e[0] == 'g') && v >= 1 && v <= kChipWarps) {
            if (grid != (e[0] == 'g')) return s;
            s.spc = v;
        }
    }
    s.spc = std::min(s.spc, kChipWarps);
    s.ctas = (n_slices + s.spc - 1) / s.spc;
    if (s.ctas > (grid ? std::min(sm_count - 1, 32 * kMaxPolls) : kMaxCluster)) s.ctas = 0;
    return s;
}

static size_t chip_slots(const ChipShape& s) { return (size_t)s.ctas * s.spc * 32; }

// One allocation of ints: order, slot_of, halo, halo_cnt; then lidx and pub.
size_t chip_plan_bytes(const ChipShape& s, int n) {
    const size_t slots = chip_slots(s);
    return sizeof(int) * (slots + n + (size_t)s.ctas * (kHaloMax + 1)) + sizeof(unsigned short) * slots * s.wmax + slots;
}

// Exchange buffers of the grid form: records, sums, steps, by parity.
size_t chip_ll_bytes(const ChipShape& s) {
    return s.grid ? 2 * (chip_slots(s) * Record<double>::n + 8 * (size_t)s.ctas + 4) * sizeof(uint4) : 0;
}
void chip_ll_carve(const ChipPlan& p, void* mem, uint4** rec, uint4** part, uint4** step) {
    const size_t slots = (size_t)p.ctas * p.spc * 32;
    *rec = static_cast<uint4*>(mem);
    *part = *rec + 2 * slots * Record<double>::n;
    *step = *part + 16 * (size_t)p.ctas;
}

// Builds the plan on the device; plan.ctas = 0 when the instance does not fit.
void chip_build_plan(ChipPlan& p, const ChipShape& s, void* mem, int n, const double2* xy, const int* slice_ptr,
                     const int* scol, int sm_count, cudaStream_t st) {
    const size_t slots = chip_slots(s);
    p.grid = s.grid;
    p.spc = s.spc;
    p.wmax = s.wmax;
    p.ctas = 0;
    int* ints = static_cast<int*>(mem);
    p.order = ints;
    int* slot_of = ints + slots;
    p.halo = slot_of + n;
    p.halo_cnt = p.halo + (size_t)s.ctas * kHaloMax;
    p.lidx = reinterpret_cast<unsigned short*>(p.halo_cnt + s.ctas);
    p.pub = reinterpret_cast<unsigned char*>(p.lidx + slots * s.wmax);
    uint2* scratch = nullptr;
    CP_CUDA(cudaMallocAsync(&scratch, 2 * sizeof(uint2) * (size_t)n, st));
    CP_CUDA(cudaMemsetAsync(p.pub, 0, slots, st));
    constexpr int order_smem = kDigits * kOrderThreads * (int)sizeof(unsigned int);
    CP_CUDA(cudaFuncSetAttribute(k_chip_order, cudaFuncAttributeMaxDynamicSharedMemorySize, order_smem));
    k_chip_order<<<1, kOrderThreads, order_smem, st>>>(n, (int)slots, xy, scratch, p.order, slot_of);
    k_chip_plan<<<s.ctas, kPlanThreads, 2 * sizeof(unsigned int) * (slots / 32), st>>>(
        (int)slots, s.spc * 32, s.wmax, slice_ptr, scol, p.order, slot_of, p.lidx, p.halo, p.halo_cnt, p.pub);
    CP_CUDA(cudaGetLastError());
    CP_CUDA(cudaFreeAsync(scratch, st));
    std::vector<int> cnt(s.ctas);
    CP_CUDA(cudaMemcpyAsync(cnt.data(), p.halo_cnt, sizeof(int) * s.ctas, cudaMemcpyDeviceToHost, st));
    CP_CUDA(cudaStreamSynchronize(st));
    int most = 0;
    for (int c : cnt) most = std::max(most, c);
    if (most > kHaloMax) return;
    p.halo_cap = (most + 7) / 8 * 8;
    p.ctas = s.ctas;
    if (!chip_schedulable<double>(p, sm_count) || !chip_schedulable<float>(p, sm_count)) p.ctas = 0;
}

template <typename T>
void chip_launch(const ChipArgs<T>& a, cudaStream_t s) {
    const ChipPlan& p = a.plan;
    CP_CHECK(p.ctas > 0, CP_ERR_INVALID, "on-chip CG: the instance does not fit");
    const size_t smem = chip_smem(p.grid, p.spc, p.wmax, p.halo_cap, sizeof(T));
    cudaLaunchAttribute attr[1];
    if (p.grid) {
        cudaLaunchConfig_t cfg = chip_config(k_chip<T, true>, p, smem, attr, s);
        CP_CUDA(cudaLaunchKernelEx(&cfg, k_chip<T, true>, a));
    } else {
        cudaLaunchConfig_t cfg = chip_config(k_chip<T, false>, p, smem, attr, s);
        CP_CUDA(cudaLaunchKernelEx(&cfg, k_chip<T, false>, a));
    }
}

template void chip_launch<double>(const ChipArgs<double>&, cudaStream_t);
template void chip_launch<float>(const ChipArgs<float>&, cudaStream_t);

}  // namespace cp
