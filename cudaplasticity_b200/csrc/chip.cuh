// Device side of the on-chip CG (cg_chip.cu): what its kernels share.
#pragma once

#include "cg.h"
#include "common.cuh"

namespace cp {

namespace {

constexpr int kRegBlocks = 9;        // blocks of a row in registers (a 4-node mesh's interior row)
constexpr int kChipWarps = 12;       // 384 threads of 168 registers per CTA
constexpr int kMaxCluster = 16;
constexpr int kSums = 5;
constexpr int kMaxPolls = 8;         // warps that poll the CTAs' sums (grid): up to 256 CTAs
constexpr int kHaloMax = 4096;       // halo nodes per CTA

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
__device__ __forceinline__ void bar_init(unsigned int bar, unsigned int arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(arrivals) : "memory");
}
// One arrival at another CTA's mbarrier, after all that the thread (and, past
// a block barrier, its block) has read and written.
__device__ __forceinline__ void bar_arrive_remote(unsigned int bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
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

// Two words of (32 bits of data, sequence number): a word is its own flag, as in
// the low-latency protocol of collective libraries (NCCL's LL). What it rests
// on is that each 8-byte half of a 16-byte access is written and read whole.
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

// Of a wait that has taken some rounds: whether it has lasted longer than
// limit nanoseconds since its first call (t0, 0 before).
__device__ __forceinline__ bool waited(unsigned long long& t0, unsigned long long limit) {
    const unsigned long long t = global_ns();
    if (t0 == 0) t0 = t;
    return t - t0 > limit;
}

// Polls N word pairs per lane until those of every lane of the warp carry seq;
// false after `limit` nanoseconds (looked at every 256 rounds). The whole warp
// takes part, with valid addresses in every lane: left to diverge, a warp of
// which some lanes polled and some did not took 3700 cycles to come together
// again.
template <int N>
__device__ __forceinline__ bool poll(const uint4* p, size_t stride, unsigned int seq, unsigned long long limit, uint4* c) {
    unsigned long long t0 = 0;
    for (unsigned int round = 1;; ++round) {
        bool ok = true;
#pragma unroll
        for (int i = 0; i < N; ++i) c[i] = ld_words(p + i * stride);
#pragma unroll
        for (int i = 0; i < N; ++i) ok = ok && c[i].y == seq && c[i].w == seq;
        if (__all_sync(0xffffffffu, ok)) return true;
        if ((round & 255u) == 0u && __any_sync(0xffffffffu, waited(t0, limit))) return false;
    }
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

// A CTA's static shared memory for the exchange.
struct CommShared {
    double wsum[16][8];                              // per warp: its sums (unused warps stay zero)
    double gsum[kMaxPolls][8];                       // grid, the adding CTA: the same of the CTAs' sums
    __align__(16) double part[2][kMaxCluster][6];    // cluster: every CTA's sums (0, 2, 1, -, 3, 4), by parity
    __align__(8) unsigned long long bar[2];          // cluster: they have arrived, and the records are written
    Step step;
    int fail;                                        // cluster: some CTA of it gave up
};

// The exchange of one iteration: the own records and sums out, the halo
// records and the next step in.
template <typename T, bool GRID>
struct Comm {
    using V2 = typename Vec2<T>::type;
    static constexpr int NR = Record<T>::n;
    CommShared& S;
    const int tid, nthr, lane, w, rank, ctas;
    int own;
    unsigned int rec_base = 0;  // cluster: records [2][3][own]
    uint4 *ll_rec, *ll_part, *ll_step;
    size_t slots;
    unsigned long long wait_ns;
    unsigned int seq_skew;
    unsigned int seq = 0;
    int par = 1;             // parity of the last exchange
    unsigned int phase = 0;  // of the mbarriers' next wait
    bool failed = false;

    // Once per kernel, whole block (cluster: whole cluster).
    __device__ __forceinline__ void init() {
        if (tid == 0) S.fail = 0;
        for (int i = tid; i < 128; i += nthr) (&S.wsum[0][0])[i] = 0.0;
        for (int i = tid; i < kMaxPolls * 8; i += nthr) (&S.gsum[0][0])[i] = 0.0;
        for (int i = tid; i < 2 * kMaxCluster * 6; i += nthr) (&S.part[0][0][0])[i] = 0.0;
        if constexpr (GRID) {
            __syncthreads();
        } else {
            if (tid == 0) {
                bar_init(smem_addr(&S.bar[0]), ctas + 1);  // every CTA's arrival and the own bar_expect
                bar_init(smem_addr(&S.bar[1]), ctas + 1);
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
                bar_expect(smem_addr(&S.bar[0]), 48u * ctas);
                bar_expect(smem_addr(&S.bar[1]), 48u * ctas);
            }
            cluster_arrive_release();
            cluster_wait();
        }
    }
    // Where the record of halo slot s is read: cluster address, or the slot (grid).
    __device__ __forceinline__ unsigned int halo_at(int s) const {
        if (GRID) return (unsigned int)s;
        const int cr = s / own;
        return mapa(rec_base + (unsigned int)((s - cr * own) * sizeof(V2)), cr);
    }
    // The record at `at` of the last exchange (whole warps, valid addresses).
    __device__ __forceinline__ void read_halo(unsigned int at, V2* q) {
        if constexpr (GRID) {
            uint4 c[NR];
            if (failed || !poll<NR>(ll_rec + (size_t)par * NR * slots + at, slots, seq, wait_ns, c)) {
                failed = true;  // (of a block that has given up: no further waits)
                return;
            }
            Record<T>::get(c, q);
        } else {
            const unsigned int s = at + (unsigned int)(par * 3 * own * sizeof(V2));
#pragma unroll
            for (int i = 0; i < 3; ++i) ld_cluster(s + (unsigned int)(i * own * sizeof(V2)), q[i]);
        }
    }
    // Between begin() and the sums: the record of the own node loc.
    __device__ __forceinline__ void begin() {
        par ^= 1;
        if (GRID) seq += 1;
    }
    __device__ __forceinline__ void put_record(V2* rec, int loc, V2 u, V2 mw, V2 mk) {
        if constexpr (GRID) {
            Record<T>::put(ll_rec + (size_t)par * NR * slots + (size_t)rank * own + loc, slots, u, mw, mk,
                           seq + seq_skew);
        } else {
            V2* o = rec + (size_t)par * 3 * own + loc;
            o[0] = u;
            o[own] = mw;
            o[2 * own] = mk;
        }
    }
    // The sums v of the thread out, the next step in (S.step); `halo` reads the
    // first halo records meanwhile. decide (cluster: warp 0 of every CTA; grid:
    // the adding CTA) makes the step of the totals.
    template <typename Halo, typename Decide>
    __device__ __forceinline__ void finish(const double* v, Halo halo, Decide decide) {
        {
            const double s = warp_sum5(v, lane);
            if ((lane & 3) == 0) S.wsum[w][lane >> 2] = s;
        }
        __syncthreads();
        // The records are plain stores of all warps, which st.async does not
        // publish: every CTA releases its own by an arrival at every CTA's
        // mbarrier (whose waits acquire), from the warp farthest from the sums:
        // 0.06 us of an iteration at 4160 nodes, 0.02 at 1024.
        if constexpr (!GRID)
            if (w == (nthr >> 5) - 1 && lane < ctas && seq_skew == 0u) bar_arrive_remote(mapa(smem_addr(&S.bar[par]), lane));
        // lane (g, j): slot j of the warps g, g + 4, ..; then over g
        const int j = lane & 7, g = lane >> 3;
        double s = 0.0;
        if (w == 0) {
            s = (S.wsum[g][j] + S.wsum[g + 4][j]) + S.wsum[g + 8][j];
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 16);
        }
        if constexpr (GRID) {
            uint4* pp = ll_part + (size_t)par * 8 * ctas;
            // slots 0, 1, 2, 4, 6 hold the values 0, 2, 1, 3, 4
            const int val = lane == 1 ? 2 : lane == 2 ? 1 : lane > 2 ? lane / 2 + 1 : 0;
            if (w == 0 && (lane < 3 || lane == 4 || lane == 6)) post(pp + (size_t)val * ctas + rank, s, seq + seq_skew);
            if (w == 0) {
                uint4 c[1];
                if (!poll<1>(ll_step + par * 4 + min(lane, kStepWords - 1), 1, seq, wait_ns, c)) failed = true;
                const double q = word_value(c[0]);
                if (lane == 0) S.step.alpha = q;
                if (lane == 1) S.step.beta = q;
                if (lane == 2) S.step.go = (int)q;
            }
            halo();
        } else {
            if (w == 0) {
                // sums (0, 2), (1, 1), (3, 4) to every CTA
                const double s2 = __shfl_sync(0xffffffffu, s, j == 4 ? 6 : j + 1);
                if (!(j & 1) && j < 6 && seq_skew == 0u) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (g + 4 * i < ctas)
                            st_async(mapa(smem_addr(&S.part[par][rank][j]), g + 4 * i),
                                     mapa(smem_addr(&S.bar[par]), g + 4 * i), s, s2);
                }
            }
            {
                const unsigned int ba = smem_addr(&S.bar[par]);
                unsigned long long t0 = 0;
                while (!bar_try(ba, phase)) {
                    if (__builtin_expect(waited(t0, wait_ns), 0)) {
                        failed = true;
                        break;
                    }
                }
            }
            if (par) phase ^= 1u;
            halo();
            if (w == 0) {
                if (lane == 0) bar_expect(smem_addr(&S.bar[par]), 48u * ctas);  // its next use
                // lane (g, j): value j of the CTAs g, g + 4, ..; then over g
                const int e = j < 6 ? j : 0;
                s = (S.part[par][g][e] + S.part[par][g + 4][e]) + (S.part[par][g + 8][e] + S.part[par][g + 12][e]);
                s += __shfl_xor_sync(0xffffffffu, s, 8);
                s += __shfl_xor_sync(0xffffffffu, s, 16);
                double tot[kSums];
#pragma unroll
                for (int i = 0; i < kSums; ++i)
                    tot[i] = __shfl_sync(0xffffffffu, s, i == 0 ? 0 : i == 1 ? 2 : i == 2 ? 1 : i + 1);
                const Step st = decide(tot);
                if (lane == 0) S.step = st;
            }
        }
        failed = __syncthreads_or(failed ? 1 : 0) != 0;
    }
    // Cluster: at the end of a solve, whole cluster: all CTAs have read each
    // other's shared memory for the last time; whether any of them gave up.
    // This and init() hold the only cluster barriers, so that a CTA that gives
    // up meets the others here wherever they are (their next wait runs out
    // too). The flag is sent to every CTA before the barrier and read from the
    // own memory after it, when the others may have gone.
    __device__ __forceinline__ bool close() {
        if (failed && tid < ctas)
            asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(mapa(smem_addr(&S.fail), tid)) : "memory");
        cluster_arrive_release();
        cluster_wait();
        return *(volatile int*)&S.fail != 0;
    }
    // Grid: the adding CTA's side of one exchange.
    template <typename Decide>
    __device__ __forceinline__ void lead(Decide decide) {
        begin();
        const uint4* pp = ll_part + (size_t)par * 8 * ctas;
        const int np = (ctas + 31) >> 5;
        for (int q = w; q < np; q += nthr >> 5) {
            double t[kSums];
            uint4 ch[kSums];
            const int c = 32 * q + lane;
            if (!poll<kSums>(pp + min(c, ctas - 1), ctas, seq, wait_ns, ch)) failed = true;
#pragma unroll
            for (int i = 0; i < kSums; ++i) t[i] = c < ctas ? word_value(ch[i]) : 0.0;
            const double r5 = warp_sum5(t, lane);
            if ((lane & 3) == 0) S.gsum[q][lane >> 2] = r5;
        }
        failed = __syncthreads_or(failed ? 1 : 0) != 0;
        if (w == 0) {
            double t = 0.0;
#pragma unroll
            for (int q = 0; q < kMaxPolls; ++q) t += S.gsum[q][lane & 7];
            double tot[kSums];
#pragma unroll
            for (int i = 0; i < kSums; ++i) tot[i] = __shfl_sync(0xffffffffu, t, sum_slot(i));
            const Step st = decide(tot);
            if (lane < kStepWords)
                post(ll_step + par * 4 + lane, lane == 0 ? st.alpha : lane == 1 ? st.beta : (double)st.go,
                     seq + seq_skew);
            if (lane == 0) S.step = st;
        }
        __syncthreads();
    }
};

// The rows of a thread's NPT nodes (node j of thread t is the CTA's node
// j nthr + t): the first kRegBlocks blocks of the first RN nodes in registers,
// the other blocks in shared memory, upper and lower rows apart. WIDE: rows
// may have more than kRegBlocks blocks; without, the first RN nodes' loops over
// the rest are left out, for the length of the code: 4160 nodes took 1.74 us per
// iteration so, 1.85 with them unrolled by 3 (1.80 now).
template <typename T, int NPT, int RN, bool WIDE>
struct ChipRows {
    using V2 = typename Vec2<T>::type;
    using V4 = typename Vec4<T>::type;
    static constexpr int W = kRegBlocks;
    V4 kr[RN][W];
    unsigned int li[RN][W];  // byte addresses in U
    int wd[NPT];
    V2 *klo, *khi;
    unsigned short* kidx;
    unsigned int u_base;
    int tid, nthr, extra;

    static __host__ __device__ size_t smem_blocks(int nthr, int wmax) {
        return (size_t)nthr * ((size_t)(wmax > W ? wmax - W : 0) * RN + (size_t)wmax * (NPT - RN));
    }
    __device__ __forceinline__ size_t at(int j, int k) const {
        return j < RN ? (size_t)((k - W) * RN + j) * nthr + tid
                      : (size_t)(extra * RN + k * (NPT - RN) + (j - RN)) * nthr + tid;
    }
    // mem: smem_blocks() blocks of values, then their local indexes
    __device__ __forceinline__ void init(V2* mem, unsigned int u, int wmax) {
        const size_t nb = smem_blocks(nthr, wmax);
        klo = mem;
        khi = mem + nb;
        kidx = reinterpret_cast<unsigned short*>(mem + 2 * nb);
        u_base = u;
        extra = wmax > W ? wmax - W : 0;
#pragma unroll
        for (int j = 0; j < NPT; ++j) {
            wd[j] = 0;
            if (j < RN)
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    kr[j][k].x = kr[j][k].y = kr[j][k].z = kr[j][k].w = (T)0;
                    li[j][k] = u + (j * nthr + tid) * (unsigned int)sizeof(V2);
                }
        }
    }
    // Node j: its blocks from block(k) (K's value of block k), lx the plan's
    // indexes (stride 32).
    template <typename Block>
    __device__ __forceinline__ void load(int j, int width, const unsigned short* lx, Block block) {
        if (j < RN) {
#pragma unroll
            for (int k = 0; k < W; ++k)
                if (k < width) {
                    kr[j][k] = block(k);
                    li[j][k] = u_base + lx[32 * k] * (unsigned int)sizeof(V2);
                }
        }
        for (int k = j < RN ? W : 0; k < width; ++k) {
            const V4 q = block(k);
            const size_t a = at(j, k);
            V2 lo, hi;
            lo.x = q.x; lo.y = q.y; hi.x = q.z; hi.y = q.w;
            klo[a] = lo;
            khi[a] = hi;
            kidx[a] = lx[32 * k];
        }
        wd[j] = width;
    }
    // Row j times U. (One fused chain per component, two operations per block
    // in place of three, is no faster and its rounding error is up to 1.4 times
    // as large; two chains per component cost the grid forms 10%.)
    __device__ __forceinline__ V2 gather(int j) const {
        V2 s;
        s.x = s.y = (T)0;
        if (j < RN) {
#pragma unroll
            for (int k = 0; k < W; ++k) {
                V2 c;
                ld_u(li[j][k], c);
                s.x += kr[j][k].x * c.x + kr[j][k].y * c.y;
                s.y += kr[j][k].z * c.x + kr[j][k].w * c.y;
            }
        }
        if (WIDE || j >= RN)
#pragma unroll(WIDE ? 3 : 1)
            for (int k = j < RN ? W : 0; k < wd[j]; ++k) {
                const size_t a = at(j, k);
                const V2 lo = klo[a], hi = khi[a];
                V2 c;
                ld_u(u_base + kidx[a] * (unsigned int)sizeof(V2), c);
                s.x += lo.x * c.x + lo.y * c.y;
                s.y += hi.x * c.x + hi.y * c.y;
            }
        return s;
    }
};

}  // namespace

}  // namespace cp
