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
//     two) together with one arrival of each CTA, which releases its records;
//     every CTA adds up all CTAs' sums in the same order, so all hold the same
//     scalars and take the same branches.
//   grid (up to one CTA per SM, a cooperative launch): records and sums go
//     through global memory (L2) in 8-byte words of 32 bits of data and their
//     sequence number, so that a reader polls the data itself: one trip
//     through L2 and no fence. One more CTA, without nodes, adds up the sums
//     and posts the next step's scalars (all CTAs reading all CTAs' sums takes
//     twice as long at 63 CTAs and more beyond: every poll then meets every
//     other on the same lines).
// Every wait of both is limited in time (kWaitNs); a CTA that gives up sets
// sc->chip_err and returns, and so do the others at their next wait.
// T is the type of K's values and of the recurrences (double, or float in the
// mixed mode); x is FP64 and every sum is accumulated and reduced in FP64.
#include <cstdlib>

#include "cg.h"
#include "chip.cuh"
#include "common.cuh"
#include "internal.h"

namespace cp {

namespace {

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

// One block per CTA of the solve: its nodes by node number, so that the
// neighbours of consecutive threads tend to be consecutive too (the gathers'
// shared-memory banks, the halo records' order): 4160 nodes 1.85 -> 1.74 us.
__global__ void __launch_bounds__(kPlanThreads) k_chip_local(int own, int* order, int* slot_of) {
    extern __shared__ int ids[];
    const int s0 = blockIdx.x * own;
    for (int i = threadIdx.x; i < own; i += blockDim.x) ids[i] = order[s0 + i];
    __syncthreads();
    for (int i = threadIdx.x; i < own; i += blockDim.x) {
        const unsigned int id = (unsigned int)ids[i];  // -1 sorts last
        int at = 0;
        for (int q = 0; q < own; ++q) at += ((unsigned int)ids[q] < id || ((unsigned int)ids[q] == id && q < i)) ? 1 : 0;
        order[s0 + at] = (int)id;
        if ((int)id >= 0) slot_of[id] = s0 + at;
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

// ---------------------------------------------------------------- kernel --

// NPT nodes per thread; of the second one (double) the whole row lies in
// shared memory.
template <typename T, bool GRID, int NPT, bool WIDE>
__global__ void __launch_bounds__(kChipWarps * 32, 1) k_chip(ChipArgs<T> a) {
    using V2 = typename Vec2<T>::type;
    using V4 = typename Vec4<T>::type;
    constexpr int RN = sizeof(T) == 4 ? NPT : 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ CommShared cs;
    const ChipPlan& P = a.plan;
    const int tid = threadIdx.x, nthr = blockDim.x, w = tid >> 5;
    const int rank = blockIdx.x, ctas = P.ctas, own = nthr * NPT;
    const bool adder = GRID && rank == ctas;  // the CTA without nodes
    Comm<T, GRID> comm{cs,        tid,       nthr,      tid & 31,          w,           rank,        ctas,
                       own,       0u,        a.ll_rec,  a.ll_part,         a.ll_step,   (size_t)ctas * own,
                       a.wait_ns, a.seq_skew};
    // shared memory: U [own + halo], then (cluster) records [2][3][own], then
    // the blocks that are not in registers
    V2* U = reinterpret_cast<V2*>(smem_raw);
    V2* rec = U + own + P.halo_cap;
    comm.rec_base = smem_addr(rec);
    ChipRows<T, NPT, RN, WIDE> rows;
    rows.tid = tid;
    rows.nthr = nthr;
    rows.init(rec + (GRID ? 0 : 6 * own), smem_addr(U), P.wmax);

    // ---- rows, r = m.(b - K x), M
    int n[NPT];
    double2 x[NPT];
    uchar2 m[NPT];
    V2 r[NPT], p[NPT], kp[NPT], wv[NPT], u[NPT];
    T mi0[NPT], mi1[NPT], mi2[NPT];  // M, symmetric as K is: m00, m01 = m10, m11
    bool publish[NPT];
    double v[kSums] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int j = 0; j < NPT; ++j) {
        const int slot = rank * own + j * nthr + tid;
        n[j] = adder ? -1 : P.order[slot];
        x[j] = make_double2(0.0, 0.0);
        m[j] = make_uchar2(0, 0);
        r[j] = p[j] = kp[j] = wv[j] = u[j] = make2<V2>(0, 0);
        mi0[j] = mi1[j] = mi2[j] = (T)0;
        publish[j] = false;
        if (n[j] < 0) continue;
        const int nd = n[j], base = a.slice_ptr[nd >> 5] + (nd & 31);
        m[j] = a.mask[nd];
        x[j] = a.x[nd];
        publish[j] = P.pub[slot] != 0;
        double k0 = 0.0, k1 = 0.0;
        double4 diag = make_double4(0.0, 0.0, 0.0, 0.0);
        rows.load(j, (a.slice_ptr[(nd >> 5) + 1] - base + 31) >> 5,
                  P.lidx + (size_t)(slot >> 5) * P.wmax * 32 + (tid & 31), [&](int k) {  // r in FP64, also for float
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
                  });
        const double2 bb = a.b[nd];
        const double r0 = m[j].x ? bb.x - k0 : 0.0, r1 = m[j].y ? bb.y - k1 : 0.0;
        r[j] = make2<V2>((T)r0, (T)r1);
        if (a.precond) {  // inverse of the diagonal block on the free DOFs
            if (m[j].x && m[j].y) {
                const double det = diag.x * diag.w - diag.y * diag.z;
                mi0[j] = (T)(diag.w / det);
                mi1[j] = (T)(-diag.y / det);
                mi2[j] = (T)(diag.x / det);
            } else if (m[j].x) {
                mi0[j] = (T)(1.0 / diag.x);
            } else if (m[j].y) {
                mi2[j] = (T)(1.0 / diag.w);
            }
        } else {
            mi0[j] = (T)(m[j].x ? 1 : 0);
            mi2[j] = (T)(m[j].y ? 1 : 0);
        }
        u[j] = make2<V2>(mi0[j] * r[j].x + mi1[j] * r[j].y, mi1[j] * r[j].x + mi2[j] * r[j].y);
        v[0] += (double)r[j].x * (double)r[j].x + (double)r[j].y * (double)r[j].y;
        v[1] += bb.x * bb.x + bb.y * bb.y;
        v[2] += r0 * r0 + r1 * r1;
        if (GRID && a.resume) {
            const V2* st = static_cast<const V2*>(a.state) + nd;
            r[j] = st[0];
            p[j] = st[(size_t)a.n];
            kp[j] = st[2 * (size_t)a.n];
            wv[j] = st[3 * (size_t)a.n];
            u[j] = st[4 * (size_t)a.n];
        }
    }
    // ---- halo: thread nthr - 1 - tid takes the first halo nodes, so that the
    // warps that wait for the sums have few of them; past the last halo node a
    // thread reads the last one again, so that whole warps read
    const int hc = adder ? 0 : P.halo_cnt[rank], h0 = nthr - 1 - tid, h_min = nthr - 32 * (w + 1);
    const int* hl = P.halo + (size_t)rank * kHaloMax;
    const unsigned int ha = hc > 0 ? comm.halo_at(hl[min(h0, hc - 1)]) : 0u;
    V2 hr[3];
    if constexpr (GRID) {
        comm.seq = *a.seq;
        comm.par = comm.seq & 1u;  // by the number, so that a solve that goes on finds its records
    }
    // ---- the scalars of the solve: warp 0 (grid: of the adding CTA)
    double rr = 0.0, rho = 0.0, rho_inv = 0.0, bnorm2 = 0.0, res64 = 0.0, normB_inv = 0.0;
    int status = 0, converged = 0, lin_done = 0;
    int iter = 0;
    if (adder && a.resume) {
        rho = a.sc->rho;
        bnorm2 = a.sc->bb;
        res64 = a.sc->res64;
        normB_inv = a.sc->normB_inv;
        iter = a.sc->iter;
    }
    const long long most = 0x7fffffffLL;
    const int max_iter = (int)(a.max_iter < most ? a.max_iter : most);
    const int cap = GRID ? (int)min((long long)max_iter, iter + a.budget) : max_iter;
    comm.init();

    auto apply_m = [&](int j, V2 q) { return make2<V2>(mi0[j] * q.x + mi1[j] * q.y, mi1[j] * q.x + mi2[j] * q.y); };
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
        const int go = (int)(rr * normB_inv > a.eps2) & (int)(iter < cap) & (int)(den > 0.0) & (int)(g > 0.0);
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
        if (comm.failed) {
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
            } else if (iter >= cap) status = CP_CHIP_CUT;
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
        sc->alpha = cs.step.alpha;
        sc->beta = cs.step.beta;
        sc->rho = rho;
        sc->ticket = 0;
        if (GRID) *a.seq = comm.seq;  // every CTA has read the old value: all have taken part in an exchange
    };
    auto exchange = [&](auto decide_now) {
        comm.begin();
#pragma unroll
        for (int j = 0; j < NPT; ++j)
            if (publish[j]) comm.put_record(rec, j * nthr + tid, u[j], apply_m(j, wv[j]), apply_m(j, kp[j]));
        comm.finish(
            v, [&] { if (h_min < hc) comm.read_halo(ha, hr); }, decide_now);
    };
    // U of the own nodes and of the halo at step (al, bt).
    auto fill_u = [&](T al, T bt) {
#pragma unroll
        for (int j = 0; j < NPT; ++j) U[j * nthr + tid] = u[j];
        if (h0 < hc)
            U[own + h0] = make2<V2>(hr[0].x - al * (hr[1].x + bt * hr[2].x), hr[0].y - al * (hr[1].y + bt * hr[2].y));
        if (hc > nthr) {
            for (int b = nthr; h_min + b < hc; b += nthr) {
                const int h = h0 + b;
                comm.read_halo(comm.halo_at(hl[min(h, hc - 1)]), hr);
                if (h < hc)
                    U[own + h] = make2<V2>(hr[0].x - al * (hr[1].x + bt * hr[2].x),
                                           hr[0].y - al * (hr[1].y + bt * hr[2].y));
            }
            if (GRID) comm.failed = __syncthreads_or(comm.failed ? 1 : 0) != 0;
        }
        __syncthreads();
    };

    if (adder) {
        auto lead = [&](auto decide_now) {
            comm.lead(decide_now);
            return cs.step.go != 0 && !comm.failed;
        };
        if (a.resume || (lead(decide_init) && lead(decide_first))) {
            do {
                rho_inv = __drcp_rn(rho);
            } while (lead(decide));
        }
        finish();
        return;
    }
    // ---- (r, r), (b, b), and u to the neighbours
    bool go = true;
    if (GRID && a.resume) {
        // the last exchange's records are where they were, and the step that
        // it made is in sc
        if (tid == 0) cs.step = {a.sc->alpha, a.sc->beta, 1};
        if (h_min < hc) comm.read_halo(ha, hr);
        go = __syncthreads_or(comm.failed ? 1 : 0) == 0;
        comm.failed = !go;
    } else {
        exchange(decide_init);
        fill_u((T)0, (T)0);
        go = cs.step.go != 0 && !comm.failed;
        if (go) {
            // ---- first step: w = K u; gamma = (r, u), delta = (w, u)
            v[0] = v[1] = v[2] = 0.0;
#pragma unroll
            for (int j = 0; j < NPT; ++j) {
                wv[j] = rows.gather(j);
                v[0] += (double)r[j].x * (double)u[j].x + (double)r[j].y * (double)u[j].y;
                v[1] += (double)wv[j].x * (double)u[j].x + (double)wv[j].y * (double)u[j].y;
            }
            exchange(decide_first);
            go = cs.step.go != 0 && !comm.failed;
        }
    }
    // ---- iterations
    while (go) {
        const double alpha = cs.step.alpha;
        if (!GRID) rho_inv = __drcp_rn(rho);  // for the next decision, off its path
        const T al = (T)alpha, bt = (T)cs.step.beta;
        V2 u0[NPT];
#pragma unroll
        for (int j = 0; j < NPT; ++j) {
            u0[j] = u[j];
            const V2 mw = apply_m(j, wv[j]), mk = apply_m(j, kp[j]);
            u[j] = make2<V2>(u0[j].x - al * (mw.x + bt * mk.x), u0[j].y - al * (mw.y + bt * mk.y));
        }
        fill_u(al, bt);
#pragma unroll
        for (int i = 0; i < kSums; ++i) v[i] = 0.0;
#pragma unroll
        for (int j = 0; j < NPT; ++j) {
            p[j] = make2<V2>(u0[j].x + bt * p[j].x, u0[j].y + bt * p[j].y);
            kp[j] = make2<V2>(wv[j].x + bt * kp[j].x, wv[j].y + bt * kp[j].y);
            x[j].x += alpha * (double)p[j].x;
            x[j].y += alpha * (double)p[j].y;
            if (m[j].x) r[j].x -= al * kp[j].x;
            if (m[j].y) r[j].y -= al * kp[j].y;
            wv[j] = rows.gather(j);
            const V2 wj = wv[j], uj = u[j], rj = r[j], pj = p[j], kj = kp[j];
            v[0] += (double)rj.x * (double)uj.x + (double)rj.y * (double)uj.y;
            v[1] += (double)wj.x * (double)uj.x + (double)wj.y * (double)uj.y;
            v[2] += (double)rj.x * (double)rj.x + (double)rj.y * (double)rj.y;
            v[3] += ((double)wj.x * (double)pj.x + (double)wj.y * (double)pj.y) +
                    ((double)kj.x * (double)uj.x + (double)kj.y * (double)uj.y);
            v[4] += (double)kj.x * (double)pj.x + (double)kj.y * (double)pj.y;
        }
        exchange(decide);
        go = cs.step.go != 0 && !comm.failed;
    }
    if constexpr (!GRID) {  // the others have read this CTA's memory for the last time
        cluster_arrive_release();
        cluster_wait();
    }
    if (comm.failed) {
        if (tid == 0) atomicExch(&a.sc->chip_err, 1);
        return;
    }
#pragma unroll
    for (int j = 0; j < NPT; ++j)
        if (n[j] >= 0) {
            a.x[n[j]] = x[j];
            if (a.inc) {
                const double2 b = a.u0[n[j]];
                a.inc[n[j]] = make_double2(x[j].x - b.x, x[j].y - b.y);
            }
            if (GRID && a.state) {
                V2* st = static_cast<V2*>(a.state) + n[j];
                st[0] = r[j];
                st[(size_t)a.n] = p[j];
                st[2 * (size_t)a.n] = kp[j];
                st[3 * (size_t)a.n] = wv[j];
                st[4 * (size_t)a.n] = u[j];
            }
        }
    if (!GRID && rank == 0) finish();
}

// Dynamic shared memory per CTA.
template <typename T, bool GRID, int NPT>
size_t chip_smem(const ChipPlan& p) {
    const int nthr = 32 * p.spc / NPT;
    const size_t own = (size_t)nthr * NPT;
    size_t b = (own + p.halo_cap) * 2 * sizeof(T);
    if (!GRID) b += 6 * own * 2 * sizeof(T);
    b += ChipRows<T, NPT, sizeof(T) == 4 ? NPT : 1, true>::smem_blocks(nthr, p.wmax) * (4 * sizeof(T) + 2);
    return (b + 15) / 16 * 16;
}

template <typename K>
cudaLaunchConfig_t chip_config(K, const ChipPlan& p, size_t smem, cudaLaunchAttribute* attr, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.ctas + (p.grid ? 1 : 0));  // the grid form's last CTA adds up the sums
    cfg.blockDim = dim3(32 * p.spc / p.npt);
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

template <typename T, bool GRID, int NPT, bool WIDE>
bool schedulable(const ChipPlan& p, int sm_count) {
    const auto k = k_chip<T, GRID, NPT, WIDE>;
    const size_t smem = chip_smem<T, GRID, NPT>(p);
    if (smem > kSmemCap || !chip_attributes(k, GRID)) return false;
    if (GRID) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * p.spc / NPT, smem) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return (long long)per_sm * sm_count >= p.ctas + 1;
    }
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = chip_config(k, p, smem, attr, nullptr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        return false;
    }
    return true;
}
template <typename T, bool WIDE>
bool chip_schedulable_as(const ChipPlan& p, int sm_count) {
    if (!p.grid) return schedulable<T, false, 1, WIDE>(p, sm_count);
    return p.npt == 2 ? schedulable<T, true, 2, WIDE>(p, sm_count) : schedulable<T, true, 1, WIDE>(p, sm_count);
}
template <typename T>
bool chip_schedulable(const ChipPlan& p, int sm_count) {
    return p.wmax > kRegBlocks ? chip_schedulable_as<T, true>(p, sm_count) : chip_schedulable_as<T, false>(p, sm_count);
}

}  // namespace

// The shape of the cluster (grid = false) or grid form for n nodes; ctas = 0
// when it does not hold them.
//   cluster: about 13 CTAs, of at least 4 slices. 1024 nodes: 8 CTAs of 4
//     slices 1.45 us per iteration, 16 of 2 1.9, 3 of 12 1.7; 4160 nodes: 13 of
//     10 1.74, 11 of 12 1.8 (the whole solve in one cluster with every
//     record read through distributed shared memory: 4.9 and 5.7). With the
//     records' release the forms taken have 1.49 and 1.80.
//   grid: about 128 CTAs, of at least 8 slices. 16104 nodes: 63 CTAs of 8
//     slices 3.31 us, 126 of 4 3.7, 42 of 12 3.7 (one launch per iteration,
//     cg_fused.cu: 10.2); 40200 nodes: 126 of 10 3.71, 105 of 12 3.8 (11.4).
//     Above 147 CTAs of 12, two nodes per thread: 65536 nodes 86 CTAs of 24
//     5.98 us (11.9); 99856 nodes 131 of 24 6.09 (16.3). At sizes that both
//     hold the cluster is the faster one (4160 nodes: 3.2 as a grid). With the
//     waits limited by time the forms taken have 3.06 (16256 nodes), 3.31 and
//     5.75.
ChipShape chip_shape(int n, int wmax, int sm_count, bool grid) {
    const int n_slices = (n + 31) / 32;
    ChipShape s;
    s.wmax = wmax;
    s.grid = grid;
    s.spc = grid ? std::max((n_slices + 127) / 128, 8) : std::max((n_slices + 12) / 13, 4);
    if (const char* e = std::getenv("CUPLAST_CHIP_FORM")) {  // c<slices per CTA> or g<slices per CTA> (measurements)
        const int v = std::atoi(e + 1);
        if ((e[0] == 'c' || e[0] == 'g') && v >= 1 && v <= (e[0] == 'g' ? 2 : 1) * kChipWarps) {
            if (grid != (e[0] == 'g')) return s;
            s.spc = v;
        }
    }
    const int most = grid ? std::min(sm_count - 1, 32 * kMaxPolls) : kMaxCluster;
    if (s.spc <= kChipWarps || !grid || (long long)most * kChipWarps >= n_slices) {
        s.spc = std::min(s.spc, kChipWarps);
    } else {  // two nodes per thread
        s.npt = 2;
        s.spc = 2 * kChipWarps;
    }
    s.ctas = (n_slices + s.spc - 1) / s.spc;
    if (s.ctas > most) s.ctas = 0;
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
void chip_build_plan(ChipPlan& p, const ChipShape& s, uint2* scratch, int n, const double2* xy, const int* slice_ptr,
                     const int* scol, int sm_count, cudaStream_t st, bool for_solve) {
    const size_t slots = chip_slots(s);
    p.grid = s.grid;
    p.spc = s.spc;
    p.npt = s.npt;
    p.wmax = s.wmax;
    p.ctas = 0;
    int* ints = reinterpret_cast<int*>(p.mem);
    p.order = ints;
    int* slot_of = ints + slots;
    p.halo = slot_of + n;
    p.halo_cnt = p.halo + (size_t)s.ctas * kHaloMax;
    p.lidx = reinterpret_cast<unsigned short*>(p.halo_cnt + s.ctas);
    p.pub = reinterpret_cast<unsigned char*>(p.lidx + slots * s.wmax);
    CP_CUDA(cudaMemsetAsync(p.pub, 0, slots, st));
    constexpr int order_smem = kDigits * kOrderThreads * (int)sizeof(unsigned int);
    CP_CUDA(cudaFuncSetAttribute(k_chip_order, cudaFuncAttributeMaxDynamicSharedMemorySize, order_smem));
    k_chip_order<<<1, kOrderThreads, order_smem, st>>>(n, (int)slots, xy, scratch, p.order, slot_of);
    k_chip_local<<<s.ctas, kPlanThreads, sizeof(int) * (size_t)s.spc * 32, st>>>(s.spc * 32, p.order, slot_of);
    k_chip_plan<<<s.ctas, kPlanThreads, 2 * sizeof(unsigned int) * (slots / 32), st>>>(
        (int)slots, s.spc * 32, s.wmax, slice_ptr, scol, p.order, slot_of, p.lidx, p.halo, p.halo_cnt, p.pub);
    CP_CUDA(cudaGetLastError());
    std::vector<int> cnt(s.ctas);
    CP_CUDA(cudaMemcpyAsync(cnt.data(), p.halo_cnt, sizeof(int) * s.ctas, cudaMemcpyDeviceToHost, st));
    CP_CUDA(cudaStreamSynchronize(st));
    int most = 0;
    for (int c : cnt) most = std::max(most, c);
    if (most > kHaloMax) return;
    p.halo_cap = (most + 7) / 8 * 8;
    p.ctas = s.ctas;
    if (for_solve && (!chip_schedulable<double>(p, sm_count) || !chip_schedulable<float>(p, sm_count))) p.ctas = 0;
}

namespace {
template <typename T, bool GRID, int NPT, bool WIDE>
void launch_as(const ChipArgs<T>& a, cudaStream_t s) {
    const auto k = k_chip<T, GRID, NPT, WIDE>;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = chip_config(k, a.plan, chip_smem<T, GRID, NPT>(a.plan), attr, s);
    CP_CUDA(cudaLaunchKernelEx(&cfg, k, a));
}
template <typename T, bool WIDE>
void launch_form(const ChipArgs<T>& a, cudaStream_t s) {
    if (!a.plan.grid) launch_as<T, false, 1, WIDE>(a, s);
    else if (a.plan.npt == 2) launch_as<T, true, 2, WIDE>(a, s);
    else launch_as<T, true, 1, WIDE>(a, s);
}
}  // namespace

template <typename T>
void chip_launch(const ChipArgs<T>& a, cudaStream_t s) {
    const ChipPlan& p = a.plan;
    CP_CHECK(p.ctas > 0, CP_ERR_INVALID, "on-chip CG: the instance does not fit");
    if (p.wmax > kRegBlocks) launch_form<T, true>(a, s);
    else launch_form<T, false>(a, s);
}

template void chip_launch<double>(const ChipArgs<double>&, cudaStream_t);
template void chip_launch<float>(const ChipArgs<float>&, cudaStream_t);

}  // namespace cp
