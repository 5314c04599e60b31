// CG launch interface (kernels in cg.cu).
#pragma once

#include "internal.h"

namespace cp {

template <typename T>
struct Vec2;
template <>
struct Vec2<double> {
    using type = double2;
};
template <>
struct Vec2<float> {
    using type = float2;
};
template <typename T>
struct Vec4;
template <>
struct Vec4<double> {
    using type = double4;
};
template <>
struct Vec4<float> {
    using type = float4;
};

// Everything the CG kernels touch, passed by value.
template <typename T>
struct CgArgs {
    using V2 = typename Vec2<T>::type;
    int n = 0;            // nodes (2 DOFs each)
    int sm_count = 148;
    int max_blocks = 0;   // capacity of the partials buffer (blocks)
    const int* slice_ptr = nullptr;  // sliced layout (see DevCsr)
    const int* scol = nullptr;
    const T* val = nullptr;         // K in the recurrence type, 4 values per block
    const double2* b = nullptr;     // right-hand side (FP64)
    const uchar2* mask = nullptr;   // 1 = free DOF
    double2* x = nullptr;           // solution, accumulated in FP64
    V2* r = nullptr;
    typename Vec4<T>::type* minv = nullptr;  // inverse 2x2 diagonal blocks (block Jacobi only)
    int precond = 0;                // 0: plain CG (reference), 1: 2x2 block-Jacobi PCG
    // per node (v, z): v = M^-1 r (r without the preconditioner), z the
    // direction; by iteration parity
    typename Vec4<T>::type* rec0 = nullptr;
    typename Vec4<T>::type* rec1 = nullptr;
    V2* zn = nullptr;               // z' from P to U
    V2* q = nullptr;
    CgScalars* sc = nullptr;
    double* partials = nullptr;     // >= 3 * max_blocks doubles
};

// Time limit of every wait between CTAs (an exchange takes microseconds).
constexpr unsigned long long kWaitNs = 2000000000ull;

// The upper half of K for cg_fused.cu's iterations: per slice of 32 nodes, u
// slots of the diagonal block and of those right of it, and l of those left of
// it, as many in every slice as the mesh's widest row takes.
struct HalfK {
    int u = 0, l = 0;
    unsigned short* width = nullptr;  // per slice: upper blocks | lower blocks << 8
    int* ucol = nullptr;              // per upper slot: its column (the node itself: padding)
    unsigned int* low = nullptr;      // per lower slot: its column and its mirror's upper slot
    double2* val = nullptr;           // per upper slot: the block, rewritten by every solve's start; null: not in use
};

// Of a numbering: HalfK's u and l, and the slices whose rows are all within the
// iterations' straight-line code.
struct HalfCount {
    int u, l, straight;
};

// The single-launch FP64 iteration of cg_fused.cu.
struct FusedArgs {
    int n = 0;
    int sm_count = 148;
    int max_blocks = 0;              // capacity of partials (blocks, 6 sums each)
    const int* slice_ptr = nullptr;
    const int* scol = nullptr;
    const double* val = nullptr;
    const double2* b = nullptr;
    const uchar2* mask = nullptr;
    double2* x = nullptr;
    double2 *r = nullptr, *w = nullptr, *p = nullptr, *kp = nullptr;
    double2 *gA = nullptr, *gB = nullptr;  // per node: u, M w, M kp (by parity)
    double4* minv = nullptr;
    int precond = 0;
    HalfK half;
    CgScalars* sc = nullptr;
    double* partials = nullptr;
    // persistent form only: time limit of each grid-barrier wait, and the
    // number of extra steps every wait asks for (0; 1 makes each wait ask for
    // a step that is never released, so that every wait runs out: the
    // time-out path's test)
    unsigned long long barrier_ns = kWaitNs;
    unsigned int barrier_skew = 0;
};

// The upper half of K: whether the iterations of an instance may read it, its
// widths (count: zero before; a.half.width is written), whether they do in this
// numbering, and, once it has its arrays, its columns.
bool fused_wants_half(int n, int wmax);
bool fused_half_pays(const HalfCount& c, int n);
size_t fused_half_bytes(int n);  // its arrays at their largest
void fused_half_widths(const FusedArgs& a, HalfCount* count, cudaStream_t s);
void fused_half_columns(const FusedArgs& a, cudaStream_t s);
void fused_launch_start(const FusedArgs& a, double eps2, long long max_iter, cudaStream_t s);
void fused_launch_iteration(const FusedArgs& a, int parity, cudaStream_t s);
// The whole solve (init, first step, iterations) as one cooperative launch;
// only when its grid is that of the kernels above (fused_persistent_fits).
bool fused_persistent_fits(const FusedArgs& a);
void fused_launch_persistent(const FusedArgs& a, double eps2, long long max_iter, cudaStream_t s);
cudaGraphExec_t fused_build_while_graph(const FusedArgs& a, int body_iters, cudaStream_t s);

// CgScalars.status of an FP32 on-chip solve whose step lost its curvature
// (internal: never returned to a caller).
constexpr int CP_ERR_DEGENERATE = 100;
// Of an on-chip solve that its budget of iterations has cut (internal too).
constexpr int CP_CHIP_CUT = 101;

// The whole linear solve on chip (cg_chip.cu): one thread-block cluster, or
// a cooperative grid of up to one CTA per SM.
struct ChipShape {
    bool grid = false;
    int ctas = 0;  // 0: the instance does not fit
    int spc = 0;   // slices of 32 nodes per CTA
    int npt = 1;   // nodes per thread
    int wmax = 0;  // widest node row, in blocks
};
struct ChipPlan {
    bool grid = false;
    int ctas = 0, spc = 0, npt = 1, wmax = 0;
    int halo_cap = 0;                // most halo nodes of a CTA (rounded up)
    unsigned char* mem = nullptr;    // chip_plan_bytes() bytes that hold the following
    int* order = nullptr;            // per slot (CTA, thread): its node, or -1
    unsigned short* lidx = nullptr;  // per block of a slot's row: index of its column in the CTA's U
    int* halo = nullptr;             // per CTA: the slots of its halo nodes
    int* halo_cnt = nullptr;         // per CTA
    unsigned char* pub = nullptr;    // per slot: in another CTA's halo
};
template <typename T>
struct ChipArgs {
    ChipPlan plan;
    const int* slice_ptr = nullptr;
    const int* scol = nullptr;
    const double* val64 = nullptr;
    const double2* b = nullptr;
    const uchar2* mask = nullptr;
    double2* x = nullptr;
    int precond = 0;
    CgScalars* sc = nullptr;
    double eps2 = 0.0, outer_eps2 = -1.0;  // as cg_launch_init
    long long max_iter = 0;
    int relative_to_r0 = 0;
    // grid form: at most `budget` iterations. A solve that this cuts ends with
    // CP_CHIP_CUT, its vectors in `state` (r, p, kp, w, u: 5 n pairs of T) and
    // its last records in the exchange buffers, and another launch with resume
    // = 1 goes on exactly where it was.
    long long budget = 0x7fffffffLL;
    void* state = nullptr;
    int n = 0, resume = 0;
    // with inc: the solve's increment x - u0 is left there (recycle.h)
    const double2* u0 = nullptr;
    double2* inc = nullptr;
    // grid exchange: records, sums and steps by parity, the last sequence
    // number in use; both exchanges: the time limit of a wait, and what is
    // added to the posted sequence numbers (0; with 1 every wait runs out, in
    // the cluster because nothing is sent: the time-out path's test)
    uint4 *ll_rec = nullptr, *ll_part = nullptr, *ll_step = nullptr;
    unsigned int* seq = nullptr;
    unsigned long long wait_ns = kWaitNs;
    unsigned int seq_skew = 0;
};
ChipShape chip_shape(int n, int wmax, int sm_count, bool grid);
size_t chip_plan_bytes(const ChipShape& s, int n);
size_t chip_ll_bytes(const ChipShape& s);
void chip_ll_carve(const ChipPlan& p, void* mem, uint4** rec, uint4** part, uint4** step);
// In p.mem; scratch: 2 n pairs. for_solve: checks that k_chip can run the plan
// (a batch brings its own kernel).
void chip_build_plan(ChipPlan& p, const ChipShape& s, uint2* scratch, int n, const double2* xy, const int* slice_ptr,
                     const int* scol, int sm_count, cudaStream_t st, bool for_solve);
template <typename T>
void chip_launch(const ChipArgs<T>& a, cudaStream_t s);
// The largest plan of an instance in a batch (batch.cu).
size_t batch_plan_bytes(int n, int wmax);

template <typename T>
void cg_launch_init(const CgArgs<T>& a, const void* valA, bool valA_is_fp64, double eps2, long long max_iter,
                    int relative_to_r0, double outer_eps2, cudaStream_t s);
template <typename T>
void cg_launch_iteration(const CgArgs<T>& a, int parity, cudaStream_t s);
template <typename T>
void cg_launch_p(const CgArgs<T>& a, int parity, cudaStream_t s);
template <typename T>
void cg_launch_u(const CgArgs<T>& a, int parity, cudaStream_t s);
template <typename T>
cudaGraphExec_t cg_build_while_graph(const CgArgs<T>& a, int body_iters, cudaStream_t s);

}  // namespace cp
