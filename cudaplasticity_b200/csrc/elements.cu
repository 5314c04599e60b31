// Element kernels: stiffness assembly into the node-blocked CSR, the fused
// strain / stress / secant update with the exit norm, Aitken relaxation of the
// secant iteration, and the plastic-strain post-processing.
//
// Element geometry is recomputed from node coordinates in every kernel (the
// reference stores B and detJ per Gauss point, 288 B per quad, computed once
// by calcBs4, src/PlasticitySolver.cu:139-144,1237-1246); reading 4 node
// coordinates costs less HBM traffic than reading B back.
#include <mutex>

#include "common.cuh"
#include "elements.cuh"
#include "internal.h"

namespace cp {

namespace {


constexpr int kAsmThreads = 128;  // = 4 slices of 32 nodes

// One thread per node, one block per tile of 4 slices. The tile's blocks are
// one contiguous range of values in the sliced layout, accumulated in shared
// memory (each thread only touches its own node's blocks: no atomics, and the
// summation order is the element order) and written out coalesced, once. The
// next incidence's element is loaded ahead of the current one's arithmetic.
// On the 1,048,576-quad plate 193 us (2.0 TB/s of its 386 MB) against 240
// before the bank-conflict-free accumulators and one block per tile in place of
// 8 per SM (6 fit: a second wave a third full); 4096 quads 10.3 against 12.4
// us. It is bound by its FP64 operations, about 600 per incidence (140 us at
// the full rate); fewer registers (5 or 6 blocks per SM) lose: 200, 216 us. The
// order of those operations is part of the result: a bilinear form in the
// nodes' signs takes 280 and 135 us, but moves K by an ulp, and solves whose
// linear iterations are capped then move by up to 1e-5 on meshes of near
// rotational symmetry, where the order of the CG's sums moves them by 1e-12.
template <bool W64, bool W32, bool Q8>
__global__ void __launch_bounds__(kAsmThreads) k_assemble(DevMesh m, DevCsr csr, MaterialDev M,
                                                          const double* __restrict__ E_c,
                                                          const double* __restrict__ nu_c) {
    extern __shared__ double2 sacc[];
    const int s0 = 4 * blockIdx.x, s1 = min(s0 + 4, csr.n_slices);
    const long long B0 = csr.slice_ptr[s0], B1 = csr.slice_ptr[s1];
    const int len = (int)(2 * (B1 - B0));
    const int n = blockIdx.x * kAsmThreads + threadIdx.x;
    int q = 0, q1 = 0, code = 0;
    double Ec = 1.0, nuc = 0.0;
    if (n < m.n_nodes) {
        q = csr.inc_pos[n];
        q1 = csr.inc_pos[n + 1];
        if (q < q1) {
            code = csr.inc[q];
            Ec = E_c[code >> 3];
            nuc = nu_c[code >> 3];
        }
    }
    for (int t = threadIdx.x; t < len; t += blockDim.x) sacc[t] = make_double2(0.0, 0.0);
    __syncthreads();
    if (n < m.n_nodes) {
        const RowAcc nb = row_acc(sacc + 2 * (csr.slice_ptr[n >> 5] - B0), n & 31);
        while (q < q1) {
            const int e = code >> 3, i = code & 7;
            const Dmat d = form_d(M.plane, Ec, nuc);
            const uint32_t kk = csr.inc_k[q], kk8 = Q8 ? csr.inc_k8[q] : 0u;
            if (++q < q1) {
                code = csr.inc[q];
                Ec = E_c[code >> 3];
                nuc = nu_c[code >> 3];
            }
            element_rows<Q8>(m, e, i, kk, kk8, d, M.h, nb);
        }
    }
    __syncthreads();
    double2* out64 = reinterpret_cast<double2*>(csr.val64 + 4 * B0);
    float2* out32 = W32 ? reinterpret_cast<float2*>(csr.val32 + 4 * B0) : nullptr;
    for (int t = threadIdx.x; t < len; t += blockDim.x) {
        const double2 v = sacc[row_unit(t)];
        if (W64) out64[t] = v;
        if (W32) out32[t] = make_float2((float)v.x, (float)v.y);
    }
}


}  // namespace
constexpr int kElemThreads = 256;

__device__ __forceinline__ bool solve_failed(const CgScalars* solve) {
    return solve && (solve->status == CP_ERR_BREAKDOWN || solve->chip_err);
}

// strain4 + plastStress + exitNorm2 (src/PlasticitySolver.cu:1517-1549,
// 1590-1610, 1664-1691) fused: element-mean strain, stress from the C of the
// last assembly, stress intensity, secant update, and the two exit-norm sums
// (reduced deterministically by the last block). With Aitken on, the raw
// secant target psi is stored as a residual and the relax kernel moves psi.
// 4 blocks per SM (64 registers) for the latency of the gathers, and a grid
// that fits once, so that the block sums and their fence are paid once per
// block: 1,048,576 quads with Hollomon hardening, whole call 125 us at 2
// blocks per SM with Newton's method on pow, 73 now (floor 26: 168 MB). With
// the 8-node element 2 blocks per SM (128 registers): 64 registers spill 656
// bytes a thread; 639,200 8-node quads, whole call with a linear and a
// Hollomon diagram 125 and 137 us at 2, 150 and 174 at 1, 162 and 172 at 3, 174
// and 175 at 4; 576 and 6144 of them 28.7 at each.
// solve: a linear solve whose outcome the host has not seen yet; where it
// failed, the elements keep their state.
template <bool Q8>
__global__ void __launch_bounds__(kElemThreads, Q8 ? 2 : 4) k_update(DevMesh m, MaterialDev M, const double2* __restrict__ u,
                                                         ElemState st, OuterScalars* sc, double* partials, int aitken,
                                                         int first, const CgScalars* solve) {
    __shared__ double sh[2 * kElemThreads / 32];
    __shared__ bool last;
    if (solve_failed(solve)) return;
    const int ne = m.c3 + m.c4 + m.c8;
    double s_num = 0.0, s_den = 0.0, s_an = 0.0, s_ad = 0.0;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += gridDim.x * blockDim.x)
        update_element<Q8>(m, M, u, st, e, aitken, s_num, s_den, s_an, s_ad);
    double2 a = block_sum2(s_num, s_den, sh);
    double2 b = aitken ? block_sum2(s_an, s_ad, sh) : make_double2(0.0, 0.0);
    if (threadIdx.x == 0) {
        partials[4 * blockIdx.x + 0] = a.x;
        partials[4 * blockIdx.x + 1] = a.y;
        partials[4 * blockIdx.x + 2] = b.x;
        partials[4 * blockIdx.x + 3] = b.y;
    }
    if (last_block_arrive(&sc->ticket, &last)) {
        double t0 = 0, t1 = 0, t2 = 0, t3 = 0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
            const volatile double* p = partials + 4 * i;
            t0 += p[0]; t1 += p[1]; t2 += p[2]; t3 += p[3];
        }
        double2 x = block_sum2(t0, t1, sh);
        double2 y = block_sum2(t2, t3, sh);
        if (threadIdx.x == 0) {
            sc->num = x.x;
            sc->den = x.y;
            sc->rel_err = sqrt(x.x / x.y);
            sc->a_num = y.x;
            sc->a_den = y.y;
            if (aitken) {  // the relaxation factor of this step, from the last one's
                double w = 1.0;
                if (!first && y.y > 0.0) w = -sc->aitken_omega * y.x / y.y;
                if (!(w >= 0.1)) w = 0.1;
                if (w > 10.0) w = 10.0;
                sc->aitken_omega = w;
            }
            sc->ticket = 0;
        }
    }
}

namespace {

// Aitken (Irons-Tuck) relaxation of the secant iteration on psi:
// psi_{k+1} = psi_k + w_k r_k, w_k = -w_{k-1} (r_{k-1}, r_k - r_{k-1}) / |r_k - r_{k-1}|^2.
// The fixed point (r = 0) is the reference's. Nothing moves after a failed
// linear solve or an exit norm that is not finite, which the host has yet to see.
__global__ void k_aitken(DevMesh m, MaterialDev M, ElemState st, const OuterScalars* sc, const CgScalars* solve) {
    if (solve_failed(solve) || !(sc->rel_err - sc->rel_err == 0.0)) return;
    const int ne = m.c3 + m.c4 + m.c8;
    const double w = sc->aitken_omega;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += gridDim.x * blockDim.x)
        relax_element(M, st, e, w);
}

// plastDeform (src/PlasticitySolver.cu:1641-1653); the reference's guard is
// e > count (one past the end), here e < count.
__global__ void k_plastic(int ne, MaterialDev M, ElemState st) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += gridDim.x * blockDim.x)
        plastic_element(M, st, e);
}

}  // namespace

template <bool Q8>
void assemble_as(const DevMesh& m, const DevCsr& csr, const MaterialDev& mat, const double* E_c, const double* nu_c,
                 bool want64, bool want32, int grid, size_t smem, cudaStream_t s) {
    if (want64 && want32) {
        CP_CUDA(cudaFuncSetAttribute(k_assemble<true, true, Q8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_assemble<true, true, Q8><<<grid, kAsmThreads, smem, s>>>(m, csr, mat, E_c, nu_c);
    } else if (want64) {
        CP_CUDA(cudaFuncSetAttribute(k_assemble<true, false, Q8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_assemble<true, false, Q8><<<grid, kAsmThreads, smem, s>>>(m, csr, mat, E_c, nu_c);
    } else {
        CP_CUDA(cudaFuncSetAttribute(k_assemble<false, true, Q8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_assemble<false, true, Q8><<<grid, kAsmThreads, smem, s>>>(m, csr, mat, E_c, nu_c);
    }
}

void launch_assemble(const DevMesh& m, const DevCsr& csr, const MaterialDev& mat, const double* E_c,
                     const double* nu_c, bool want64, bool want32, cudaStream_t s, int sm_count) {
    const int ntiles = (m.n_nodes + kAsmThreads - 1) / kAsmThreads;
    const size_t smem = (size_t)kAsmThreads * 4 * csr.max_width * sizeof(double);
    CP_CHECK(smem <= 200 * 1024, CP_ERR_UNSUPPORTED, "node degree too large for the assembly tile");
    const int grid = std::max(ntiles, 1);
    if (m.c8)
        assemble_as<true>(m, csr, mat, E_c, nu_c, want64, want32, grid, smem, s);
    else
        assemble_as<false>(m, csr, mat, E_c, nu_c, want64, want32, grid, smem, s);
    CP_CUDA(cudaGetLastError());
}

// Threads per block of the element kernels: small meshes in small blocks, so
// that they spread over the SMs (4096 quads: 64 blocks of 64).
int elem_threads(int ne, int sm_count) { return ne <= 2 * 64 * sm_count ? 64 : kElemThreads; }

int update_grid(int ne, int sm_count) {
    const int t = elem_threads(ne, sm_count);
    int g = (ne + t - 1) / t;
    int cap = sm_count * 4;
    return g < 1 ? 1 : (g < cap ? g : cap);
}

void launch_update(const DevMesh& m, const MaterialDev& mat, const double2* u, ElemState& st, OuterScalars* sc,
                   double* partials, int aitken, int first, const CgScalars* solve, cudaStream_t s, int sm_count) {
    const int ne = m.c3 + m.c4 + m.c8;
    const auto k = m.c8 ? k_update<true> : k_update<false>;
    k<<<update_grid(ne, sm_count), elem_threads(ne, sm_count), 0, s>>>(m, mat, u, st, sc, partials, aitken, first, solve);
    CP_CUDA(cudaGetLastError());
}

void launch_aitken_relax(const DevMesh& m, const MaterialDev& mat, ElemState& st, const OuterScalars* sc,
                         const CgScalars* solve, cudaStream_t s, int sm_count) {
    const int ne = m.c3 + m.c4 + m.c8;
    k_aitken<<<update_grid(ne, sm_count), elem_threads(ne, sm_count), 0, s>>>(m, mat, st, sc, solve);
    CP_CUDA(cudaGetLastError());
}

void launch_plastic(const DevMesh& m, const MaterialDev& mat, ElemState& st, cudaStream_t s, int sm_count) {
    const int ne = m.c3 + m.c4 + m.c8;
    k_plastic<<<update_grid(ne, sm_count), elem_threads(ne, sm_count), 0, s>>>(ne, mat, st);
    CP_CUDA(cudaGetLastError());
}

}  // namespace cp

// ------------------------------------------------ allocation-free update --
//
// Some callers cannot allocate device memory: code inside a framework that
// owns the whole device memory pool through its own caching allocator (a
// cudaMalloc beside it fails or fragments that pool), and embedded or
// real-time loops whose memory budget is fixed up front. For
// them cp_secant_update_noalloc runs the fused strain / stress / secant-update
// kernel (k_update above) on buffers the caller already owns. Its only scratch
// -- the block partial sums of the exit norm and the reduction's scalars --
// lives in the file-scope array below, which every GPU that loads this library
// keeps until the process exits.
namespace {

// Partial-sum slots. The call's limit, 1,048,576 elements, is one block of 256
// per slot; the grid takes at most 4 blocks per SM of them.
constexpr int kNoAllocMaxBlocks = 4096;
constexpr int kNoAllocScalarBytes = 256;  // cp::OuterScalars, padded
static_assert(sizeof(cp::OuterScalars) <= kNoAllocScalarBytes, "scalars do not fit the scratch header");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScalarBytes + 4 * 8 * kNoAllocMaxBlocks];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of the scratch array on the current device. In host code the
// array's name is only a host-side stand-in, so the address is looked up once
// per device (with that device current) and cached.
int noalloc_scratch(int device, unsigned char** out) {
    if (device < 0 || device >= kNoAllocMaxDevices) return CP_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[device]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return CP_ERR_CUDA;
        g_noalloc_ptr[device] = p;
    }
    *out = static_cast<unsigned char*>(g_noalloc_ptr[device]);
    return CP_OK;
}

}  // namespace

extern "C" CP_API int cp_secant_update_noalloc(void* stream, const cp_material* mat, int node_count,
                                               const double* d_node_xy, int count4, const int* d_elem4,
                                               const double* d_uv, double* d_E_c, double* d_nu_c, double* d_psi,
                                               double* d_fields, double* rel_err) {
    if (!mat || !d_node_xy || !d_elem4 || !d_uv || !d_E_c || !d_nu_c || !d_psi || !d_fields || !rel_err)
        return CP_ERR_INVALID;
    if (node_count <= 0 || count4 <= 0) return CP_ERR_INVALID;
    if ((long long)count4 > (long long)kNoAllocMaxBlocks * cp::kElemThreads) return CP_ERR_INVALID;  // > 1,048,576
    if (((uintptr_t)d_node_xy | (uintptr_t)d_elem4 | (uintptr_t)d_uv) & 15u) return CP_ERR_INVALID;
    if (!(mat->E > 0) || !(mat->nu > -1.0 && mat->nu < 0.5) || mat->diagram < CP_DIAGRAM_ELASTIC ||
        mat->diagram > CP_DIAGRAM_PIECEWISE || (mat->diagram == CP_DIAGRAM_PIECEWISE &&
                                                 (mat->n_points < 2 || mat->n_points > CP_MAX_PW)))
        return CP_ERR_INVALID;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return CP_ERR_NO_DEVICE;
    unsigned char* scratch = nullptr;
    int st = noalloc_scratch(device, &scratch);
    if (st != CP_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cp::OuterScalars* sc = reinterpret_cast<cp::OuterScalars*>(scratch);
    double* partials = reinterpret_cast<double*>(scratch + kNoAllocScalarBytes);
    // the array keeps the previous call's contents: the reduction ticket must start at zero
    if (cudaMemsetAsync(sc, 0, sizeof(cp::OuterScalars), s) != cudaSuccess) return CP_ERR_CUDA;
    cp::MaterialDev M{};
    M.E = mat->E; M.nu = mat->nu; M.h = mat->h; M.plane = mat->plane; M.diagram = mat->diagram;
    M.sigma_t = mat->sigma_t; M.k_t = mat->k_t; M.a = mat->a; M.m = mat->m; M.eps0 = mat->eps0; M.n = mat->n;
    M.n_points = mat->n_points;
    for (int i = 0; i < CP_MAX_PW; ++i) { M.pw_eps[i] = mat->pw_eps[i]; M.pw_sig[i] = mat->pw_sig[i]; }
    cp::DevMesh m;
    m.n_nodes = node_count;
    m.c3 = 0;
    m.c4 = count4;
    m.xy = reinterpret_cast<double2*>(const_cast<double*>(d_node_xy));
    m.e4 = reinterpret_cast<int4*>(const_cast<int*>(d_elem4));
    cp::ElemState es{};
    const size_t ne = (size_t)count4;
    es.exx = d_fields; es.eyy = d_fields + ne; es.gam = d_fields + 2 * ne; es.eps_i = d_fields + 3 * ne;
    es.sxx = d_fields + 4 * ne; es.syy = d_fields + 5 * ne; es.tau = d_fields + 6 * ne; es.sig_i = d_fields + 7 * ne;
    es.table_s = d_fields + 8 * ne;
    es.psi = d_psi; es.E_c = d_E_c; es.nu_c = d_nu_c;
    const int threads = cp::elem_threads(count4, cp::kB200Sms);
    const int grid = cp::update_grid(count4, cp::kB200Sms);  // <= kNoAllocMaxBlocks
    cp::k_update<false><<<grid, threads, 0, s>>>(m, M, reinterpret_cast<const double2*>(d_uv), es, sc, partials, 0, 0, nullptr);
    if (cudaGetLastError() != cudaSuccess) return CP_ERR_CUDA;
    double host_err = 0.0;
    if (cudaMemcpyAsync(&host_err, &sc->rel_err, sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return CP_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return CP_ERR_CUDA;
    *rel_err = host_err;
    return CP_OK;
}
