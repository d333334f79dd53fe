// Projection hash of float64 rows: X . P^T on the double-precision matrix instructions (mma.sync
// m16n8k8 f64; tcgen05 has no f64 kind) with the quantise-and-pack epilogue of the CUDA-core kernel
// (rplsh/hash.cuh:24-48, pslsh/hash.cuh:26-47).
//
// The f64 pipe bounds it (64 FMA a cycle and SM).  The CUDA-core kernel reads twelve 8-byte words of
// shared memory for every 32 FMA of a thread and waits for its loads once per 16 features; a matrix
// instruction takes 32 FMA a lane from six words, and the tiles come through a ring of three
// stages with cp.async (8 bytes each: rows of an odd number of features start on 8-byte
// boundaries only).  A CTA takes 64 rows and up to 128 hash columns of whole tables; two of them share an
// SM, so that one packs its keys while the other multiplies (one CTA of 128 rows: 0.49 ms instead of
// 0.46 below).  The columns are spread evenly over the groups and, in steps of eight, over
// the two halves of the warps, so that 224 columns are 2 x 112 and no column past the last step of
// eight is computed.
// 200,003 x 100 rows, 224 columns: 0.97 ms on the CUDA cores, 0.46 here (20 TFLOP/s).
#pragma once

#include "common.cuh"
#include "project_simt.cuh"

namespace culsh_b200 {

constexpr int PF_BM = 64;
constexpr int PF_BN = 128;   // columns of a group at most
constexpr int PF_BK = 16;    // features per stage
constexpr int PF_PITCH = PF_BK + 4;  // 160-byte rows: the eight rows of a fragment fall on all banks
constexpr int PF_STAGES = 3;
constexpr int PF_THREADS = 256;
constexpr size_t PF_STAGE = (size_t)(PF_BM + PF_BN) * PF_PITCH;  // doubles
constexpr size_t PF_SMEM = PF_STAGES * PF_STAGE * sizeof(double);
static_assert(PF_SMEM >= sizeof(int32_t) * PF_BM * (PF_BN + 1), "the hash values take the place of the stages");

__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

template <int FAMILY>
__global__ void __launch_bounds__(PF_THREADS, 2)
project_f64_kernel(ProjectArgs a) {
    extern __shared__ __align__(16) unsigned char pf_smem[];
    double* stages = reinterpret_cast<double*>(pf_smem);
    int32_t* hbuf = reinterpret_cast<int32_t*>(pf_smem);  // after the last stage: [PF_BM][GC | 1]

    const double* __restrict__ X = static_cast<const double*>(a.X);
    const double* __restrict__ P = static_cast<const double*>(a.P);
    const double* __restrict__ bias = static_cast<const double*>(a.bias);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = a.tables_per_group;
    const int n_groups = (a.L + G - 1) / G;
    const int group = blockIdx.x % n_groups;  // fastest: the groups of one row block share X in L2
    const int row0 = (blockIdx.x / n_groups) * PF_BM;
    const int GC = G * a.k;
    const int col_base = group * GC;
    const int gc_valid = min(GC, a.L * a.k - col_base);
    const int n_steps = (a.d + PF_BK - 1) / PF_BK;

    // a thread copies feature tid % 16 of rows (columns) tid / 16, + 16, ...; rows and columns past the
    // end and features past d are zero
    const int lf = tid & 15, lr = tid >> 4;
    auto load = [&](int step) {
        double* xs = stages + (size_t)(step % PF_STAGES) * PF_STAGE;
        double* ps = xs + (size_t)PF_BM * PF_PITCH;
        const int f = step * PF_BK + lf;
        const bool f_ok = f < a.d;
#pragma unroll
        for (int i = 0; i < PF_BM / 16; ++i) {
            const int r = lr + 16 * i;
            const bool ok = f_ok && row0 + r < a.n;
            cp_async8(xs + r * PF_PITCH + lf, ok ? X + (size_t)(row0 + r) * a.d + f : X, ok);
        }
#pragma unroll
        for (int i = 0; i < PF_BN / 16; ++i) {
            const int c = lr + 16 * i;
            const bool ok = f_ok && c < gc_valid;
            cp_async8(ps + c * PF_PITCH + lf, ok ? P + (size_t)(col_base + c) * a.d + f : P, ok);
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

    // warp tile: 16 rows and every second step of eight columns
    const int wm = (warp >> 1) * 16, wn = warp & 1;
    const int g = lane >> 2, t = lane & 3;
    const int n_frag = (gc_valid + 7) / 8;
    double acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.0;

    load(0);
    commit();
    if (n_steps > 1) load(1);
    commit();
    for (int step = 0; step < n_steps; ++step) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // the stage has landed for every thread, and the one that is refilled now has been read
        if (step + 2 < n_steps) load(step + 2);
        commit();
        const double* xs = stages + (size_t)(step % PF_STAGES) * PF_STAGE;
        const double* ps = xs + (size_t)PF_BM * PF_PITCH;
#pragma unroll
        for (int kk = 0; kk < PF_BK; kk += 8) {
            const double* x = xs + (wm + g) * PF_PITCH + kk + t;
            const double af[4] = {x[0], x[8 * PF_PITCH], x[4], x[8 * PF_PITCH + 4]};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int frag = 2 * j + wn;
                if (frag < n_frag) {  // uniform
                    const double* p = ps + (frag * 8 + g) * PF_PITCH + kk + t;
                    const double bf[2] = {p[0], p[4]};
                    mma_f64(acc[j], af, bf);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    const int pitch = GC | 1;  // odd: the packing threads read one column of many rows
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c0 = (2 * j + wn) * 8 + 2 * t;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = c0 + e;
            if (c < gc_valid) {
                const double bv = FAMILY == CULSH_PSLSH ? bias[col_base + c] : 0.0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double v = acc[j][2 * h + e];
                    const int32_t q = FAMILY == CULSH_RPLSH
                                          ? (int32_t)((__float_as_uint((float)v) >> 31) ^ 1u)  // rplsh/hash.cuh:47
                                          : static_cast<int32_t>(floor(v + bv));               // pslsh/hash.cuh:46
                    hbuf[(wm + 8 * h + g) * pitch + c] = q;
                }
            }
        }
    }
    __syncthreads();
    pack_hash_values<FAMILY>(a, RowMajorHashes{hbuf, pitch}, row0, PF_BM, group * G, gc_valid / a.k, PF_THREADS);
}

// Tables of at most 128 hashes (a group holds whole tables); the caller takes the CUDA-core kernel else.
inline bool launch_project_f64(const CtxPtr& c, cudaStream_t stream, int family, const double* X, const double* P,
                               const double* bias, int n, int d, int L, int k, const KeySpec& ks, uint32_t* keys,
                               uint8_t* ovf_rows, int row_offset, int n_total) {
    if (k > PF_BN || PF_SMEM > c->smem_optin) return false;
    if (n == 0) return true;
    const int most = std::min(L, PF_BN / k);
    const int groups = (int)ceil_div(L, most);
    ProjectArgs a{};
    a.X = X; a.P = P; a.bias = bias; a.keys = keys; a.ovf_rows = ovf_rows;
    a.d_error = c->d_error;
    a.range = family == CULSH_PSLSH && ks.elem_bytes == 1 && !ovf_rows ? c->d_error + 2 : nullptr;
    a.n = n; a.d = d; a.L = L; a.k = k;
    a.tables_per_group = (int)ceil_div(L, groups);
    a.key_words = ks.key_words;
    a.elem_bytes = ks.elem_bytes;
    a.row_offset = row_offset;
    a.n_total = n_total;
    const dim3 grid((unsigned)(ceil_div(L, a.tables_per_group) * ceil_div(n, PF_BM)));
    auto kern = family == CULSH_RPLSH ? project_f64_kernel<CULSH_RPLSH> : project_f64_kernel<CULSH_PSLSH>;
    CU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PF_SMEM));
    kern<<<grid, PF_THREADS, PF_SMEM, stream>>>(a);
    KERNEL_CHECK();
    return true;
}

}  // namespace culsh_b200
