// Projection hash of float32 rows that the tensor-core kernels cannot take (rows that do not start on
// 16-byte boundaries, keys of more than 32 bytes): fp32 multiply-adds in the order of the features, as
// the kernel of project_simt.cuh does them, so that the sums are the same to the last bit.
//
// The fp32 pipe bounds it (128 multiply-adds a cycle and SM).  A CTA takes 128 rows and the hash columns
// of whole tables, at most 128, evenly over the groups; a thread 8 x 8 of them (8 x 4 when a group
// has at most 64 columns), in two halves 64 apart, so that four 16-byte shared-memory reads serve
// 64 multiply-adds.  The tiles arrive feature-major through a ring of three stages: 4-byte cp.async,
// the only size that rows of any length allow, turns them on the way.  Features past d are not multiplied; the zero that
// they add (project_simt_kernel pads to sixteen) is added once.
//
// Rows of few features are over in a few steps, and what surrounds them weighs more: a CTA stays for many row blocks of
// its group of columns and fetches the first stages of the next block before it packs the keys of this one.  The hash
// values lie column by column, a thread's four rows together and their place turned by the column, so that 16-byte
// stores and the packing's reads meet all banks.  (128 columns a thread group: stages and hash values do not fit twice an
// SM, and the values take the stages' place as the last step is done.)
// 333,337 x 50 rows, 60 columns: 155 us with project_simt_kernel, with one block of rows a CTA 112.7, now 108.9.
#pragma once

#include "common.cuh"
#include "index_math.h"
#include "project_simt.cuh"

namespace culsh_b200 {

constexpr int PG_BM = 128;
constexpr int PG_BK = 16;      // the steps of project_simt_kernel: features past d enter as zeros there, too
constexpr int PG_PITCH = 132;
constexpr int PG_STAGES = 3;
constexpr int PG_THREADS = 256;
template <int BN>
struct ProjectF32Cfg {
    static constexpr int P_PITCH = BN + 4;
    static constexpr int STAGE = PG_BK * (PG_PITCH + P_PITCH);  // floats
    static constexpr size_t STAGES_BYTES = sizeof(float) * PG_STAGES * (size_t)STAGE;
    static constexpr size_t HASH_BYTES = sizeof(int32_t) * PG_BM * (size_t)BN;
    static constexpr bool APART = BN == 64;  // hash values and stages
    static constexpr size_t SMEM = APART ? STAGES_BYTES + HASH_BYTES : STAGES_BYTES > HASH_BYTES ? STAGES_BYTES : HASH_BYTES;
};
static_assert(2 * (ProjectF32Cfg<64>::SMEM + 1024) <= 227 * 1024 && 2 * (ProjectF32Cfg<128>::SMEM + 1024) <= 227 * 1024, "two CTAs an SM");

// [column][row], the rows in groups of four whose number is turned by the column's
struct TurnedHashes {
    int32_t* v;
    __device__ __forceinline__ int at(int row4, int col) const { return col * PG_BM + ((row4 ^ ((col >> 2) & 7)) << 2); }
    __device__ __forceinline__ int32_t operator()(int row, int col) const { return v[at(row >> 2, col) + (row & 3)]; }
};

__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 4 : 0)
                 : "memory");
}

template <int FAMILY, int BN>
__global__ void __launch_bounds__(PG_THREADS, 2)
project_f32_kernel(ProjectArgs a) {
    using Cfg = ProjectF32Cfg<BN>;
    constexpr int HALVES = BN / 64;  // of a thread's columns
    extern __shared__ __align__(16) unsigned char pg_smem[];
    float* stages = reinterpret_cast<float*>(pg_smem);
    const TurnedHashes hashes{reinterpret_cast<int32_t*>(pg_smem + (Cfg::APART ? Cfg::STAGES_BYTES : 0))};

    const float* __restrict__ X = static_cast<const float*>(a.X);
    const float* __restrict__ P = static_cast<const float*>(a.P);
    const float* __restrict__ bias = static_cast<const float*>(a.bias);

    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int G = a.tables_per_group;
    const int n_groups = (a.L + G - 1) / G;
    const int group = blockIdx.x % n_groups;  // fastest: the groups of one row block share X in L2
    const int n_blocks = row_blocks(a.n, PG_BM), block_step = gridDim.x / n_groups;  // the grid is a multiple of the groups
    const int GC = G * a.k;
    const int col_base = group * GC;
    const int gc_valid = min(GC, a.L * a.k - col_base);
    const int n_steps = (a.d + PG_BK - 1) / PG_BK;

    // a thread copies feature tid % 16 of rows (columns) tid / 16, + 16, ...; rows and columns past the
    // end and features past d are zero
    auto load = [&](int block, int step, int slot) {
        float* xs = stages + (size_t)slot * Cfg::STAGE + tx * PG_PITCH;
        float* ps = stages + (size_t)slot * Cfg::STAGE + PG_BK * PG_PITCH + tx * Cfg::P_PITCH;
        const int f = step * PG_BK + tx, row0 = block * PG_BM;
        const bool f_ok = f < a.d;
#pragma unroll
        for (int i = 0; i < PG_BM / 16; ++i) {
            const int r = ty + 16 * i;
            const bool ok = f_ok && r < a.n - row0;
            cp_async4(xs + r, ok ? X + (size_t)(row0 + r) * a.d + f : X, ok);
        }
#pragma unroll
        for (int i = 0; i < BN / 16; ++i) {
            const int c = ty + 16 * i;
            const bool ok = f_ok && c < gc_valid;
            cp_async4(ps + c, ok ? P + (size_t)(col_base + c) * a.d + f : P, ok);
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    auto next_slot = [](int slot) { return slot + 1 == PG_STAGES ? 0 : slot + 1; };

    int slot = 0;  // of the step that is multiplied; the two after it are in flight
    auto begin = [&](int block) {
        load(block, 0, slot);
        commit();
        if (n_steps > 1) load(block, 1, next_slot(slot));
        commit();
    };
    int block = blockIdx.x / n_groups;
    if (block < n_blocks) begin(block);
    for (; block < n_blocks; block += block_step) {
        float acc[8][4 * HALVES];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4 * HALVES; ++j) acc[i][j] = 0.f;
        for (int step = 0; step < n_steps; ++step) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();  // the stage has landed for every thread, and the one that is refilled now has been read
            if (step + 2 < n_steps) load(block, step + 2, next_slot(next_slot(slot)));
            commit();
            const float* xs = stages + (size_t)slot * Cfg::STAGE + ty * 4;
            const float* ps = stages + (size_t)slot * Cfg::STAGE + PG_BK * PG_PITCH + tx * 4;
            auto feature = [&](int kk) {
                float4 xv4[2], pv4[HALVES];
#pragma unroll
                for (int h = 0; h < 2; ++h) xv4[h] = *reinterpret_cast<const float4*>(xs + kk * PG_PITCH + 64 * h);
#pragma unroll
                for (int h = 0; h < HALVES; ++h) pv4[h] = *reinterpret_cast<const float4*>(ps + kk * Cfg::P_PITCH + 64 * h);
                const float* xv = reinterpret_cast<const float*>(xv4);
                const float* pv = reinterpret_cast<const float*>(pv4);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4 * HALVES; ++j) acc[i][j] = fmaf(xv[i], pv[j], acc[i][j]);
            };
            const int here = a.d - step * PG_BK;
            if (here >= PG_BK) {
#pragma unroll
                for (int kk = 0; kk < PG_BK; ++kk) feature(kk);
            } else {
#pragma unroll 1
                for (int kk = 0; kk < here; ++kk) feature(kk);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4 * HALVES; ++j) acc[i][j] += 0.f;  // a sum of -0 becomes +0
            }
            slot = next_slot(slot);
        }
        // The two stages after the last one read are free: nothing was loaded into them, and every thread is past
        // the step before the last.  So is the last one behind the barrier below.
        if (Cfg::APART) {
            if (block + block_step < n_blocks) begin(block + block_step);
        } else {
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < 4 * HALVES; ++j) {
            const int c = 64 * (j >> 2) + tx * 4 + (j & 3);
            if (c < gc_valid) {
                const float bv = FAMILY == CULSH_PSLSH ? bias[col_base + c] : 0.f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    int32_t q[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        q[i] = FAMILY == CULSH_RPLSH
                                   ? (int32_t)((__float_as_uint(acc[4 * h + i][j]) >> 31) ^ 1u)  // rplsh/hash.cuh:47
                                   : static_cast<int32_t>(floor(acc[4 * h + i][j] + bv));        // pslsh/hash.cuh:46
                    *reinterpret_cast<int4*>(hashes.v + hashes.at(16 * h + ty, c)) = make_int4(q[0], q[1], q[2], q[3]);
                }
            }
        }
        __syncthreads();
        pack_hash_values<FAMILY>(a, hashes, block * PG_BM, PG_BM, group * G, gc_valid / a.k, PG_THREADS);
        if (!Cfg::APART) {
            __syncthreads();
            if (block + block_step < n_blocks) begin(block + block_step);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Tables of at most 128 hashes (a group holds whole tables); the caller takes project_simt_kernel else.
inline bool launch_project_f32(const CtxPtr& c, cudaStream_t stream, int family, const float* X, const float* P,
                               const float* bias, int n, int d, int L, int k, const KeySpec& ks, uint32_t* keys,
                               uint8_t* ovf_rows, int row_offset, int n_total) {
    if (k > 128 || ProjectF32Cfg<128>::SMEM > c->smem_optin) return false;
    if (n == 0) return true;
    const int groups = (int)ceil_div(L, std::min(L, 128 / k));
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
    // A whole number of CTAs for each group that stay for all of its blocks, two an SM, where that many groups leave no more than a
    // tenth of the places empty, else a CTA for each block and group.  200,003 x 50 rows, staying and not: 64 columns 58 and 58 us (p-stable
    // 62 and 68), 128 columns 99 and 99; 20,000 x 33 rows, 6,400 columns in 50 groups 419 and 356.
    const size_t n_groups = ceil_div(L, a.tables_per_group), n_blocks = row_blocks(n, PG_BM), places = 2 * (size_t)c->sm_count;
    const bool stay = places / n_groups * n_groups * 10 >= places * 9;
    const dim3 grid((unsigned)(n_groups * (stay ? std::min<size_t>(n_blocks, places / n_groups) : n_blocks)));
    auto go = [&](auto kern, size_t smem) {
        CU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, PG_THREADS, smem, stream>>>(a);
        KERNEL_CHECK();
    };
    const bool rp = family == CULSH_RPLSH;
    if (a.tables_per_group * k <= 64) {
        if (rp) go(project_f32_kernel<CULSH_RPLSH, 64>, ProjectF32Cfg<64>::SMEM);
        else go(project_f32_kernel<CULSH_PSLSH, 64>, ProjectF32Cfg<64>::SMEM);
    } else {
        if (rp) go(project_f32_kernel<CULSH_RPLSH, 128>, ProjectF32Cfg<128>::SMEM);
        else go(project_f32_kernel<CULSH_PSLSH, 128>, ProjectF32Cfg<128>::SMEM);
    }
    return true;
}

}  // namespace culsh_b200
