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
// the two halves of the warps, so that 224 columns are 2 x 112; the number of steps is a template argument, without
// which every instruction stood behind a branch of its own.  Steps of eight features past d are left out.
//
// A row of a few dozen features is over in two or three stages of a microsecond, and what surrounds them weighs as much: a CTA
// then stays for many row blocks of its group of columns (see launch_project_f64) and, for sign bits, fetches the first stages of
// the next block before it packs the keys of this one.  The bits of a step of eight columns are one byte a row, made from ballots.
// 200,003 x 100 rows, 224 columns: 0.97 ms on the CUDA cores, with one block of rows a CTA and a branch before every instruction 0.46 (with 2,001 queries), with CTAs that stay 0.367, now 0.353.
#pragma once

#include "common.cuh"
#include "index_math.h"
#include "project_simt.cuh"

namespace culsh_b200 {

constexpr int PF_BM = 64;
constexpr int PF_BN = 128;   // columns of a group at most
constexpr int PF_BK = 16;    // features per stage
constexpr int PF_PITCH = PF_BK + 4;  // 160-byte rows: the eight rows of a fragment fall on all banks
constexpr int PF_STAGES = 3;
constexpr int PF_THREADS = 256;
constexpr size_t PF_STAGE = (size_t)(PF_BM + PF_BN) * PF_PITCH;  // doubles
constexpr int PF_BITS = PF_BN / 8 + 4;  // bytes of a row's sign bits, and a word that the last one's neighbour is read from
constexpr size_t PF_STAGES_BYTES = PF_STAGES * PF_STAGE * sizeof(double);
constexpr size_t PF_SMEM = PF_STAGES_BYTES + PF_BM * PF_BITS;
static_assert(PF_STAGES_BYTES >= sizeof(int32_t) * PF_BM * (PF_BN + 1), "p-stable hash values take the place of the stages");
static_assert(2 * (PF_SMEM + 1024) <= 227 * 1024, "two CTAs an SM");

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

// bit t of n to bit 6 - 2 t
__device__ __forceinline__ uint32_t spread_nibble(uint32_t n) {
    return ((n & 1u) << 6) | ((n & 2u) << 3) | (n & 4u) | ((n & 8u) >> 3);
}

// Keys of the tables of a block of rows from their bits in shared memory, hash 0 in the top bit of byte 0 of its row.
__device__ __forceinline__ void pack_sign_bits(const ProjectArgs& a, const uint32_t* __restrict__ bits, int row0, int first_table, int tables_here) {
    const int NW = a.key_words;
    for (int idx = threadIdx.x; idx < PF_BM * tables_here; idx += PF_THREADS) {
        const int r = idx % PF_BM, g = idx / PF_BM, row = row0 + r;
        if (row >= a.n) continue;
        const uint32_t* line = bits + r * (PF_BITS / 4);
        uint32_t* dst = a.keys + ((size_t)(first_table + g) * a.n_total + a.row_offset + row) * NW;
        for (int w = 0; w < NW; ++w) {
            const int end = a.k - 32 * (NW - 1 - w), len = min(32, end);  // the word's bits of the table: [end - len, end)
            uint32_t v = 0;
            if (end > 0) {
                const int at = g * a.k + end - len;
                const uint32_t hi = __byte_perm(line[at >> 5], 0, 0x0123), lo = __byte_perm(line[(at >> 5) + 1], 0, 0x0123);
                v = __funnelshift_l(lo, hi, at & 31) >> (32 - len);
            }
            dst[w] = v;
        }
    }
}

template <int FAMILY, int NF>  // NF: steps of eight columns of a warp
__global__ void __launch_bounds__(PF_THREADS, 2)
project_f64_kernel(ProjectArgs a) {
    constexpr bool BITS = FAMILY == CULSH_RPLSH;
    extern __shared__ __align__(16) unsigned char pf_smem[];
    double* stages = reinterpret_cast<double*>(pf_smem);
    int32_t* hbuf = reinterpret_cast<int32_t*>(pf_smem);  // p-stable, after the last stage: [PF_BM][GC | 1]
    unsigned char* bits = pf_smem + PF_STAGES_BYTES;      // sign bits: [PF_BM][PF_BITS]

    const double* __restrict__ X = static_cast<const double*>(a.X);
    const double* __restrict__ P = static_cast<const double*>(a.P);
    const double* __restrict__ bias = static_cast<const double*>(a.bias);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = a.tables_per_group;
    const int n_groups = (a.L + G - 1) / G;
    const int group = blockIdx.x % n_groups;  // fastest: the groups of one row block share X in L2
    const int n_blocks = row_blocks(a.n, PF_BM), block_step = gridDim.x / n_groups;  // the grid is a multiple of the groups
    const int GC = G * a.k;
    const int col_base = group * GC;
    const int gc_valid = min(GC, a.L * a.k - col_base);
    const int n_steps = (a.d + PF_BK - 1) / PF_BK;

    // a thread copies feature tid % 16 of rows (columns) tid / 16, + 16, ...; rows and columns past the
    // end and features past d are zero
    const int lf = tid & 15, lr = tid >> 4;
    auto load = [&](int block, int step, int slot) {
        double* xs = stages + (size_t)slot * PF_STAGE;
        double* ps = xs + (size_t)PF_BM * PF_PITCH;
        const int f = step * PF_BK + lf, row0 = block * PF_BM;
        const bool f_ok = f < a.d;
#pragma unroll
        for (int i = 0; i < PF_BM / 16; ++i) {
            const int r = lr + 16 * i;
            const bool ok = f_ok && r < a.n - row0;
            cp_async8(xs + r * PF_PITCH + lf, ok ? X + (size_t)(row0 + r) * a.d + f : X, ok);
        }
#pragma unroll
        for (int i = 0; i < NF; ++i) {  // 16 * NF columns are multiplied
            const int c = lr + 16 * i;
            const bool ok = f_ok && c < gc_valid;
            cp_async8(ps + c * PF_PITCH + lf, ok ? P + (size_t)(col_base + c) * a.d + f : P, ok);
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    auto next_slot = [](int slot) { return slot + 1 == PF_STAGES ? 0 : slot + 1; };
    int slot = 0;  // of the step that is multiplied; the two after it are in flight
    auto begin = [&](int block) {
        load(block, 0, slot);
        commit();
        if (n_steps > 1) load(block, 1, next_slot(slot));
        commit();
    };

    // warp tile: 16 rows and every second step of eight columns
    const int wm = (warp >> 1) * 16, wn = warp & 1;
    const int g = lane >> 2, t = lane & 3;
    int block = blockIdx.x / n_groups;
    if (block < n_blocks) begin(block);
    for (; block < n_blocks; block += block_step) {
        double acc[NF][4];
#pragma unroll
        for (int j = 0; j < NF; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[j][e] = 0.0;
        for (int step = 0; step < n_steps; ++step) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();  // the stage has landed for every thread, and the one that is refilled now has been read
            if (step + 2 < n_steps) load(block, step + 2, next_slot(next_slot(slot)));
            commit();
            const double* xs = stages + (size_t)slot * PF_STAGE + (wm + g) * PF_PITCH + t;
            const double* ps = stages + (size_t)slot * PF_STAGE + (size_t)(PF_BM + wn * 8 + g) * PF_PITCH + t;
#pragma unroll
            for (int kk = 0; kk < PF_BK; kk += 8) {
                if (kk == 0 || a.d - step * PF_BK > kk) {  // uniform
                    const double af[4] = {xs[kk], xs[8 * PF_PITCH + kk], xs[kk + 4], xs[8 * PF_PITCH + kk + 4]};
#pragma unroll
                    for (int j = 0; j < NF; ++j) {
                        const double bf[2] = {ps[16 * j * PF_PITCH + kk], ps[16 * j * PF_PITCH + kk + 4]};
                        mma_f64(acc[j], af, bf);
                    }
                }
            }
            slot = next_slot(slot);
        }
        const int left = a.d % PF_BK;
        if (left > 0 && left <= 8) {  // what the step left out would have added: a sum of -0 becomes +0
#pragma unroll
            for (int j = 0; j < NF; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[j][e] += 0.0;
        }
        // The two stages after the last one read are free: nothing was loaded into them, and every thread is past
        // the step before the last.  So is the last one behind the barrier below.
        if constexpr (BITS) {
            if (block + block_step < n_blocks) begin(block + block_step);
#pragma unroll
            for (int j = 0; j < NF; ++j) {
                uint32_t b[4];  // rows g, columns 2 t and 2 t + 1; the same of rows g + 8
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    b[e] = __ballot_sync(0xFFFFFFFFu, (__float_as_uint((float)acc[j][e]) >> 31) == 0);  // rplsh/hash.cuh:47
                const int sh = 4 * (lane & 7);
                const uint32_t even = ((lane & 8 ? b[2] : b[0]) >> sh) & 15u, odd = ((lane & 8 ? b[3] : b[1]) >> sh) & 15u;
                if (lane < 16) bits[(wm + lane) * PF_BITS + 2 * j + wn] = (unsigned char)((spread_nibble(even) << 1) | spread_nibble(odd));
            }
            __syncthreads();
            pack_sign_bits(a, reinterpret_cast<const uint32_t*>(bits), block * PF_BM, group * G, gc_valid / a.k);
        } else {
            __syncthreads();
            const int pitch = GC | 1;  // odd: the packing threads read one column of many rows
#pragma unroll
            for (int j = 0; j < NF; ++j) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = (2 * j + wn) * 8 + 2 * t + e;
                    if (c < gc_valid) {
                        const double bv = bias[col_base + c];
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            hbuf[(wm + 8 * h + g) * pitch + c] = static_cast<int32_t>(floor(acc[j][2 * h + e] + bv));  // pslsh/hash.cuh:46
                    }
                }
            }
            __syncthreads();
            pack_hash_values<FAMILY>(a, RowMajorHashes{hbuf, pitch}, block * PF_BM, PF_BM, group * G, gc_valid / a.k, PF_THREADS);
            __syncthreads();
            if (block + block_step < n_blocks) begin(block + block_step);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
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
    // Rows of few features, and few rows: a whole number of CTAs for each group that stay for all of its blocks, two an SM, where that
    // many groups leave no more than a tenth of the places empty.  Else a CTA for each block and group: from four stages on
    // (from five on with up to 32 columns, p-stable 64) it is the faster one, as packing and multiplying of the CTAs of an SM spread
    // in time.  200,003 rows, staying and not: 17 features x 128 columns 69 and 74 us, 33 x 128 97 and 95 (p-stable 115 and 119), 50 x
    // 128 137 and 120, 98 x 224 355 and 342, 201 x 1,008 2,963 and 2,760, p-stable 98 x 128 243 and 218; 17 x 16 27 and 31, 50 x 32
    // 45 and 48, 66 x 32 55 and 55; 20,000 x 100 x 128 33.5 and 35.3.
    const int steps = (int)ceil_div(a.tables_per_group * k, 16);  // of eight columns, of a warp
    const size_t n_groups = ceil_div(L, a.tables_per_group), n_blocks = row_blocks(n, PF_BM), places = 2 * (size_t)c->sm_count;
    const int stay_stages = steps <= (family == CULSH_PSLSH ? 4 : 2) ? 4 : 3;
    const bool stay = ((int)ceil_div(d, PF_BK) <= stay_stages || n_blocks * n_groups <= 2 * places) &&
                      places / n_groups * n_groups * 10 >= places * 9;
    const dim3 grid((unsigned)(n_groups * (stay ? std::min<size_t>(n_blocks, places / n_groups) : n_blocks)));
    auto go = [&](auto kern) {
        CU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PF_SMEM));
        kern<<<grid, PF_THREADS, PF_SMEM, stream>>>(a);
        KERNEL_CHECK();
    };
    auto with_steps = [&](auto nf) {
        constexpr int NF = decltype(nf)::value;
        if (family == CULSH_RPLSH) go(project_f64_kernel<CULSH_RPLSH, NF>);
        else go(project_f64_kernel<CULSH_PSLSH, NF>);
    };
    // Forms of every second number of steps, and 7, which two groups of 112 columns take; the others round up to columns of
    // zeros.  That is still faster than a branch before every step, which left these out: 100 features x 80 columns in 6 steps for 5
    // 160 us in place of 225, x 48 in 4 for 3 116 in place of 216, x 16 in 2 for 1 72 in place of 207.
    if (steps <= 2) with_steps(std::integral_constant<int, 2>{});
    else if (steps <= 4) with_steps(std::integral_constant<int, 4>{});
    else if (steps <= 6) with_steps(std::integral_constant<int, 6>{});
    else if (steps == 7) with_steps(std::integral_constant<int, 7>{});
    else with_steps(std::integral_constant<int, 8>{});
    return true;
}

}  // namespace culsh_b200
