// Tensor-core (tcgen05) tile kernel for pointwise Conv2D / Gemm / MatMul, int8 and int16.
//
//   out[m, n] = epilogue( sum_k A[m, k] * W[n][k] + bias[n] )         m = pixel, n = output channel
//
// Replaces dl::base::conv2d<> for 1x1 filters (esp-dl/dl/base/dl_base_conv2d.cpp:9-60 conv2d_11cn,
// epilogue esp-dl/dl/base/dl_base_activate_buffer.hpp:27-73), which is also what Gemm and MatMul
// run (esp-dl/dl/module/include/dl_module_gemm.hpp:85-123).
//
// Structure (one persistent CTA per SM, 18 warps):
//   warp 0    TMA producer: cp.async.bulk.tensor 2-D tiles of A (128 rows x SWZ bytes of K) and of W (BLOCK_N rows x
//             SWZ bytes) into a ring of shared-memory stages, swizzled so that the MMA reads them without bank
//             conflicts; rows/columns past the tensor are zero-filled by the TMA unit, so ragged M, N and K need no
//             separate code.
//   warp 1    MMA issuer: one thread issues tcgen05.mma kind::i8 (M=128, N=BLOCK_N, K=32 per instruction), accumulating
//             int32 in TMEM; tcgen05.commit releases the stage and, at the end of a tile, hands the accumulator over.
//   warps 2-17 epilogue, four groups of four warps (a warp may read only its quarter of the 128 TMEM lanes).  With
//             four accumulator buffers each group owns one buffer and every fourth tile; with two buffers two groups
//             share a tile and split its columns.  tcgen05.ld, bias + ESP-DL's shift/round/saturate with per-channel
//             shifts, ReLU, optional 8-bit LUT, then a warp's 32 rows leave with a TMA store of their own.
//             Most layers the network workloads bring are memory bound with a few hundred int8 outputs per input
//             row, so the epilogue's instruction count per output decides the kernel's speed: per-channel constants
//             are staged once in shared memory in a form that needs one add and one shift per output (see
//             tc_common.cuh), and saturation happens inside the pack instruction.  A thread holds fragments of several rows
//             (epilogue_frag), so that a constant read from shared memory serves four results; a thread holds a row
//             where the columns are no multiple of 16, every image has its own filter, or a table is fused in.
//
// Short reductions over many rows keep the filter in shared memory (RES, plan_resident), a form of the kernel of its own.
//
// int16 operands: Blackwell tensor cores have no 16-bit integer MMA.  A pre-pass (pack.cu) writes each operand as two byte
// planes, the input's x = 256*hi + lo (hi signed) and the shifted filter's w + 32768 = 256*uh + ul (both unsigned), and the
// tile kernel accumulates hi*uh, hi*ul + lo*uh and lo*ul in three neighbouring TMEM accumulators: the filter's planes lie one
// behind the other in shared memory, so ONE instruction of twice the width multiplies hi by both (into accumulators 0, 1)
// and one multiplies lo by both (into 1, 2): half the instructions of four separate products, and each wide enough to be bound
// by its math (max(N/2, 32 + N/4) cycles at M = 128).  The epilogue recombines in two 32-bit halves (requant_wide; 64 bits for
// shifts outside 1 .. 31) and takes off 32768 * (sum of the input row).  Exact as long as K <= 16384 (a partial sum stays below
// 97,665 * K < 2^31).  4096x1024x1024 with the packing: 85 us with four products and 64-bit sums, 25 with one set of accumulators, 23 now.
//
// Every mbarrier wait is bounded (about two seconds); on expiry the kernel records ESPDL_ERR_TIMEOUT in the mapped host word
// (common.cuh) that espdl_b200_stream_sync reports, and all roles leave.
#include "tc_common.cuh"

#include <mutex>

namespace espdl {

__device__ int *g_tc_error = nullptr; // the status word of bounded waits (common.cuh)

int bind_device_error(int *word)
{
    ESPDL_CUDA_TRY(cudaMemcpyToSymbol(g_tc_error, &word, sizeof(word)));
    return ESPDL_OK;
}

// Role cycle counters of the tile kernel, compiled in only with -DESPDL_TC_TIMING (a measurement build; the product
// build carries none of it): per CTA, cycles the producer waited for a free stage, the MMA issuer waited for an
// accumulator / for a stage / spent issuing, and epilogue group 0 waited for an accumulator / spent working.
#ifdef ESPDL_TC_TIMING
__device__ long long g_tc_timing[256 * 8];
#define TC_LAP_INIT long long t_ = clock64()
#define TC_LAP(var) do { const long long n_ = clock64(); (var) += n_ - t_; t_ = n_; } while (0)
#define TC_REC(slot, var) g_tc_timing[blockIdx.x * 8 + (slot)] = (var)
__device__ long long g_tc_clock[256 * 4]; // per CTA: clock64 and globaltimer at entry and at exit
#define TC_STAMP(i) do { if (threadIdx.x == 0) { unsigned long long g_; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(g_)); \
    g_tc_clock[blockIdx.x * 4 + 2 * (i)] = clock64(); g_tc_clock[blockIdx.x * 4 + 2 * (i) + 1] = (long long)g_; } } while (0)
#else
#define TC_STAMP(i)
#define TC_LAP_INIT
#define TC_LAP(var)
#define TC_REC(slot, var)
#endif

namespace {

using namespace tc;

constexpr int BLOCK_M = 128;
constexpr int EPI_WARPS = 16;
constexpr int NUM_THREADS = 64 + EPI_WARPS * 32; // 1 TMA warp + 1 MMA warp + 16 epilogue warps
constexpr int MAX_STAGES = 12;
constexpr int MAX_ACC = 8;

struct TcParams {
    int early; // bias, exponents and table are constants of the model: read ahead of the previous kernel's end
    int filter_early; // so is the filter: not one that was packed, which the launch directly before writes
    int M, N, K;    // rows per matrix, output channels, reduction length
    int batch;      // independent matrices (1 unless every image has its own filter)
    int block_n, n_tiles, m_tiles;
    int swz;        // bytes of K per stage row: 32, 64 or 128
    int k_blocks;   // ceil(K / swz)
    int stages;
    int acc_stages; // TMEM accumulator buffers: 8, 4, 2 or 1 (int8), 2 or 1 sets of three (int16)
    int tmem_cols;  // power of two >= 32
    int out_pw;     // staged epilogue: bytes per row of a group's output piece (0 = rows are stored directly); int16: a quarter
                    // of the bytes per row of the one tile that all groups share
    int one_tile;   // a CTA has one tile: all four epilogue groups share it, and it is staged in the memory its loads came through
    int out_rows;   // the staging tiles leave row by row, a warp per row (rows that no TMA store can address), not as one TMA store
    int out_mask;   // swizzle mask of the staging tiles (7, 3, 1, 0)
    int frag;       // staged epilogue on fragments: the columns of a tile are channels in the order frag_channel (map_b has five dimensions)
    void *out;
    long long ops;  // output row stride in elements
    const int *row_sum; // int16: sum of every row of A
    const int8_t *res; // optional residual added to the result (same rows as the output), or null
    long long rps;     // residual row stride in elements
    long long peer_delta[7]; // byte distance from `out` to the same buffer on other GPUs: every result row is stored there too
    int n_peer;
    unsigned *sched; // {next tile, CTAs done}: the tiles from static_tiles on are handed out by this counter; null = fixed walk
    int static_tiles; // tiles walked in the fixed order (a multiple of the grid size; all of them without a counter); resident: row tiles
    int resident;     // the filter stays in shared memory, see plan_resident: column tiles of a CTA (0: tiles bring their part of it with them)
    int in_turn;      // resident: epilogue groups take two accumulators in turn and stage pieces of 64 columns in two buffers, see plan_resident
    int n_groups;     // resident: groups of CTAs, each with its own column tiles (resident_share)
    int share, shares; // what a row tile costs a group, and all groups (the last one's columns may be fewer)
    EpiConfig epi;
};

constexpr int TILE_RING = 32; // tile numbers on their way from the producer to the MMA issuer (more than stages + accumulators)

// Epilogue of one int8 tile for outputs that cannot go through the staged path (piece widths that are not whole
// 16-byte groups, unaligned rows, channels outside the fast form): rows are stored directly from registers.  WIDE: in 256-bit stores where they
// are aligned, as part of the kernel only: in a function of its own such a store wrote its first word and no more (nvcc 12.9).
template <bool EVEN, bool WIDE>
__device__ __forceinline__ void epilogue_direct(const TcParams &p, const FastParam *fast_s, uint32_t fp_base, uint32_t t0, long long m, int n0,
                                                bool row_ok, bool fast, int parts, int part, uint32_t tbl)
{
    int8_t *orow = (int8_t *)p.out + m * p.ops + n0;
    const bool vec_ok = (p.ops % 16 == 0) && ((((uintptr_t)p.out) + n0) % 16 == 0);
    // what every row start (and every 16-column step from it) is aligned to
    const uintptr_t amix = (uintptr_t)p.ops | (((uintptr_t)p.out) + (uintptr_t)n0) | 16u;
    const int out_align = (int)(amix & (~amix + 1));
    if (fast && !tbl && vec_ok && p.N % 16 == 0 && !p.res && p.n_peer == 0) {
        // whole 16-column groups, aligned rows, one-add-one-shift constants
        const bool wide = WIDE && (p.ops % 32 == 0) && ((((uintptr_t)p.out) + n0) % 32 == 0);
        const uint32_t fp = fp_base + (uint32_t)n0 * 8u;
        const int ncols = min(p.block_n, p.N - n0);
        if (p.epi.relu)
            epilogue_lean<true, EVEN>(t0, fp, orow, ncols, parts, part, row_ok, wide);
        else
            epilogue_lean<false, EVEN>(t0, fp, orow, ncols, parts, part, row_ok, wide);
        return;
    }
    int chunk = 0;
    for (int c0 = 0; c0 < p.block_n; c0 += 32, chunk++) {
        if (chunk % parts != part)
            continue;
        const bool two = c0 + 32 <= p.block_n;
        int32_t v[32];
        ld16(t0 + c0, v);
        if (two)
            ld16(t0 + c0 + 16, v + 16);
        ld_wait16(v);
        tie16(v + 16);
        uint32_t pk[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (fast) {
            if (p.epi.relu) {
                requant16_fast<true, EVEN>(v, fast_s + n0 + c0, pk);
                if (two)
                    requant16_fast<true, EVEN>(v + 16, fast_s + n0 + c0 + 16, pk + 4);
            } else {
                requant16_fast<false, EVEN>(v, fast_s + n0 + c0, pk);
                if (two)
                    requant16_fast<false, EVEN>(v + 16, fast_s + n0 + c0 + 16, pk + 4);
            }
            if (tbl) { // a fused table on rows that leave unstaged (`tbl`: its shared-memory copy): same lookups on the packed words
#pragma unroll
                for (int q = 0; q < 8; q++) pk[q] = lut4(pk[q], tbl);
            }
        } else {
            requant16_general(v, p.epi, n0 + c0, p.N, pk);
            if (two)
                requant16_general(v + 16, p.epi, n0 + c0 + 16, p.N, pk + 4);
        }
        if (row_ok) {
            const int count = min(two ? 32 : 16, p.N - (n0 + c0));
            if (count > 0 && p.res) { // folded Add: saturating byte sums with the residual's row
                const int8_t *rrow = p.res + m * p.rps + n0 + c0;
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (j < count) {
                        const int sum = (int)(int8_t)(pk[j >> 2] >> (8 * (j & 3))) + (int)rrow[j];
                        pk[j >> 2] = (pk[j >> 2] & ~(0xffu << (8 * (j & 3)))) | (((uint32_t)max(-128, min(127, sum)) & 0xffu) << (8 * (j & 3)));
                    }
            }
            // copies of the rows in other GPUs' memory (peer-mapped pointers): plain stores, the same words
            for (int pi = 0; pi < p.n_peer && count > 0; pi++) {
                int8_t *prow = orow + c0 + p.peer_delta[pi];
                store_bytes(prow, pk, min(count, 16), out_align);
                if (count > 16)
                    store_bytes(prow + 16, pk + 4, count - 16, out_align);
            }
            if (WIDE && count > 0) {
                store_bytes(orow + c0, pk, count, out_align);
            } else if (count > 0) {
                store_bytes(orow + c0, pk, min(count, 16), out_align);
                if (count > 16)
                    store_bytes(orow + c0 + 16, pk + 4, count - 16, out_align);
            }
        }
    }
}

// Out of line: the other paths of a kernel then carry none of this code's registers.
template <bool EVEN>
__device__ __noinline__ void epilogue_direct_tile(const TcParams &p, const FastParam *fast_s, uint32_t fp_base, uint32_t t0, long long m, int n0, bool row_ok, bool fast,
                                                  int parts, int part, uint32_t tbl)
{
    epilogue_direct<EVEN, false>(p, fast_s, fp_base, t0, m, n0, row_ok, fast, parts, part, tbl);
}

// The general epilogue of a tile whose columns are channels in the order frag_channel (a channel outside the fast form, or tables of channels): 16 columns
// at a time, put back into order, columns whole groups of 16.  Residual rows are 16-byte aligned, rows of results begin anywhere (those that leave by warps).
__device__ __noinline__ void epilogue_frag_general(const TcParams &p, uint32_t t0, long long m, int n0, bool row_ok, int parts, int part)
{
    const int ncols = min(p.block_n, p.N - n0);
    int8_t *orow = (int8_t *)p.out + m * p.ops + n0;
    const int8_t *rrow = p.res + m * p.rps + n0;
    const uintptr_t amix = (uintptr_t)p.ops | (uintptr_t)p.out | (uintptr_t)n0 | 16u; // see epilogue_direct
    const int out_align = (int)(amix & (~amix + 1));
#pragma unroll 1
    for (int c0 = 16 * part; c0 < ncols; c0 += 16 * parts) {
        int32_t u[16], v[16];
        ld16(t0 + c0, u);
        ld_wait16(u);
#pragma unroll
        for (int j = 0; j < 16; j++) v[frag_channel(j)] = u[j];
        uint32_t pk[4];
        requant16_general(v, p.epi, n0 + c0, p.N, pk);
        if (!row_ok)
            continue;
        if (p.res) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t r = *(const uint32_t *)(rrow + c0 + 4 * q);
                uint32_t w = 0;
#pragma unroll
                for (int i = 0; i < 4; i++)
                    w |= ((uint32_t)max(-128, min(127, (int)(int8_t)(pk[q] >> (8 * i)) + (int)(int8_t)(r >> (8 * i)))) & 0xffu) << (8 * i);
                pk[q] = w;
            }
        }
        store_bytes(orow + c0, pk, 16, out_align);
    }
}

// One row of a staging tile to global memory by a whole warp: `len` bytes at offset `at` of the tile at `buf` (16-byte chunks swizzled
// as the stages wrote them) to `dst`, any alignment.  A thread that stores its own unaligned row issues byte stores that touch 32
// rows each; here a store instruction covers 128 consecutive bytes (25385 rows of 409 bytes, K = 170: 128 us before).
__device__ __forceinline__ uint32_t staged_word(uint32_t buf, uint32_t off, uint32_t mask)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(buf + (off ^ (((off >> 7) & mask) << 4))));
    return v;
}

// `rows` of them, `step` bytes apart in the tile and `pitch` in global memory.  Four at a time: one row's loads, shifts and stores after the other's took a tile
// 3.3 us whatever its width (49314 rows of 16 -> 1634: 114 us, now 72; 20000 of 256 -> 333 25.4 / 15.6; 60000 of 48 -> 99 19.1 / 11.6).
__device__ __forceinline__ void store_staged_rows(int8_t *dst, long long pitch, uint32_t buf, uint32_t at, uint32_t step, int rows, int len, uint32_t mask, int lane)
{
    constexpr int U = 4;
    const int eu = lane >> 3, ei = lane & 7; // head and tail bytes, at most six a row: eight lanes a row
    for (int i = 0; i < rows; i += U, dst += U * pitch, at += U * step) {
        for (int w = lane; 4 * (w - lane) < len; w += 32) {
            uint32_t a[U], b[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int head = (int)((0u - (uint32_t)(uintptr_t)(dst + u * pitch)) & 3u);
                const uint32_t off = at + (uint32_t)u * step + 4u * (uint32_t)w; // the aligned word that holds the first byte (head < 4)
                a[u] = b[u] = 0u;
                if (i + u < rows && head + 4 * w + 4 <= len) {
                    a[u] = staged_word(buf, off, mask);
                    if (head)
                        b[u] = staged_word(buf, off + 4, mask);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int head = (int)((0u - (uint32_t)(uintptr_t)(dst + u * pitch)) & 3u);
                if (i + u < rows && head + 4 * w + 4 <= len)
                    *(uint32_t *)(dst + u * pitch + head + 4 * w) = __funnelshift_r(a[u], b[u], 8u * (uint32_t)head);
            }
        }
        int8_t *edge = dst + eu * pitch;
        const int head = min((int)((0u - (uint32_t)(uintptr_t)edge) & 3u), len), words = (len - head) >> 2;
        if (i + eu < rows && ei < len - 4 * words) {
            const int byte = ei < head ? ei : ei + 4 * words;
            const uint32_t off = at + (uint32_t)eu * step + (uint32_t)byte;
            edge[byte] = (int8_t)(staged_word(buf, off & ~3u, mask) >> (8 * (off & 3u)));
        }
    }
}

// The three sums of an int16 result in halves (HalvesParam; K <= 16384 keeps H below 2^30).  64-bit sums took 4100 cycles for 16 columns of a tile, and
// 31 us for 4096x1024x1024, 26 so.
template <bool EVEN>
__device__ __forceinline__ int requant_wide(int vh, int vm, int vl, int row_h, int row_l, const HalvesParam c)
{
    return shift_halves<EVEN>(vh + (vm >> 8) + (c.h + row_h), (int)__byte_perm((uint32_t)vm, 0u, 0x4404) + vl + c.l + row_l, c); // (the low byte of vm in the second)
}

// Whose column tiles a CTA has: group g has tiles g * resident .. + resident - 1 of the filter and a share of the CTAs in proportion to what a row tile costs it.
struct ResidentShare {
    int first, across;   // column tiles
    int member, members; // this CTA's place in its group
};
__device__ __forceinline__ ResidentShare resident_share(const TcParams &p)
{
    const int grid = (int)gridDim.x;
    int g = 0, begin = 0, end = grid;
    for (; g < p.n_groups; g++, begin = end) {
        end = g + 1 == p.n_groups ? grid : (int)((long long)grid * ((g + 1) * p.share) / p.shares);
        if ((int)blockIdx.x < end)
            break;
    }
    return {g * p.resident, min(p.resident, p.n_tiles - g * p.resident), (int)blockIdx.x - begin, end - begin};
}

// The producer's walk with a resident filter (plan_resident): the CTA's column tiles of the filter once, then the rows of its tiles, each row tile
// once for all neighbouring column tiles.  A ring entry is the first of `count` tiles.  With a counter the CTAs go through the first p.static_tiles row
// tiles side by side and the tiles of the others are handed out one at a time, asked for one ahead; without, a CTA has an equal run of its
// group's tiles.  False when a wait ran out.
__device__ __forceinline__ bool produce_resident(const TcParams &p, const CUtensorMap &map_a, const CUtensorMap &map_b, uint32_t smem, uint64_t *full_bar,
                                                 uint64_t *empty_bar, uint64_t *filter_bar, volatile int *ring_row, volatile int *ring_col)
{
    const int a_bytes = BLOCK_M * p.swz, b_bytes = p.block_n * p.swz;
    const ResidentShare share = resident_share(p);
    const int first = share.first, across = share.across, member = share.member, members = share.members;
    if (!p.filter_early)
        grid_dep_wait(); // outside a model's plan a caller may just have written the filter, and a packed one is what the launch before writes
    const uint32_t fbar = smem_u32(filter_bar), filter = smem + (uint32_t)(p.stages * a_bytes);
    mbar_arrive_expect_tx(fbar, (uint32_t)(across * p.k_blocks * b_bytes));
    for (int j = 0; j < across; j++)
        for (int kb = 0; kb < p.k_blocks; kb++) {
            const uint32_t to = filter + (uint32_t)((j * p.k_blocks + kb) * b_bytes);
            if (p.frag)
                tma_load_5d(to, &map_b, kb * p.swz, 0, 0, 0, (first + j) * p.block_n >> 4, fbar);
            else
                tma_load_3d(to, &map_b, kb * p.swz, (first + j) * p.block_n, 0, fbar);
        }
    grid_dep_wait();
    int stage = 0, local = 0;
    uint32_t phase = 0;
    auto put = [&](int row, int j, int count) {
        ring_row[local & (TILE_RING - 1)] = row;
        ring_col[local & (TILE_RING - 1)] = first + j + (count << 16);
        local++;
        for (int kb = 0; kb < p.k_blocks; kb++) {
            if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1))
                return false;
            const uint32_t bar = smem_u32(&full_bar[stage]);
            mbar_arrive_expect_tx(bar, (uint32_t)a_bytes);
            tma_load_3d(smem + (uint32_t)(stage * a_bytes), &map_a, kb * p.swz, row * BLOCK_M, 0, bar);
            if (++stage == p.stages)
                stage = 0, phase ^= 1;
        }
        return true;
    };
    const int total = p.m_tiles * across, fixed = p.static_tiles * across;
    if (p.sched) {
        int next = fixed + (int)atomicAdd(p.sched, 1u);
        for (int row = member; row < p.static_tiles; row += members)
            if (!put(row, 0, across))
                return false;
        while (next < total) {
            const int row = next / across, j = next - row * across;
            next = fixed + (int)atomicAdd(p.sched, 1u);
            if (!put(row, j, 1))
                return false;
        }
    } else {
        const int end = (int)((long long)total * (member + 1) / members);
        for (int u = (int)((long long)total * member / members); u < end;) {
            const int row = u / across, j = u - row * across, count = min(across - j, end - u);
            if (!put(row, j, count))
                return false;
            u += count;
        }
    }
    ring_row[local & (TILE_RING - 1)] = -1; // the end: one stage without data
    if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1))
        return false;
    mbar_arrive(smem_u32(&full_bar[stage]));
    return true;
}

// The MMA issuer's side: the row tile's stages are waited for at the first of its tiles and given back at the last.  One thread does this beside warps
// that keep its scheduler busy, so its instructions count: with the descriptors, barriers and divisions worked out for each tile it took 740 cycles for
// a tile whose products take 256 (128 x 128, K = 128).
__device__ __forceinline__ bool multiply_resident(const TcParams &p, uint32_t smem, uint32_t tmem_base, uint64_t *full_bar, uint64_t *empty_bar, uint64_t *filter_bar,
                                                  uint64_t *tfull_bar, uint64_t *tempty_bar, volatile int *ring_row, volatile int *ring_col, volatile int *epi_row, volatile int *epi_col)
{
    const uint32_t idesc = idesc_i8(1, 1, BLOCK_M, p.block_n);
    const int b_bytes = p.block_n * p.swz, ksteps = p.swz / 32;
    const int last_ksteps = (p.K - (p.k_blocks - 1) * p.swz + 31) / 32; // see the other walk
    const uint32_t a_units = (uint32_t)(BLOCK_M * p.swz) >> 4, b_units = (uint32_t)b_bytes >> 4; // 16-byte units, as descriptors count
    const uint64_t a_desc = smem_desc_swizzled(smem, p.swz), b_desc = smem_desc_swizzled(smem + (uint32_t)(p.stages * BLOCK_M * p.swz), p.swz);
    const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar), tfull0 = smem_u32(tfull_bar), tempty0 = smem_u32(tempty_bar);
    const uint32_t filter_units = (uint32_t)p.k_blocks * b_units;
    const int first = resident_share(p).first;
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 1, d0 = tmem_base;
    if (!mbar_wait(smem_u32(filter_bar), 0))
        return false;
    long long w_tempty = 0, w_full = 0, w_issue = 0;
    (void)w_tempty, (void)w_full, (void)w_issue;
    TC_LAP_INIT;
    for (int local = 0;; local++) {
        TC_LAP(w_issue);
        if (!mbar_wait(full0 + 8u * (uint32_t)stage, phase))
            return false;
        TC_LAP(w_full);
        const int row = ring_row[local & (TILE_RING - 1)], cols = ring_col[local & (TILE_RING - 1)];
        if (row < 0)
            break;
        const int col0 = cols & 0xffff, end = col0 + (cols >> 16);
        uint64_t db = b_desc + (uint32_t)(col0 - first) * filter_units;
        int s = stage;
        uint32_t ph = phase;
        for (int col = col0; col < end; col++) {
            TC_LAP(w_issue);
            if (!mbar_wait(tempty0 + 8u * (uint32_t)acc, acc_phase))
                return false;
            TC_LAP(w_tempty);
            fence_after();
            epi_row[acc] = row;
            epi_col[acc] = col;
            s = stage, ph = phase;
            for (int kb = 0; kb < p.k_blocks; kb++) {
                if (kb != 0 && col == col0) {
                    if (!mbar_wait(full0 + 8u * (uint32_t)s, ph))
                        return false;
                    fence_after();
                }
                const uint64_t da = a_desc + (uint32_t)s * a_units;
                const int ks = kb == p.k_blocks - 1 ? last_ksteps : ksteps;
                mma_i8(d0, da, db, idesc, kb != 0 ? 1u : 0u);
                if (ks > 1)
                    mma_i8(d0, da + 2, db + 2, idesc, 1u);
                if (ks > 2)
                    mma_i8(d0, da + 4, db + 4, idesc, 1u);
                if (ks > 3)
                    mma_i8(d0, da + 6, db + 6, idesc, 1u);
                if (col == end - 1)
                    commit(empty0 + 8u * (uint32_t)s);
                db += b_units;
                if (++s == p.stages)
                    s = 0, ph ^= 1;
            }
            commit(tfull0 + 8u * (uint32_t)acc);
            mbar_arrive(tfull0 + 8u * (uint32_t)acc); // publishes epi_row / epi_col[acc]
            d0 += (uint32_t)p.block_n;
            if (++acc == p.acc_stages)
                acc = 0, acc_phase ^= 1, d0 = tmem_base;
        }
        stage = s, phase = ph; // (a row tile may have more blocks than the ring has stages)
    }
    TC_REC(2, w_tempty);
    TC_REC(3, w_full);
    TC_REC(4, w_issue);
    for (int a = 0; a < p.acc_stages; a++) { // every accumulator's epilogue groups are told, in the order they wait
        if (!mbar_wait(tempty0 + 8u * (uint32_t)acc, acc_phase))
            return false;
        epi_row[acc] = -1;
        mbar_arrive(tfull0 + 8u * (uint32_t)acc);
        mbar_arrive(tfull0 + 8u * (uint32_t)acc);
        if (++acc == p.acc_stages)
            acc = 0, acc_phase ^= 1;
    }
    return true;
}

// The epilogue beside a resident filter: pieces of 64 columns.  A loop of its own, one for each KIND (0 plain, 1 fused table, 2 folded Add): what a warp does for
// a piece besides requantising it stands between its tiles.  A warp stores its own 32 rows, so the warps of a group need no
// barrier, and an accumulator is given back when its sums are in registers.  False when a wait ran out.
template <bool EVEN, int KIND>
__device__ __forceinline__ bool epilogue_resident(const TcParams &p, const CUtensorMap &map_out, uint32_t tmem_base, uint32_t fp_base, uint32_t stage, uint64_t *tfull_bar,
                                                  uint64_t *tempty_bar, volatile int *epi_row, volatile int *epi_col, uint32_t tbl, int group, int lane_group, int lane)
{
    constexpr int PIECE = 64, PIECE_BYTES = BLOCK_M * PIECE;
    const int sets = p.acc_stages / 2, last_part = 4 / sets - 1, set = group % sets, block_n = p.block_n, N = p.N, M = p.M - lane_group * 32;
    const int floor_q = p.epi.relu ? 0 : INT_MIN;
    const uint32_t tfull0 = smem_u32(tfull_bar), tempty0 = smem_u32(tempty_bar), tmem = tmem_base + ((uint32_t)(lane_group * 32) << 16);
    int acc = set, part = group / sets;
    uint32_t phase = 0, buf = stage + (uint32_t)(2 * group * PIECE_BYTES);
    long long w_tfull = 0, w_work = 0, w_store = 0;
    (void)w_tfull, (void)w_work, (void)w_store;
    TC_LAP_INIT;
    while (true) {
        TC_LAP(w_work);
        if (!mbar_wait(tfull0 + 8u * (uint32_t)acc, phase))
            return false;
        TC_LAP(w_tfull);
        const int row = epi_row[acc];
        if (row < 0)
            break;
        const int n = epi_col[acc] * block_n + part * PIECE, cols = min(PIECE, N - n);
        fence_after();
        if (elect_one())
            bulk_wait_read_but_one(); // the store out of this buffer has read it, the other buffer's (the last piece's) may be under way
        __syncwarp();
        TC_LAP(w_store);
        const uint32_t t0 = tmem + (uint32_t)(acc * block_n + part * PIECE), fp = fp_base + (uint32_t)n * 8u;
        auto loaded = [&] {
            fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(tempty0 + 8u * (uint32_t)acc);
        };
        if (KIND == 0 && cols == 64) {
            epilogue_frag<PIECE, 64, EVEN>(t0, fp, buf, lane_group, lane, floor_q, loaded);
        } else if (KIND == 0 && cols == 32) {
            epilogue_frag<PIECE, 32, EVEN>(t0, fp, buf, lane_group, lane, floor_q, loaded);
        } else {
            if (KIND == 1)
                epilogue_frag_lut<EVEN>(t0, fp, buf, lane_group, lane, cols, PIECE, 3u, floor_q, tbl);
            else if (KIND == 2)
                epilogue_frag_residual<EVEN>(t0, fp, buf, lane_group, lane, cols, PIECE, 3u, floor_q, p.res + (long long)row * BLOCK_M * p.rps + n, p.rps, p.M - row * BLOCK_M);
            else
                epilogue_frag_each(t0, fp, buf, lane_group, lane, cols, PIECE, 3u, [=](const int32_t *v, int i, const FragConst &k) { return frag_word<EVEN>(v, i, k, floor_q); });
            loaded();
        }
        fence_async_smem();
        __syncwarp();
        if (elect_one()) {
            if (cols > 0 && row * BLOCK_M < M) // rows >= M and columns >= N are clipped
                tma_store_3d(&map_out, buf + (uint32_t)(lane_group * 32 * PIECE), n, row * BLOCK_M + lane_group * 32, 0);
            bulk_commit(); // an empty group for a piece without columns, too: the wait above counts pieces
        }
        __syncwarp();
        // The other accumulator and buffer.  Pieces of a tile of 65 to 127 columns change hands, they are not two of 64.
        part = last_part - part;
        if (acc == set) {
            acc = set + sets, buf += PIECE_BYTES;
        } else {
            acc = set, buf -= PIECE_BYTES;
            phase ^= 1;
        }
    }
    if (elect_one())
        bulk_wait_all(); // shared memory stays allocated until the last store has left it
    __syncwarp();
    if (group == 0 && lane_group == 2 && lane == 0) {
        TC_REC(5, w_tfull);
        TC_REC(6, w_work);
        TC_REC(7, w_store);
    }
    return true;
}

// RES: the filter is resident (plan_resident), a kernel of its own so that neither form carries the other's code.
template <bool I16, bool EVEN, bool RES>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_a_lo, const __grid_constant__ CUtensorMap map_b_lo,
               const __grid_constant__ CUtensorMap map_out, const __grid_constant__ TcParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int NPLANE = I16 ? 2 : 1;
    constexpr int NACC = I16 ? 3 : 1;
    const int a_bytes = BLOCK_M * p.swz;
    const int b_bytes = p.block_n * p.swz;
    const int stage_bytes = RES ? a_bytes : NPLANE * (a_bytes + b_bytes);
    const int load_bytes = p.stages * stage_bytes + (RES ? (p.resident * p.k_blocks * b_bytes + 1023) & ~1023 : 0); // the ring, then a resident filter
    const int n_pad = p.n_tiles * p.block_n;
    uint8_t *out_stage = p.one_tile ? smem : smem + load_bytes; // 4 tiles of [128][out_pw] bytes, 1024-byte aligned each
    const int out_tile_bytes = ((BLOCK_M * p.out_pw + 1023) & ~1023) << (RES ? p.in_turn : 0); // (in turn: of two buffers)
    uint8_t *aux = smem + load_bytes + (p.one_tile ? 0 : 4 * (size_t)out_tile_bytes);
    FastParam *fast_s = (FastParam *)aux; // n_pad entries, 16-byte aligned (block_n % 16 == 0)
    HalvesParam *wide_s = (HalvesParam *)aux; // int16: the current tile's columns
    uint64_t *bars = (uint64_t *)(aux + (I16 ? sizeof(HalvesParam) * (size_t)p.block_n : sizeof(FastParam) * (size_t)n_pad));
    uint64_t *full_bar = bars, *empty_bar = bars + MAX_STAGES, *tfull_bar = bars + 2 * MAX_STAGES, *tempty_bar = tfull_bar + MAX_ACC;
    uint64_t *filter_bar = tempty_bar + MAX_ACC;
    uint32_t *tmem_slot = (uint32_t *)(filter_bar + 2); // (16-byte aligned)
    int *slow_flag = (int *)(tmem_slot + 1);
    uint8_t *lut_s = (uint8_t *)(slow_flag + 3); // the fused 8-bit table, 256 bytes, 16-byte aligned
    volatile int *ring_row = (volatile int *)(lut_s + 256); // TILE_RING tiles, producer -> MMA issuer: row tile, column tile
    volatile int *ring_col = ring_row + TILE_RING;          // (resident: the first of `col >> 16` neighbouring ones)
    volatile int *epi_row = ring_col + TILE_RING;           // MAX_ACC tiles, MMA issuer -> the accumulator's epilogue groups
    volatile int *epi_col = epi_row + MAX_ACC;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    TC_STAMP(0);
    const int total_tiles = p.batch * p.m_tiles * p.n_tiles;
    const int sets = RES && p.in_turn ? p.acc_stages / 2 : p.acc_stages;
    const int parts = I16 ? 4 : 4 / sets; // epilogue groups that share one tile (they split its columns)
    // Tiles are numbered n-fastest: tile = row_tile * n_tiles + n_tile with row_tile running over batch x m_tiles.  A CTA
    // starts with tile blockIdx.x; every further tile comes from a global counter (p.sched), so that an SM that runs
    // slower than the others (measured: one in ten takes 15-25 % longer per tile) gets fewer tiles instead of setting
    // the kernel's duration.  The producer fetches the numbers and passes them on through shared memory: to the MMA
    // issuer in a ring (published by the arrive on the first stage's "full" barrier), from there to the epilogue groups
    // (published by a plain arrive on the accumulator's "full" barrier, which therefore counts two arrivals: that one
    // and the tensor cores' commit).  A negative number ends the walk.

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int a = 0; a < MAX_ACC; a++) {
            mbar_init(smem_u32(&tfull_bar[a]), 2);
            mbar_init(smem_u32(&tempty_bar[a]), 4 * parts);
        }
        mbar_init(smem_u32(filter_bar), 1);
        *slow_flag = 0;
        fence_barrier_init();
    }
    if (threadIdx.x == 32 * 2) { // an epilogue thread: the descriptors are in the cache when the first copies are issued
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_b);
        if (I16) {
            prefetch_tensormap(&map_a_lo);
            prefetch_tensormap(&map_b_lo);
        }
        if (p.out_pw && !p.out_rows)
            prefetch_tensormap(&map_out);
    }
    if (warp == 1)
        tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // This CTA is set up: the next kernel's CTAs may take SMs as they become free.  The producer below waits for the previous kernel before
    // its first load, so do the epilogue warps before they read the channels' constants (outside a model's plan, where a caller may
    // just have written these), and every other role only ever acts on what the producer brought in.
    if (threadIdx.x == 0)
        grid_dep_launch();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        // One elected lane runs the loop and issues the copies.
        const bool issuer = elect_one();
        if (RES && issuer) {
            if (!produce_resident(p, map_a, map_b, smem_u32(smem), full_bar, empty_bar, filter_bar, ring_row, ring_col))
                report_timeout(g_tc_error);
        } else if (issuer) {
        grid_dep_wait(); // the previous kernel's output, and its use of the tile counter, before the first load
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        long long w_empty = 0, w_load = 0;
        (void)w_empty, (void)w_load;
        TC_LAP_INIT;
        // Tiles below p.static_tiles are walked in the fixed order (blockIdx.x, + gridDim.x, ...); the rest is handed out
        // by the counter, one number per tile and asked for one tile ahead (an atomic on a word that every SM hammers
        // takes ~1000 cycles to answer: with every tile handed out that way the producer no longer ran ahead)
        int tile = blockIdx.x; // the grid never has more CTAs than there are tiles
        bool handed = false;
        auto after = [&](int cur) {
            if (!handed && cur + (int)gridDim.x < p.static_tiles)
                return cur + (int)gridDim.x;
            if (!p.sched)
                return handed || cur + (int)gridDim.x >= total_tiles ? total_tiles : cur + (int)gridDim.x;
            handed = true;
            return p.static_tiles + (int)atomicAdd(p.sched, 1u);
        };
        int next = after(tile);
        int local = 0;
        for (; tile < total_tiles && ok; local++) {
            const int rows = tile / p.n_tiles, nt = tile - rows * p.n_tiles;
            ring_row[local & (TILE_RING - 1)] = rows;
            ring_col[local & (TILE_RING - 1)] = nt;
            const int bi = p.batch == 1 ? 0 : rows / p.m_tiles;
            const int m0 = (p.batch == 1 ? rows : rows % p.m_tiles) * BLOCK_M;
            const int n0 = nt * p.block_n;
            for (int kb = 0; kb < p.k_blocks; kb++) {
                TC_LAP(w_load);
                if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1)) {
                    ok = false;
                    break;
                }
                TC_LAP(w_empty);
                const uint32_t bar = smem_u32(&full_bar[stage]);
                const uint32_t st = smem_u32(smem) + (uint32_t)(stage * stage_bytes);
                mbar_arrive_expect_tx(bar, (uint32_t)stage_bytes);
                tma_load_3d(st, &map_a, kb * p.swz, m0, bi, bar);
                if (!I16 && p.frag)
                    tma_load_5d(st + a_bytes, &map_b, kb * p.swz, 0, 0, 0, n0 >> 4, bar);
                else
                    tma_load_3d(st + NPLANE * a_bytes, &map_b, kb * p.swz, n0, bi, bar);
                if (I16) {
                    tma_load_3d(st + a_bytes, &map_a_lo, kb * p.swz, m0, bi, bar);
                    tma_load_3d(st + 2 * a_bytes + b_bytes, &map_b_lo, kb * p.swz, n0, bi, bar);
                }
                if (++stage == p.stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            // the number after next is asked for one tile ahead of its use: the answer is back long before it is needed
            tile = next;
            if (tile < total_tiles)
                next = after(tile);
        }
        if (ok) {
            // end of the walk: one stage without data whose ring entry is negative
            ring_row[local & (TILE_RING - 1)] = -1;
            if (mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1))
                mbar_arrive(smem_u32(&full_bar[stage]));
            else
                ok = false;
        }
        if (!ok)
            report_timeout(g_tc_error);
        TC_REC(0, w_empty);
        TC_REC(1, w_load);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        // One elected lane runs the loop and issues.  A tcgen05.mma of M = 128 costs it about 50 cycles (250 when the lane was chosen by its
        // number, see elect_one), so that N = 128 and wider keep the tensor cores busy.
        const bool issuer = elect_one();
        if (RES && issuer) {
            if (!multiply_resident(p, smem_u32(smem), tmem_base, full_bar, empty_bar, filter_bar, tfull_bar, tempty_bar, ring_row, ring_col, epi_row, epi_col))
                report_timeout(g_tc_error);
        } else if (issuer) {
        int stage = 0;
        uint32_t phase = 0;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        long long w_tempty = 0, w_full = 0, w_issue = 0;
        (void)w_tempty, (void)w_full, (void)w_issue;
        TC_LAP_INIT;
        const uint32_t idesc_ss = idesc_i8(1, 1, BLOCK_M, p.block_n);
        const uint32_t idesc_su = idesc_i8(1, 0, BLOCK_M, 2 * p.block_n), idesc_uu = idesc_i8(0, 0, BLOCK_M, 2 * p.block_n); // int16: both planes
        const uint32_t idesc_uu1 = idesc_i8(0, 0, BLOCK_M, p.block_n);
        const int ksteps = p.swz / 32;
        const int last_ksteps = (p.K - (p.k_blocks - 1) * p.swz + 31) / 32; // 32-byte K steps of the last block that hold data
        const uint32_t smem_base = smem_u32(smem);
        for (int local = 0; ok; local++) {
            TC_LAP(w_issue);
            // the tile's first stage: its arrival publishes the tile number
            if (!mbar_wait(smem_u32(&full_bar[stage]), phase)) {
                ok = false;
                break;
            }
            TC_LAP(w_full);
            const int row = ring_row[local & (TILE_RING - 1)], col = ring_col[local & (TILE_RING - 1)];
            if (row < 0) {
                // end of the walk: every accumulator's epilogue groups are told, in the order they wait
                for (int a = 0; a < p.acc_stages && ok; a++) {
                    if (!mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1)) {
                        ok = false;
                        break;
                    }
                    epi_row[acc] = -1;
                    mbar_arrive(smem_u32(&tfull_bar[acc]));
                    mbar_arrive(smem_u32(&tfull_bar[acc]));
                    if (++acc == p.acc_stages) {
                        acc = 0;
                        acc_phase ^= 1;
                    }
                }
                break;
            }
            if (!mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1)) {
                ok = false;
                break;
            }
            TC_LAP(w_tempty);
            fence_after();
            epi_row[acc] = row;
            epi_col[acc] = col;
            const uint32_t d0 = tmem_base + (uint32_t)(acc * NACC * p.block_n);
            for (int kb = 0; kb < p.k_blocks; kb++) {
                TC_LAP(w_issue);
                if (kb != 0 && !mbar_wait(smem_u32(&full_bar[stage]), phase)) {
                    ok = false;
                    break;
                }
                TC_LAP(w_full);
                fence_after();
                const uint32_t st = smem_base + (uint32_t)(stage * stage_bytes);
                const uint64_t da = smem_desc_swizzled(st, p.swz);
                const uint64_t db = smem_desc_swizzled(st + NPLANE * a_bytes, p.swz);
                // the reduction's last block may end early: its K steps past the end would multiply the TMA unit's zero fill
                const int ks = kb == p.k_blocks - 1 ? last_ksteps : ksteps;
                if (!I16) {
                    const uint32_t first = kb != 0 ? 1u : 0u;
                    mma_i8(d0, da, db, idesc_ss, first);
                    if (ks > 1)
                        mma_i8(d0, da + 2, db + 2, idesc_ss, 1u);
                    if (ks > 2)
                        mma_i8(d0, da + 4, db + 4, idesc_ss, 1u);
                    if (ks > 3)
                        mma_i8(d0, da + 6, db + 6, idesc_ss, 1u);
                    commit(smem_u32(&empty_bar[stage]));
                } else {
                    const uint64_t da_lo = smem_desc_swizzled(st + a_bytes, p.swz); // the filter's low plane follows its high plane
                    for (int k = 0; k < ks; k++) {
                        const uint64_t koff = (uint64_t)(k * 2); // 32 bytes of K, in 16-byte units
                        if (kb | k) {
                            mma_i8(d0, da + koff, db + koff, idesc_su, 1u);                 // hi * (uh | ul)
                            mma_i8(d0 + p.block_n, da_lo + koff, db + koff, idesc_uu, 1u);  // lo * (uh | ul)
                        } else { // the first step starts each accumulator once
                            const uint64_t db_lo = smem_desc_swizzled(st + 2 * a_bytes + b_bytes, p.swz);
                            mma_i8(d0, da, db, idesc_su, 0u);
                            mma_i8(d0 + 2 * p.block_n, da_lo, db_lo, idesc_uu1, 0u);
                            mma_i8(d0 + p.block_n, da_lo, db, idesc_uu1, 1u);
                        }
                    }
                    commit(smem_u32(&empty_bar[stage]));
                }
                if (++stage == p.stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            if (!ok)
                break;
            commit(smem_u32(&tfull_bar[acc]));
            mbar_arrive(smem_u32(&tfull_bar[acc])); // publishes epi_row / epi_col[acc]
            if (++acc == p.acc_stages) {
                acc = 0;
                acc_phase ^= 1;
            }
        }
        if (!ok)
            report_timeout(g_tc_error);
        TC_REC(2, w_tempty);
        TC_REC(3, w_full);
        TC_REC(4, w_issue);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..17)
        const int ew = warp - 2;
        const int group = ew >> 2;               // 0..3
        const int own_acc = I16 ? 0 : group % sets; // accumulator buffer this group reads (in turn: with the one `sets` further; int16: all in turn)
        const int part = I16 ? group : group / sets; // which share of the tile's columns
        int turn = 0;
        const int lane_group = warp & 3;         // TMEM lanes this warp may read: 32*lane_group .. +31
        const int row_in_tile = lane_group * 32 + lane;

        // Per-channel constants {bias_half, shift}, once per kernel: of every output channel, or of the only tile's.  The first loads are on
        // their way meanwhile (when all warps did this before them, a lone tile of 128x256x1024 took 1.1 us longer).
        bool fast = false;
        const int et0 = (int)threadIdx.x - 64;
        if (!I16) {
            // Only the threads that read wait, us a call read ahead / this way / all sixteen warps: 4096x1024x1024 7.85 / 7.91 / 7.97, 28038x1184x76
            // 14.5 / 15.1.  One wait by the producer and a barrier behind it took 8.2 and 15.3, first loads ahead of the producer's 8.5 and 15.1.
            if (!p.early && (p.epi.lut || et0 < (p.one_tile ? p.block_n : n_pad)))
                grid_dep_wait();
            EpiConfig epi = p.epi;
            const int first = p.one_tile ? (int)blockIdx.x % p.n_tiles * p.block_n : 0;
            if (epi.bias)
                epi.bias = (const int32_t *)epi.bias + first;
            if (epi.per_channel)
                epi.ew += first;
            stage_fast_params(epi, fast_s + first, p.N - first, p.one_tile ? p.block_n : n_pad, et0, EPI_WARPS * 32, slow_flag);
            if (p.epi.lut)
                stage_lut(p.epi.lut, lut_s, et0, EPI_WARPS * 32);
            named_bar(1, EPI_WARPS * 32);
            fast = !*slow_flag && !p.epi.lut_stride && p.K <= 32768; // one table rides on the staged form and on the packed words of unstaged rows; per-channel tables take the general path
        }
        const uint32_t fp_base = epi_param_base(fast_s);
        uint32_t acc_phase = 0;
        bool ok = true;
        long long w_tfull = 0, w_work = 0, w_store = 0;
        (void)w_tfull, (void)w_work, (void)w_store;
        TC_LAP_INIT;
        const bool own_loop = RES && fast && p.in_turn;
        if (RES && own_loop) {
            const uint32_t stage = smem_u32(out_stage), tbl = smem_u32(lut_s);
            if (p.epi.lut)
                ok = epilogue_resident<EVEN, 1>(p, map_out, tmem_base, fp_base, stage, tfull_bar, tempty_bar, epi_row, epi_col, tbl, group, lane_group, lane);
            else if (p.res)
                ok = epilogue_resident<EVEN, 2>(p, map_out, tmem_base, fp_base, stage, tfull_bar, tempty_bar, epi_row, epi_col, tbl, group, lane_group, lane);
            else
                ok = epilogue_resident<EVEN, 0>(p, map_out, tmem_base, fp_base, stage, tfull_bar, tempty_bar, epi_row, epi_col, tbl, group, lane_group, lane);
        }
        while (ok && !own_loop) {
            const int acc = RES || I16 ? own_acc + turn : own_acc;
            TC_LAP(w_work);
            if (!mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase)) {
                ok = false;
                break;
            }
            TC_LAP(w_tfull);
            const int rows = epi_row[acc];
            if (rows < 0)
                break;
            const int nt = epi_col[acc];
            const int bi = p.batch == 1 ? 0 : rows / p.m_tiles;
            const int m0 = (p.batch == 1 ? rows : rows % p.m_tiles) * BLOCK_M;
            const int n0 = nt * p.block_n;
            fence_after();
            const bool row_ok = m0 + row_in_tile < p.M;
            const long long m = (long long)bi * p.M + m0 + row_in_tile; // row of the output tensor
            const uint32_t t0 = tmem_base + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)(acc * NACC * p.block_n);
            acc_phase ^= 1;
            if (I16 && p.acc_stages == 2) {
                acc_phase ^= 1 ^ turn;
                turn ^= 1;
            }
            if (RES && p.in_turn) { // (general epilogue: a channel outside the fast form)
                if (!turn)
                    acc_phase ^= 1;
                turn = sets - turn;
            }
            if (!I16) {
                if (fast && p.out_pw) {
                    // staged: every warp requantises its 32 rows into its part of the group's shared-memory tile and sends them off with a TMA store of
                    // its own.  (One store for the four warps took two barriers a tile, at which a group stood for a seventh of its time.)
                    const uint32_t buf = smem_u32(out_stage + (size_t)group * out_tile_bytes);
                    const int col0 = part * p.out_pw;
                    if (!p.out_rows && elect_one())
                        bulk_wait_read_all(); // the previous store out of these rows has read them
                    __syncwarp();
                    TC_LAP(w_store);
                    const int floor_q = p.epi.relu ? 0 : INT_MIN;
                    if (p.frag) {
                        const int cols = min(p.block_n / parts, p.N - (n0 + col0));
                        const uint32_t tc = t0 + col0, fpp = fp_base + (uint32_t)(n0 + col0) * 8u;
                        if (p.res)
                            epilogue_frag_residual<EVEN>(tc, fpp, buf, lane_group, lane, cols, p.out_pw, (uint32_t)p.out_mask, floor_q, p.res + (long long)m0 * p.rps + n0 + col0,
                                                         p.rps, p.M - m0);
                        else if (p.out_pw == 128 && cols == 128)
                            epilogue_frag<128, 128, EVEN>(tc, fpp, buf, lane_group, lane, floor_q, [] {});
                        else if (p.out_pw == 64 && cols == 64)
                            epilogue_frag<64, 64, EVEN>(tc, fpp, buf, lane_group, lane, floor_q, [] {});
                        else
                            epilogue_frag_each(tc, fpp, buf, lane_group, lane, cols, p.out_pw, (uint32_t)p.out_mask,
                                               [=](const int32_t *v, int i, const FragConst &k) { return frag_word<EVEN>(v, i, k, floor_q); });
                    } else if (p.epi.lut) {
                        epilogue_stage_lut<EVEN>(t0 + col0, fp_base + (uint32_t)(n0 + col0) * 8u, buf, row_in_tile, p.out_pw, (uint32_t)p.out_mask, floor_q, smem_u32(lut_s));
                    } else if (p.res)
                        epilogue_stage_residual<EVEN>(t0 + col0, fp_base + (uint32_t)(n0 + col0) * 8u, buf, row_in_tile, p.out_pw, (uint32_t)p.out_mask, floor_q,
                                                p.res + m * p.rps + n0 + col0, row_ok, p.N - (n0 + col0));
                    else if (p.out_pw == 128)
                        epilogue_stage<128, EVEN>(t0 + col0, fp_base + (uint32_t)(n0 + col0) * 8u, buf, row_in_tile, 128, floor_q);
                    else if (p.out_pw == 96)
                        epilogue_stage<96, EVEN>(t0 + col0, fp_base + (uint32_t)(n0 + col0) * 8u, buf, row_in_tile, 96, floor_q);
                    else if (p.out_pw == 64)
                        epilogue_stage<64, EVEN>(t0 + col0, fp_base + (uint32_t)(n0 + col0) * 8u, buf, row_in_tile, 64, floor_q);
                    else
                        epilogue_stage<0, EVEN>(t0 + col0, fp_base + (uint32_t)(n0 + col0) * 8u, buf, row_in_tile, p.out_pw, floor_q);
                    // the accumulator is free as soon as this warp's TMEM loads are done: hand it back before the
                    // shared-memory tile is completed and stored, so that the MMAs of the tile after next start earlier
                    fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(smem_u32(&tempty_bar[acc]));
                    if (p.out_rows) {
                        const int len = min(p.out_pw, p.N - (n0 + col0)), rows_left = min(32, p.M - m0 - lane_group * 32);
                        int8_t *dst = (int8_t *)p.out + ((long long)bi * p.M + m0 + lane_group * 32) * p.ops + n0 + col0;
                        if (len > 0)
                            store_staged_rows(dst, p.ops, buf, (uint32_t)(lane_group * 32 * p.out_pw), (uint32_t)p.out_pw, rows_left, len, (uint32_t)p.out_mask, lane);
                        continue;
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (m0 + lane_group * 32 < p.M && n0 + col0 < p.N && elect_one()) { // rows >= M and columns >= N are clipped
                        tma_store_3d(&map_out, buf + (uint32_t)(lane_group * 32 * p.out_pw), n0 + col0, m0 + lane_group * 32, bi);
                        bulk_commit();
                    }
                    __syncwarp();
                    continue;
                }
                if (p.frag)
                    epilogue_frag_general(p, t0, m, n0, row_ok, parts, part);
                else if (RES)
                    epilogue_direct_tile<EVEN>(p, fast_s, fp_base, t0, m, n0, row_ok, fast, parts, part, p.epi.lut ? smem_u32(lut_s) : 0u);
                else
                    epilogue_direct<EVEN, true>(p, fast_s, fp_base, t0, m, n0, row_ok, fast, parts, part, p.epi.lut ? smem_u32(lut_s) : 0u);
            } else {
                // all groups share the tile: constants of its columns, then 16 columns at a time into a staging tile of [128][2 * block_n]
                // bytes, then whole rows
                constexpr int EPI_BAR = 6;
                const int et = (int)threadIdx.x - 64;
                const int sum = row_ok ? p.row_sum[m] : 0; // times -32768 is added to the row's results
                if (!p.out_rows && et == 0)
                    bulk_wait_read_all();
                named_bar(EPI_BAR, EPI_WARPS * 32); // the previous tile's rows and constants have been read
                if (et == 0)
                    *slow_flag = 0;
                named_bar(EPI_BAR, EPI_WARPS * 32);
                for (int j = et; j < p.block_n; j += EPI_WARPS * 32) {
                    const int n = min(n0 + j, p.N - 1);
                    const int e = p.epi.per_channel ? __ldg(p.epi.ew + n) : p.epi.ew_scalar, sh = p.epi.e_shift_base - e;
                    const long long b = p.epi.bias ? __ldg((const long long *)p.epi.bias + n) : 0ll;
                    if (!halves_fit(b, sh))
                        *slow_flag = 1;
                    wide_s[j] = halves_param<EVEN>(b, sh);
                }
                named_bar(EPI_BAR, EPI_WARPS * 32);
                const bool slow = *(volatile int *)slow_flag;
                const long long base = -(long long)sum * 32768;
                const int row_h = (int)(base >> 16), row_l = (int)(base & 0xffff);
                // staged rows: pieces of 64 columns for a TMA store each, or whole rows for one (without its swizzle) or for the warps
                const bool pieces = !p.out_rows && p.block_n % 64 == 0;
                const uint32_t buf = smem_u32(out_stage), pitch = pieces ? 128u : 2u * (uint32_t)p.block_n, mask = p.out_rows || pieces ? 7u : 0u;
                int chunk = 0;
                for (int c0 = 0; c0 < p.block_n; c0 += 16, chunk++) {
                    if (chunk % parts != part)
                        continue;
                    int32_t vh[16], vm[16], vl[16];
                    ld16(t0 + c0, vh);
                    ld16(t0 + p.block_n + c0, vm);
                    ld16(t0 + 2 * p.block_n + c0, vl);
                    ld_wait16(vh);
                    tie16(vm);
                    tie16(vl);
                    uint32_t pk[8];
                    if (!slow) {
#pragma unroll
                        for (int j = 0; j < 16; j += 2) {
                            const int q0 = requant_wide<EVEN>(vh[j], vm[j], vl[j], row_h, row_l, wide_s[c0 + j]);
                            const int q1 = requant_wide<EVEN>(vh[j + 1], vm[j + 1], vl[j + 1], row_h, row_l, wide_s[c0 + j + 1]);
                            asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(pk[j >> 1]) : "r"(q1), "r"(q0));
                            if (p.epi.relu)
                                asm("max.s16x2 %0, %0, %1;" : "+r"(pk[j >> 1]) : "r"(0));
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            const long long w = base + (long long)vh[j] * 65536 + (long long)vm[j] * 256 + (long long)vl[j];
                            const int n = min(n0 + c0 + j, p.N - 1);
                            const int e = p.epi.per_channel ? __ldg(p.epi.ew + n) : p.epi.ew_scalar;
                            const int shift = max(-62, min(62, p.epi.e_shift_base - e));
                            const int q = requant16(w, p.epi.bias ? __ldg((const long long *)p.epi.bias + n) : 0ll, shift, p.epi.relu, p.epi.half_even);
                            pk[j >> 1] = j & 1 ? pk[j >> 1] | ((uint32_t)q << 16) : (uint32_t)q & 0xffffu;
                        }
                    }
                    const uint32_t off = (!pieces ? 2u * (uint32_t)c0 : (uint32_t)(c0 >> 6) * (BLOCK_M * 128u) + 2u * (uint32_t)(c0 & 63)) + (uint32_t)row_in_tile * pitch;
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + (off ^ (((off >> 7) & mask) << 4))), "r"(pk[0]), "r"(pk[1]), "r"(pk[2]), "r"(pk[3]) : "memory");
                    const uint32_t off2 = off + 16u;
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + (off2 ^ (((off2 >> 7) & mask) << 4))), "r"(pk[4]), "r"(pk[5]), "r"(pk[6]), "r"(pk[7]) : "memory");
                }
                fence_before(); // the accumulator is free before the rows leave
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(smem_u32(&tempty_bar[acc]));
                if (!p.out_rows)
                    fence_async_smem();
                named_bar(EPI_BAR, EPI_WARPS * 32);
                if (!p.out_rows) {
                    if (et == 0) { // rows >= M and columns >= N are clipped
                        for (int c0 = 0; c0 < p.block_n; c0 += pieces ? 64 : p.block_n) tma_store_3d(&map_out, buf + (uint32_t)(c0 >> 6) * (BLOCK_M * 128u), 2 * (n0 + c0), m0, bi);
                        bulk_commit();
                    }
                    continue;
                }
                const int len = 2 * min(p.block_n, p.N - n0);
                const int row0 = ew * (BLOCK_M / EPI_WARPS);
                store_staged_rows((int8_t *)p.out + 2 * (((long long)bi * p.M + m0 + row0) * p.ops + n0), 2 * p.ops, buf, (uint32_t)row0 * pitch, pitch,
                                  min(BLOCK_M / EPI_WARPS, p.M - m0 - row0), len, mask, lane);
                continue;
            }
            fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&tempty_bar[acc]));
        }
        if (!ok && lane == 0)
            report_timeout(g_tc_error);
        if (ew == 0 && lane == 0 && !own_loop) {
            TC_LAP(w_work);
            TC_REC(5, w_tfull);
            TC_REC(6, w_work);
            TC_REC(7, w_store);
        }
        if (I16 ? !p.out_rows && et0 == 0 : p.out_pw && !p.out_rows && elect_one())
            bulk_wait_all(); // shared memory stays allocated until the last store has left it
        __syncwarp();
    }

    fence_before();
    __syncthreads();
    TC_STAMP(1);
    if (warp == 1) {
        fence_after();
        tmem_dealloc(tmem_base, p.tmem_cols);
    }
    // the last CTA to get here leaves the counters as it found them (thread 0 is also the one that asked for tiles)
    if (p.sched && threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(p.sched + 1, 1u) == gridDim.x - 1) {
            p.sched[0] = 0;
            p.sched[1] = 0;
        }
    }
}

// ------------------------------------------------------------------------------------------ CTA pairs (large int8 Gemm)
// For a reduction long enough to be bound by the tensor pipe, the tile above needs (128 + 256) * 128 bytes per 4 MMA
// steps and SM; the bytes a shared memory can keep in flight then cover less than the load latency and the tensor
// pipe idles about half of the time (measured: 45 % active at 65536x1024x1024).  Here two CTAs of a cluster (the two
// SMs of a TPC) work on one 256 x block_n tile with tcgen05.mma.cta_group::2: each loads its own 128 rows of A and only
// HALF of the B tile (the tensor cores read the other half from the peer's shared memory), i.e. a third fewer bytes
// per MMA and SM, so the same shared memory holds half as many more stages.  The even CTA of the pair issues the MMAs
// for both; barriers: every TMA load of either CTA completes bytes on the even CTA's "full" barrier, the MMA
// issuer's commits arrive on both CTAs' "empty" and "accumulator full" barriers (one commit per CTA, addressed with
// mapa), both CTAs' epilogue warps arrive on the even CTA's "accumulator empty" barrier.  Epilogue: direct row stores.
__device__ __forceinline__ uint32_t cluster_ctarank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same shared-memory variable in the CTA with rank `rank`
__device__ __forceinline__ uint32_t mapa_rank(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, uint32_t leader_bar)
{
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
                 "l"(map), "r"(leader_bar), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void mma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(z)
        : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t cluster_bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t slot_smem, uint32_t cols)
{
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t base, uint32_t cols)
{
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b_half, const TcParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int a_bytes = BLOCK_M * p.swz;
    const int bh_bytes = (p.block_n / 2) * p.swz;
    const int stage_bytes = a_bytes + bh_bytes;
    const int n_pad = p.n_tiles * p.block_n;
    uint8_t *aux = smem + (size_t)p.stages * stage_bytes;
    FastParam *fast_s = (FastParam *)aux;
    uint64_t *bars = (uint64_t *)(aux + sizeof(FastParam) * (size_t)n_pad);
    uint64_t *full_bar = bars, *empty_bar = bars + MAX_STAGES, *tfull_bar = bars + 2 * MAX_STAGES, *tempty_bar = tfull_bar + MAX_ACC;
    uint32_t *tmem_slot = (uint32_t *)(tempty_bar + MAX_ACC);
    int *slow_flag = (int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair_m_tiles = (p.m_tiles + 1) / 2;
    const int total_pairs = pair_m_tiles * p.n_tiles;
    const int pair_id = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int parts = 4 / p.acc_stages;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int a = 0; a < MAX_ACC; a++) {
            mbar_init(smem_u32(&tfull_bar[a]), 1);
            mbar_init(smem_u32(&tempty_bar[a]), 2 * 4 * parts); // the epilogue warps of both CTAs
        }
        *slow_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1)
        tmem_alloc_pair(smem_u32(tmem_slot), p.tmem_cols); // the same warp of both CTAs, the same slot address
    fence_before();
    __syncthreads();
    cluster_sync_all(); // both CTAs' barriers exist before either touches the other's
    fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (both CTAs)
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int t = pair_id; t < total_pairs && ok; t += n_pairs) {
                const int m0 = (t / p.n_tiles) * 2 * BLOCK_M + (int)rank * BLOCK_M;
                const int n0 = (t % p.n_tiles) * p.block_n + (int)rank * (p.block_n / 2);
                for (int kb = 0; kb < p.k_blocks; kb++) {
                    if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1)) {
                        ok = false;
                        break;
                    }
                    if (rank == 0)
                        mbar_arrive_expect_tx(smem_u32(&full_bar[stage]), (uint32_t)(2 * stage_bytes)); // the bytes of both CTAs
                    const uint32_t bar = mapa_rank(smem_u32(&full_bar[stage]), 0);
                    uint8_t *st = smem + (size_t)stage * stage_bytes;
                    tma_load_3d_pair(smem_u32(st), &map_a, kb * p.swz, m0, 0, bar);
                    tma_load_3d_pair(smem_u32(st + a_bytes), &map_b_half, kb * p.swz, n0, 0, bar);
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok)
                report_timeout(g_tc_error);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (even CTA only)
        if (rank == 0 && elect_one()) {
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            const uint32_t idesc = idesc_i8(1, 1, 2 * BLOCK_M, p.block_n);
            const int ksteps = p.swz / 32;
            for (int t = pair_id; t < total_pairs && ok; t += n_pairs) {
                if (!mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1)) {
                    ok = false;
                    break;
                }
                fence_after();
                const uint32_t d0 = tmem_base + (uint32_t)(acc * p.block_n);
                for (int kb = 0; kb < p.k_blocks; kb++) {
                    if (!mbar_wait(smem_u32(&full_bar[stage]), phase)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint32_t st = smem_u32(smem + (size_t)stage * stage_bytes);
                    const uint64_t da = smem_desc_swizzled(st, p.swz);
                    const uint64_t db = smem_desc_swizzled(st + a_bytes, p.swz);
                    for (int k = 0; k < ksteps; k++) mma_i8_pair(d0, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) != 0);
                    commit_pair(mapa_rank(smem_u32(&empty_bar[stage]), 0));
                    commit_pair(mapa_rank(smem_u32(&empty_bar[stage]), 1));
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok)
                    break;
                commit_pair(mapa_rank(smem_u32(&tfull_bar[acc]), 0));
                commit_pair(mapa_rank(smem_u32(&tfull_bar[acc]), 1));
                if (++acc == p.acc_stages) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            }
            if (!ok)
                report_timeout(g_tc_error);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..17 of both CTAs)
        const int ew = warp - 2;
        const int group = ew >> 2;
        const int acc = group % p.acc_stages;
        const int part = group / p.acc_stages;
        const int lane_group = warp & 3;
        const int row_in_tile = lane_group * 32 + lane;
        const int et = threadIdx.x - 64;
        stage_fast_params(p.epi, fast_s, p.N, n_pad, et, EPI_WARPS * 32, slow_flag);
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
        const bool fast = !*slow_flag && !p.epi.half_even && !p.epi.lut && p.K <= 32768;
        const uint32_t fp_base = epi_param_base(fast_s);
        const uint32_t tempty_leader = mapa_rank(smem_u32(&tempty_bar[acc]), 0);
        uint32_t acc_phase = 0;
        bool ok = true;
        int local = 0;
        for (int t = pair_id; t < total_pairs && ok; t += n_pairs, local++) {
            if (local % p.acc_stages != acc)
                continue;
            const int m0 = (t / p.n_tiles) * 2 * BLOCK_M + (int)rank * BLOCK_M;
            const int n0 = (t % p.n_tiles) * p.block_n;
            if (!mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase)) {
                ok = false;
                break;
            }
            acc_phase ^= 1;
            fence_after();
            const bool row_ok = m0 + row_in_tile < p.M;
            const long long m = (long long)m0 + row_in_tile;
            const uint32_t t0 = tmem_base + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)(acc * p.block_n);
            // 128-bit stores: in this kernel the 256-bit form stored only the first word of each 32 bytes
            epilogue_direct_tile<false>(p, fast_s, fp_base, t0, m, n0, row_ok, fast, parts, part, 0u);
            fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive_cluster(tempty_leader);
        }
        if (!ok && lane == 0)
            report_timeout(g_tc_error);
    }

    fence_before();
    __syncthreads();
    cluster_sync_all(); // neither CTA leaves (or frees TMEM) while the other may still read its shared memory or barriers
    if (warp == 1) {
        fence_after();
        tmem_dealloc_pair(tmem_base, p.tmem_cols);
    }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

// uint8 tensor [mats][rows][cols] with `row_stride` bytes between rows and `mat_stride` bytes between matrices;
// box = 1 x box_rows x box_cols.
int make_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols, uint64_t row_stride, uint32_t box_rows,
             uint32_t box_cols, int swz, uint64_t mats = 1, uint64_t mat_stride = 0)
{
    EncodeTiledFn enc = get_encode();
    if (!enc)
        return set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled entry point not found");
    if (mats <= 1)
        mat_stride = (rows * row_stride + 15) / 16 * 16; // unused with a single matrix, but it must be a legal stride
    cuuint64_t dims[3] = {cols, rows, mats ? mats : 1};
    cuuint64_t strides[2] = {row_stride, mat_stride};
    cuuint32_t box[3] = {box_cols, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapSwizzle sw = swz == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
        : (swz == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : (swz == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE));
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
        return ESPDL_ERR_CUDA;
    }
    return ESPDL_OK;
}

// The filter's rows in the order of the fragments (frag_channel): [N / 16][2][4][2] rows of K bytes, a box of box_rows of them.
int make_frag_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols, uint32_t box_rows, int swz)
{
    EncodeTiledFn enc = get_encode();
    if (!enc)
        return set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled entry point not found");
    cuuint64_t dims[5] = {cols, 2, 4, 2, rows / 16};
    cuuint64_t strides[4] = {cols, 4 * cols, 2 * cols, 16 * cols};
    cuuint32_t box[5] = {(cuuint32_t)swz, 2, 4, 2, box_rows / 16};
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUtensorMapSwizzle sw = swz == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (swz == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    if (enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
        return ESPDL_ERR_CUDA;
    }
    return ESPDL_OK;
}

// Bytes of K per stage row (= TMA box width = swizzle width).  Wide rows move fastest through the TMA unit, so
// 128 is used as soon as K fills three quarters of such a row; columns past K are zero-filled, not fetched.
int pick_swz(int K)
{
    if (K >= 96)
        return 128;
    if (K > 32)
        return 64;
    return 32;
}

constexpr size_t SMEM_BUDGET = 200 * 1024;      // stages + staging tiles of the layers whose epilogue is staged
constexpr size_t SMEM_BUDGET_DEEP = 225 * 1024; // long reductions with direct row stores: one more stage in flight (1.79 -> 1.97 POPS
                                                // at 65536x1024x1024); for the staged layers the larger budget measured 5 % slower

size_t aux_bytes(const TcParams &p, bool i16 = false)
{
    return (i16 ? sizeof(HalvesParam) * (size_t)p.block_n : sizeof(FastParam) * (size_t)p.n_tiles * p.block_n) + (2 * MAX_STAGES + 2 * MAX_ACC + 2) * 8 + 32 + 256 + 2 * (TILE_RING + MAX_ACC) * 4;
}

// A filter that stays in shared memory.  With tiles that bring their part of the filter along, a tile of a short reduction loads more of the filter than
// of the rows, two or three stages hold it all, and the next tile's loads come too late (401408 rows of 128 -> 768: the MMA issuer
// waited for loads half of the time).  Here a CTA loads as many column tiles as fit beside a ring of row tiles once - groups of CTAs share the column
// tiles out where they do not all fit - and every row tile serves all of them.  Tiles are 128 columns wide: two accumulators for each of two sets of
// epilogue warps, so that a warp finds the next tile's sums ready (64 columns and fewer: for each of four).  us before / after (floor: bytes): 401408 x 128 ->
// 768 93 / 73 (55), 802816 x 96 -> 96 56 / 28 (24), 200704 x 64 -> 384 27.4 / 23.5 (14), 50176 x 320 -> 1280 46 / 30 (12), 65536 x 384 -> 384 24 / 15 (8).
// From two row tiles a CTA on: below, the filter is not used often enough (8192 x 256 -> 1024: 7.1 us, 8.5 resident).  Results that overwrite the inputs
// stay with one column tile (up to 256 columns without a resident filter), which has all of a row before any of it is written: here a row tile's columns may be two CTAs'.
void plan_resident(const espdl_conv_desc &d, TcParams &p)
{
    p.resident = p.in_turn = 0, p.n_groups = 1;
    if (p.one_tile || !p.out_pw || p.batch != 1)
        return;
    TcParams q = p;
    if (q.N % 16 == 0 && !q.out_rows) {
        q.block_n = min(128, q.N), q.n_tiles = (q.N + q.block_n - 1) / q.block_n;
        q.in_turn = 1, q.acc_stages = q.block_n > 64 ? 4 : 8;
        for (q.tmem_cols = 32; q.tmem_cols < q.acc_stages * q.block_n;) q.tmem_cols *= 2; // (what they leave serves kernels of parallel branches)
        q.out_pw = 64, q.out_mask = 3;
    }
    if (q.n_tiles > p.n_tiles && p.n_tiles == 1 && overlaps(d))
        return;
    const size_t a_stage = (size_t)BLOCK_M * q.swz, b_tile = (size_t)q.block_n * q.k_blocks * q.swz;
    const size_t room = SMEM_BUDGET_DEEP - aux_bytes(q) - 4 * ((size_t)((BLOCK_M * q.out_pw + 1023) & ~1023) << q.in_turn) - 2048;
    // one column tile: a row tile's stages are free as soon as they are multiplied; several: two row tiles
    const size_t ring = a_stage * (q.n_tiles == 1 ? 4 : max(2 * q.k_blocks, 3));
    if (room < ring + b_tile)
        return;
    const int fit = (int)min((long long)q.n_tiles, (long long)((room - ring) / b_tile));
    q.n_groups = (q.n_tiles + fit - 1) / fit;
    q.resident = (q.n_tiles + q.n_groups - 1) / q.n_groups;
    q.n_groups = (q.n_tiles + q.resident - 1) / q.resident;
    if (q.n_groups > num_sms() / 8 || (long long)q.m_tiles * q.n_groups < 2ll * num_sms())
        return;
    // more memory than the other plans take only for what has to fit: what it leaves of an SM's serves kernels of parallel branches
    q.stages = (int)min((size_t)MAX_STAGES, max(ring, room - q.resident * b_tile - min(room - q.resident * b_tile, SMEM_BUDGET_DEEP - SMEM_BUDGET)) / a_stage);
    // A row tile costs a group its columns' results (4.5 ns each; the two sets of epilogue warps take the tiles in turn, so that with an even number of them one set has
    // the wide ones), and no less than the way of its 128 x K bytes into shared memory (26 bytes a cycle when all SMs load) or the latency of that, shared by the row
    // tiles that the ring holds (1.6 us).  By columns alone a last group of 16 had two of 148 CTAs for as many rows as the others.
    const int across = q.n_tiles - (q.n_groups - 1) * q.resident, load = max(5 * q.K / 8, 360 * q.k_blocks / q.stages);
    q.share = max(q.resident * q.block_n, load);
    q.shares = (q.n_groups - 1) * q.share + max(across % 2 ? q.N - (q.n_tiles - across) * q.block_n : across * q.block_n, load);
    // Several groups load the rows several times: not where that outweighs the columns (65536 x 384 -> 144 8.6 us, 10.8 resident), where rows leave by warps (31646 x 160 -> 2648
    // 62 / 115), and where parts of a 32-byte sector are written by different groups and rows and results are more than L2 holds, unless
    // the rows' own sectors are cut as well and tiles of 256 columns read them oftener (90000 x 64 -> 3088 81 / 105, 60000 x 192 -> 2032 45 / 50; 84843 x 144 -> 1616 72 / 59).
    const long long ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c, ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    const bool cut = ops % 32 && q.M * (ops + ips) > 126000000ll && (q.k_blocks == 1 || q.K % 32 == 0);
    if (q.n_groups > 1 && (!q.in_turn || 5 * q.shares > 12 * q.N || cut))
        return;
    if (q.resident > 1 && q.stages < 2 * q.k_blocks) // (more stages than there are barriers)
        return;
    p = q;
}

// int16 products in tiles of bn columns: rounds of tiles over the SMs; a tile's instructions (two of twice the width every 32 bytes of K), its loads of two planes at
// 64 bytes a cycle, and its results at 35 cycles a column and 2400 a tile (rows that leave by warps: a column of whole groups of 64), beside the next tile's products
// where there are two sets of accumulators.
double int16_tile_cycles(const TcParams &p, int bn, bool by_warps)
{
    const double rounds = ceil((double)p.m_tiles * ((p.N + bn - 1) / bn) / num_sms()), results = 2400 + 35.0 * (by_warps ? (bn + 63) / 64 * 64 : bn);
    const double products = max((p.K + 31) / 32 * 2.0 * max(bn, 32 + bn / 2), 2.0 * (BLOCK_M + bn) * p.K / 64);
    return 6 * bn <= 512 ? rounds * max(products, results) + results : rounds * (products + results);
}

bool plan(const espdl_conv_desc &d, TcParams &p, bool force_direct = false)
{
    const bool i16 = d.dtype == ESPDL_DTYPE_INT16;
    // one matrix over all pixels of all images, or - when every image has its own filter - one matrix per image
    const bool batched = d.filter_image_stride != 0;
    if (batched && (i16 || d.filter_image_stride % 16 != 0))
        return false;
    const long long M = (batched ? 1ll : (long long)d.n) * d.out_h * d.out_w;
    if (M > 0x7fffffffll || d.out_c > 8192)
        return false;
    p.M = (int)M, p.N = d.out_c, p.K = d.in_c;
    p.batch = batched ? d.n : 1;
    int max_bn = i16 ? 128 : 256;
    if (const char *cap = getenv("ESPDL_B200_MAX_BLOCK_N")) // tile width cap (a multiple of 16), for experiments
        max_bn = max(16, min(max_bn, atoi(cap) / 16 * 16));
    p.m_tiles = (p.M + BLOCK_M - 1) / BLOCK_M;
    // Few rows: narrower tiles put more SMs to work while they still make one wave - a tile's time is the stream of its filter rows
    // through one SM plus its columns' epilogue.
    while (max_bn > 32 && 2ll * p.batch * p.m_tiles * ((p.N + max_bn - 1) / max_bn) <= num_sms()) max_bn /= 2;
    const auto width = [&](int cap) {
        const int tiles = (p.N + cap - 1) / cap;
        return (((p.N + tiles - 1) / tiles) + 15) / 16 * 16;
    };
    const long long ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    const bool rows16 = ops % 8 != 0 || p.N % 8 != 0 || ((uintptr_t)d.output % 16) != 0; // int16 rows that leave by warps (see below)
    if (i16 && max_bn > 64) {
        // Tiles of up to 80 columns leave room for a second set of accumulators, so that a tile is multiplied while the one before it is requantised; wider ones
        // load less for a result.  Cycles by what either takes (int16_tile_cycles), within 0.8 % of the best of the three over 190 products; without a tile's
        // own cost the choice lost up to 13 % of the widest.  us at most 128 / 80 / 64 columns: 4096x1024x1024 24.7 / 23.1 / 25.9, 2887x1072x3768 72 / 62 / 68,
        // 65536x512x128 57.2 / - / 52.9, 4096x2048x512 22.7 / 26.1 / 24.9, 65536x96x2048 215 / 240 / 245; by warps 65536x256x1006 164 / 214 / 198.
        const double wide = int16_tile_cycles(p, width(max_bn), rows16), mid = int16_tile_cycles(p, width(80), rows16), narrow = int16_tile_cycles(p, width(64), rows16);
        if (min(mid, narrow) < 0.95 * wide)
            max_bn = mid < narrow ? 80 : 64;
    }
    p.n_tiles = (p.N + max_bn - 1) / max_bn;
    p.block_n = width(max_bn);
    if (!i16 && p.block_n > 128)
        p.block_n = (p.block_n + 31) / 32 * 32; // two epilogue groups split a wide tile into whole 16-byte pieces
    p.n_tiles = (p.N + p.block_n - 1) / p.block_n;
    p.swz = pick_swz(p.K);
    if (i16 && p.swz == 128 && p.block_n > 80)
        p.swz = 64; // a stage holds two planes of each operand: 64-byte rows leave room for five stages beside a wide output tile
    p.k_blocks = (p.K + p.swz - 1) / p.swz;
    p.acc_stages = i16 ? (6 * p.block_n <= 512 ? 2 : 1) : (4 * p.block_n <= 512 ? 4 : 2);
    const long long rps = d.residual_pixel_stride ? d.residual_pixel_stride : d.out_c;
    const bool res_ok = !d.residual || (rps % 16 == 0 && ((uintptr_t)d.residual % 16) == 0);
    const bool stageable = res_ok && !force_direct && !getenv("ESPDL_B200_DIRECT_STORES");
    // A CTA with one tile has nothing to overlap its epilogue with: four groups instead of two take it, and staging costs no memory (4096x1024x1024:
    // 10.1 -> 8.0 us; direct row stores took 3.8 us of it).
    p.one_tile = !i16 && stageable && p.block_n % 64 == 0 && (long long)p.batch * p.m_tiles * p.n_tiles <= num_sms();
    if (p.one_tile)
        p.acc_stages = 1;
    int cols = p.acc_stages * (i16 ? 3 : 1) * p.block_n;
    int pow2 = 32;
    while (pow2 < cols) pow2 *= 2;
    if (pow2 > 512)
        return false;
    p.tmem_cols = pow2;
    // staged epilogue (int8): each group of four epilogue warps owns a piece of block_n / parts columns
    p.out_pw = 0, p.out_mask = 0;
    p.out_rows = 0;
    if (i16) {
        p.out_pw = p.block_n / 2; // four times [128][out_pw] = the tile
        p.out_rows = rows16;
    } else if (stageable) {
        // A TMA store clips rows in units of 16 bytes: behind a row that ends in the middle of one it would write the neighbour's columns.
        p.out_rows = ops % 16 != 0 || p.N % 16 != 0 || ((uintptr_t)d.output % 16) != 0;
        const int parts = 4 / p.acc_stages;
        // Rows that no TMA store can address: staged, a tile of any width takes its warps as long as a thread of theirs some stores of its own row (131072 rows of 64,
        // us from registers / staged: 13 stores of four bytes 12.4 / 14.8, 15 14.4 / 14.9, 17 16.8 / 15.4, 25 21.8 / 16.1; of two 9 11.3 / 15.2, 11 15.5 / 15.2,
        // 13 21.8 / 15.2; of one 13 9.4 / 14.9, 21 14.7 / 15.2).
        const uintptr_t mixed = (uintptr_t)ops | (uintptr_t)d.output | (p.n_tiles > 1 ? (uintptr_t)p.block_n : 16u) | 16u;
        const int bytes = (int)(mixed & (~mixed + 1)), stores = min(p.N, p.block_n) / bytes;
        const bool few_stores = p.out_rows && stores < (bytes >= 4 ? 16 : bytes == 2 ? 11 : 21);
        if (few_stores)
            p.out_rows = 0;
        else if (p.block_n % (16 * parts) == 0 && p.block_n / parts <= 128) {
            p.out_pw = p.block_n / parts;
            p.out_mask = p.out_pw == 128 ? 7 : (p.out_pw == 64 ? 3 : 0);
        }
    }
    size_t out_bytes = p.one_tile ? 0 : 4 * (size_t)((BLOCK_M * p.out_pw + 1023) & ~1023);
    size_t stage_bytes = (size_t)(i16 ? 2 : 1) * (BLOCK_M + p.block_n) * p.swz;
    int stages = (int)((SMEM_BUDGET - aux_bytes(p, i16) - out_bytes - 1024) / stage_bytes);
    // A wide tile with a reduction of two 128-byte blocks and room for only two or three stages has barely one tile's loads
    // in flight, and every tile then waits a full load latency (192 -> 256 columns over 3.3 M rows: 0.39 ms).  Blocks of 64
    // bytes make stages half as large: more of them, more tiles in flight (0.28 ms), although the TMA unit moves 64-byte
    // rows more slowly - so only where the 128-byte form is starved.
    if (!i16 && p.swz == 128 && p.k_blocks == 2 && stages < 3 * p.k_blocks / 2 + 1 && !getenv("ESPDL_B200_NO_NARROW_K")) {
        const size_t stage64 = (size_t)(BLOCK_M + p.block_n) * 64;
        const int kb64 = (p.K + 63) / 64;
        const int stages64 = (int)std::min<size_t>((SMEM_BUDGET - aux_bytes(p) - out_bytes - 1024) / stage64, MAX_STAGES);
        if (stages64 * p.k_blocks > stages * kb64) { // more tiles in flight
            p.swz = 64, p.k_blocks = kb64, stage_bytes = stage64, stages = stages64;
        }
    }
    if (!i16 && p.out_rows && p.out_pw && stages < 4)
        stages = (int)((SMEM_BUDGET_DEEP - aux_bytes(p) - out_bytes - 1024) / stage_bytes);
    p.resident = p.in_turn = 0;
    if (!i16)
        plan_resident(d, p);
    if (p.resident) { // (rows that leave by warps have no fragment form with a table)
        p.frag = p.N % 16 == 0 && (p.in_turn || !d.lut);
        return true;
    }
    if (!i16 && !p.one_tile && p.out_pw && !p.out_rows && p.k_blocks > 2 && stages < 4) {
        // a long reduction needs the deep load pipeline more than the output needs staging
        p.out_pw = 0, p.out_mask = 0, out_bytes = 0;
        stages = (int)((SMEM_BUDGET_DEEP - aux_bytes(p) - 1024) / stage_bytes);
    }
    if (stages < 2)
        return false;
    p.stages = stages > MAX_STAGES ? MAX_STAGES : stages;
    // (a fused table's lookups outweigh the constants: a network of such layers at 16 images 817 us by rows, 822 on fragments)
    p.frag = !i16 && p.out_pw && !batched && p.N % 16 == 0 && !d.lut;
    return true;
}

// The CTA-pair kernel takes large int8 products without a per-image filter: long reductions, wide outputs, enough tiles.
bool pair_plan(const espdl_conv_desc &d, TcParams &p)
{
    // Off unless ESPDL_B200_CTA_PAIRS=1: measured slower than the one-CTA kernel so far (65536x1024x1024: 79 us against 70 us).
    const char *on = getenv("ESPDL_B200_CTA_PAIRS");
    if (d.dtype != ESPDL_DTYPE_INT8 || d.filter_image_stride != 0 || !on || atoi(on) == 0)
        return false;
    const long long M = (long long)d.n * d.out_h * d.out_w;
    if (M > 0x7fffffffll || d.out_c > 8192 || d.out_c < 256 || d.in_c < 512 || M < 2048)
        return false;
    p.M = (int)M, p.N = d.out_c, p.K = d.in_c, p.batch = 1;
    p.n_tiles = (p.N + 255) / 256;
    p.block_n = ((p.N + p.n_tiles - 1) / p.n_tiles + 31) / 32 * 32;
    p.n_tiles = (p.N + p.block_n - 1) / p.block_n;
    p.m_tiles = (p.M + BLOCK_M - 1) / BLOCK_M;
    p.swz = 128;
    p.k_blocks = (p.K + p.swz - 1) / p.swz;
    p.acc_stages = 2 * p.block_n <= 512 ? 2 : 1;
    if (p.acc_stages < 2)
        return false;
    p.tmem_cols = 512;
    p.out_pw = 0, p.out_mask = 0, p.frag = 0, p.resident = p.in_turn = 0;
    const size_t stage_bytes = (size_t)(BLOCK_M + p.block_n / 2) * p.swz;
    const int stages = (int)((SMEM_BUDGET_DEEP - aux_bytes(p) - 1024) / stage_bytes);
    if (stages < 3)
        return false;
    p.stages = stages > MAX_STAGES ? MAX_STAGES : stages;
    return true;
}

int launch_pair(const espdl_conv_desc &d, TcParams &p, cudaStream_t s)
{
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    CUtensorMap ma, mb;
    int st;
    if ((st = make_map(&ma, d.input, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)ips, BLOCK_M, (uint32_t)p.swz, p.swz, 1, (uint64_t)p.M * ips)))
        return st;
    if ((st = make_map(&mb, d.filter, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)p.K, (uint32_t)(p.block_n / 2), (uint32_t)p.swz, p.swz, 1, 0)))
        return st;
    const size_t stage_bytes = (size_t)(BLOCK_M + p.block_n / 2) * p.swz;
    const size_t smem = 1024 + (size_t)p.stages * stage_bytes + aux_bytes(p);
    static std::once_flag attr_once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(attr_once, [] { attr_err = cudaFuncSetAttribute(gemm_tc_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(SMEM_BUDGET_DEEP + 2048)); });
    if (attr_err != cudaSuccess)
        return set_cuda_error(attr_err, "cudaFuncSetAttribute(gemm_tc_pair_kernel)");
    const long long pairs = (long long)((p.m_tiles + 1) / 2) * p.n_tiles;
    const int grid = 2 * (int)min(pairs, (long long)(num_sms() / 2));
    gemm_tc_pair_kernel<<<grid, NUM_THREADS, smem, s>>>(ma, mb, p); // cluster size 2 is a compile-time attribute of the kernel
    count_launch();
    return check_launch("gemm_tc_pair");
}

} // namespace

bool conv2d_tc_supported(const espdl_conv_desc &d)
{
    if (d.group != 1 || d.kh != 1 || d.kw != 1 || d.stride_h != 1 || d.stride_w != 1)
        return false;
    if (d.pad_top || d.pad_bottom || d.pad_left || d.pad_right)
        return false;
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    if (d.dtype == ESPDL_DTYPE_INT8) {
        if (d.in_c % 16 || ips % 16 || ((uintptr_t)d.input % 16) || ((uintptr_t)d.filter % 16))
            return false;
    } else {
        if (d.in_c % 16 || d.in_c > 16384) // planes are dense [rows][K] bytes: K % 16 keeps TMA strides legal
            return false;
    }
    TcParams p;
    return plan(d, p);
}

size_t conv2d_tc_workspace_bytes(const espdl_conv_desc &d)
{
    if (d.dtype != ESPDL_DTYPE_INT16)
        return 0;
    const size_t M = (size_t)d.n * d.out_h * d.out_w;
    const size_t a = (M * d.in_c + 255) / 256 * 256, b = ((size_t)d.out_c * d.in_c + 255) / 256 * 256;
    return 2 * a + 2 * b + M * sizeof(int);
}

namespace {

// Operands already packed: the tile kernel over rows of `o.Kp` bytes.
int launch_tc(const espdl_conv_desc &d, TcParams &p, const PackedOperands *o, cudaStream_t s);

} // namespace

int conv2d_tc(const espdl_conv_desc &d, void *workspace, size_t workspace_bytes, cudaStream_t s, const long long *peer_delta, int n_peer, int *row_sums)
{
    TcParams p;
    if (n_peer < 0 || n_peer > 7 || (n_peer > 0 && (d.dtype != ESPDL_DTYPE_INT8 || !peer_delta)))
        return ESPDL_ERR_UNSUPPORTED;
    if (!plan(d, p, n_peer > 0))
        return ESPDL_ERR_UNSUPPORTED;
    p.n_peer = n_peer;
    p.sched = nullptr, p.static_tiles = 0;
    for (int i = 0; i < 7; i++) p.peer_delta[i] = i < n_peer ? peer_delta[i] : 0;
    if (d.dtype != ESPDL_DTYPE_INT16)
        return launch_tc(d, p, nullptr, s);
    const size_t a = ((size_t)p.M * p.K + 255) / 256 * 256, b = ((size_t)p.N * p.K + 255) / 256 * 256;
    if (workspace_bytes < 2 * a + 2 * b + (row_sums ? 0 : p.M * sizeof(int)) || !workspace || ((uintptr_t)workspace % 16))
        return ESPDL_ERR_INVALID_ARG;
    uint8_t *w = (uint8_t *)workspace;
    const PackedOperands o = {w, w + a, w + 2 * a, w + 2 * a + b, row_sums ? row_sums : (int *)(w + 2 * a + 2 * b), p.K};
    const int st = pack_operands(d, 0, p.M, true, o, s);
    return st ? st : launch_tc(d, p, &o, s);
}

namespace {

int launch_tc(const espdl_conv_desc &d, TcParams &p, const PackedOperands *o, cudaStream_t s)
{
    const int n_peer = p.n_peer;
    const bool i16 = d.dtype == ESPDL_DTYPE_INT16;
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    p.early = in_model_scope();
    p.filter_early = p.early && !o;
    p.out = d.output;
    p.ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.row_sum = o ? o->row_sum : nullptr;
    p.res = (const int8_t *)d.residual;
    p.rps = d.residual_pixel_stride ? d.residual_pixel_stride : d.out_c;
    p.epi.bias = d.bias, p.epi.ew = d.filter_exponents, p.epi.lut = d.lut, p.epi.lut_stride = d.lut_channel_stride;
    p.epi.e_shift_base = d.out_exponent - d.in_exponent;
    p.epi.ew_scalar = d.filter_exponent, p.epi.per_channel = d.per_channel;
    p.epi.relu = d.activation == ESPDL_ACT_RELU, p.epi.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    p.epi.acc_bound = min(p.K, 65536) << 14;
    {
        TcParams pp = p;
        if (!i16 && n_peer == 0 && ips % 16 == 0 && pair_plan(d, pp))
            return launch_pair(d, pp, s);
    }

    CUtensorMap ma, mb, ma_lo, mb_lo;
    int st;
    if (!i16) {
        if ((st = make_map(&ma, d.input, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)ips, BLOCK_M, (uint32_t)p.swz, p.swz, (uint64_t)p.batch,
                           (uint64_t)p.M * ips)))
            return st;
        st = p.frag ? make_frag_map(&mb, d.filter, (uint64_t)p.N, (uint64_t)p.K, (uint32_t)p.block_n, p.swz)
                    : make_map(&mb, d.filter, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)p.K, (uint32_t)p.block_n, (uint32_t)p.swz, p.swz, (uint64_t)p.batch,
                               (uint64_t)d.filter_image_stride);
        if (st)
            return st;
        ma_lo = ma, mb_lo = mb;
    } else if ((st = make_map(&ma, o->a_hi, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)p.K, BLOCK_M, (uint32_t)p.swz, p.swz)) ||
               (st = make_map(&ma_lo, o->a_lo, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)p.K, BLOCK_M, (uint32_t)p.swz, p.swz)) ||
               (st = make_map(&mb, o->b_hi, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)p.K, (uint32_t)p.block_n, (uint32_t)p.swz, p.swz)) ||
               (st = make_map(&mb_lo, o->b_lo, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)p.K, (uint32_t)p.block_n, (uint32_t)p.swz, p.swz))) {
        return st;
    }
    const size_t stage_bytes = (size_t)(i16 ? 2 : 1) * (BLOCK_M + p.block_n) * p.swz;
    const size_t filter_bytes = p.resident ? ((size_t)p.resident * p.k_blocks * p.block_n * p.swz + 1023) & ~(size_t)1023 : 0;
    size_t smem = 1024 + (size_t)p.stages * (p.resident ? (size_t)BLOCK_M * p.swz : stage_bytes) + filter_bytes + (p.one_tile ? 0 : 4 * ((size_t)((BLOCK_M * p.out_pw + 1023) & ~1023) << p.in_turn)) + aux_bytes(p, i16);
    CUtensorMap mo = ma;
    if (!i16 && p.out_pw && !p.out_rows) {
        const int osw = p.out_pw == 128 ? 128 : (p.out_pw == 64 ? 64 : 0);
        if ((st = make_map(&mo, d.output, (uint64_t)p.M, (uint64_t)p.N, (uint64_t)p.ops, 32, (uint32_t)p.out_pw, osw, (uint64_t)p.batch,
                           (uint64_t)p.M * (uint64_t)p.ops)))
            return st;
    }
    if (i16 && !p.out_rows && (st = p.block_n % 64 == 0 ? make_map(&mo, d.output, (uint64_t)p.M, 2 * (uint64_t)p.N, 2 * (uint64_t)p.ops, BLOCK_M, 128, 128)
                                                        : make_map(&mo, d.output, (uint64_t)p.M, 2 * (uint64_t)p.N, 2 * (uint64_t)p.ops, BLOCK_M, 2 * (uint32_t)p.block_n, 0)))
        return st;
    if (smem < 120 * 1024) // more than half an SM's shared memory: one CTA per SM, so TMEM allocation never waits on a neighbour
        smem = 120 * 1024;
    const long long all_tiles = (long long)p.batch * p.m_tiles * p.n_tiles;
    if (all_tiles > 0x7fffffffll)
        return ESPDL_ERR_TOO_LARGE;
    const int grid = (int)min(all_tiles, (long long)num_sms());
    // three quarters of the tiles in the fixed order, the last quarter to whichever SM is free
    p.sched = all_tiles >= 4ll * grid && all_tiles < (1ll << 30) ? sched_counters(s) : nullptr;
    p.static_tiles = p.sched ? (int)(all_tiles * 3 / 4 / grid) * grid : (int)all_tiles;
    if (p.resident) { // row tiles; a group of CTAs among several has no counter of its own (65536 x 256 -> 256 without / with one: 10.8 / 11.4 us)
        if (p.n_groups > 1 || p.m_tiles < 4 * grid)
            p.sched = nullptr;
        p.static_tiles = p.sched ? p.m_tiles * 3ll / 4 / grid * grid : p.m_tiles;
    }
    static std::once_flag attr_once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(attr_once, [] {
        for (auto k : {gemm_tc_kernel<false, false, false>, gemm_tc_kernel<false, true, false>, gemm_tc_kernel<true, false, false>, gemm_tc_kernel<true, true, false>,
                       gemm_tc_kernel<false, false, true>, gemm_tc_kernel<false, true, true>})
            if (attr_err == cudaSuccess)
                attr_err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(SMEM_BUDGET_DEEP + 2048));
    });
    if (attr_err != cudaSuccess)
        return set_cuda_error(attr_err, "cudaFuncSetAttribute(gemm_tc_kernel)");
    const bool even = p.epi.half_even;
    const auto kernel = i16 ? (even ? gemm_tc_kernel<true, true, false> : gemm_tc_kernel<true, false, false>)
        : p.resident        ? (even ? gemm_tc_kernel<false, true, true> : gemm_tc_kernel<false, false, true>)
                            : (even ? gemm_tc_kernel<false, true, false> : gemm_tc_kernel<false, false, false>);
    launch_overlapped(kernel, dim3(grid), dim3(NUM_THREADS), smem, s, ma, mb, ma_lo, mb_lo, mo, p);
    count_launch();
    return check_launch("gemm_tc");
}

// The product that a packed conv is: rows = its output pixels, K = its window rounded up to 16 elements.
espdl_conv_desc packed_product(const espdl_conv_desc &d, int rows)
{
    espdl_conv_desc g = d;
    g.n = 1, g.in_h = g.out_h = 1, g.in_w = g.out_w = rows, g.in_c = (d.kh * d.kw * d.in_c + 15) / 16 * 16;
    g.kh = g.kw = g.stride_h = g.stride_w = g.dilation_h = g.dilation_w = 1;
    g.pad_top = g.pad_bottom = g.pad_left = g.pad_right = 0;
    g.in_pixel_stride = 0;
    g.out_pixel_stride = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    g.residual_pixel_stride = d.residual_pixel_stride ? d.residual_pixel_stride : d.out_c;
    return g;
}

constexpr size_t PACK_CHUNK = 64u << 20; // bytes of packed input per launch: it stays in L2 between the packing and the product

int packed_rows(const espdl_conv_desc &d)
{
    const long long M = (long long)d.n * d.out_h * d.out_w;
    const long long row = (long long)((d.kh * d.kw * d.in_c + 15) / 16 * 16) * (d.dtype == ESPDL_DTYPE_INT16 ? 2 : 1);
    return (int)min(M, max(1ll, (long long)PACK_CHUNK / row / BLOCK_M) * BLOCK_M);
}

size_t round256(size_t v) { return (v + 255) / 256 * 256; }

} // namespace

bool conv2d_packed_supported(const espdl_conv_desc &d)
{
    const bool i16 = d.dtype == ESPDL_DTYPE_INT16;
    if (d.group != 1 || d.filter_image_stride != 0 || (i16 && (d.lut || d.residual)))
        return false;
    const long long M = (long long)d.n * d.out_h * d.out_w, K = (long long)d.kh * d.kw * d.in_c;
    // Packing and product are two launches of a few microseconds each; below that the CUDA-core kernel reads the operands in place.
    if (K > (i16 ? 16384 : 65536) || M > 0x7fffffffll || conv2d_simt_estimate_us(d) < (i16 ? 13.f : 11.f))
        return false;
    TcParams p;
    return plan(packed_product(d, packed_rows(d)), p);
}

size_t conv2d_packed_workspace_bytes(const espdl_conv_desc &d)
{
    const size_t planes = d.dtype == ESPDL_DTYPE_INT16 ? 2 : 1, Kp = (size_t)(d.kh * d.kw * d.in_c + 15) / 16 * 16, rows = packed_rows(d);
    return planes * (round256(rows * Kp) + round256(d.out_c * Kp)) + (planes == 2 ? rows * sizeof(int) : 0);
}

int conv2d_packed(const espdl_conv_desc &d, void *workspace, size_t workspace_bytes, cudaStream_t s)
{
    if (workspace_bytes < conv2d_packed_workspace_bytes(d) || !workspace || ((uintptr_t)workspace % 16))
        return ESPDL_ERR_INVALID_ARG;
    const bool i16 = d.dtype == ESPDL_DTYPE_INT16;
    const long long M = (long long)d.n * d.out_h * d.out_w;
    const int chunk = packed_rows(d), Kp = (d.kh * d.kw * d.in_c + 15) / 16 * 16;
    const size_t a = round256((size_t)chunk * Kp), b = round256((size_t)d.out_c * Kp), es = i16 ? 2 : 1;
    uint8_t *w = (uint8_t *)workspace;
    PackedOperands o = {w, w + a, w + es * a, w + es * a + b, (int *)(w + 2 * a + 2 * b), Kp};
    for (long long row = 0; row < M; row += chunk) {
        const int rows = (int)min((long long)chunk, M - row);
        int st = pack_operands(d, row, rows, row == 0, o, s);
        if (st)
            return st;
        espdl_conv_desc g = packed_product(d, rows);
        g.input = o.a_hi, g.filter = o.b_hi;
        g.output = (char *)d.output + (size_t)row * g.out_pixel_stride * es;
        if (d.residual)
            g.residual = (const char *)d.residual + (size_t)row * g.residual_pixel_stride;
        TcParams p;
        if (!plan(g, p))
            return ESPDL_ERR_UNSUPPORTED;
        p.n_peer = 0;
        for (long long &delta : p.peer_delta) delta = 0;
        st = launch_tc(g, p, &o, s);
        if (st)
            return st;
    }
    return ESPDL_OK;
}

} // namespace espdl

// ------------------------------------------------------------------ allocation-free int16 Gemm / pointwise conv
// Fixed scratch for espdl_b200_gemm_s16_static: the byte planes of both int16 operands live in this array
// instead of a caller-provided or cached cudaMalloc buffer.  It is part of the library image, so every GPU
// that loads the library carries it until the process exits.
namespace espdl {
static __device__ __align__(256) unsigned char g_static_limb_scratch[ESPDL_B200_STATIC_SCRATCH_BYTES];
static __device__ int g_static_row_sums[ESPDL_B200_STATIC_SCRATCH_BYTES / 2 / 16]; // one per row; a row's planes take 32 bytes at least
}

extern "C" int espdl_b200_gemm_s16_static(const espdl_conv_desc *desc, void *stream)
{
    using namespace espdl;
    // the same descriptor checks as espdl_b200_conv2d, before anything is planned or launched
    const int st = conv_validate(desc);
    if (st)
        return st;
    if (desc->dtype != ESPDL_DTYPE_INT16 || desc->lut || desc->residual || desc->filter_image_stride != 0 || !conv2d_tc_supported(*desc))
        return ESPDL_ERR_UNSUPPORTED;
    if (desc->n == 0)
        return ESPDL_OK;
    const size_t need = conv2d_tc_workspace_bytes(*desc) - (size_t)desc->n * desc->out_h * desc->out_w * sizeof(int); // the planes
    if (need > (size_t)ESPDL_B200_STATIC_SCRATCH_BYTES)
        return set_error_text(ESPDL_ERR_TOO_LARGE,
                              "espdl_b200_gemm_s16_static: %zu bytes of scratch needed, the fixed array holds %u; use "
                              "espdl_b200_conv2d_ws with a caller-owned buffer",
                              need, (unsigned)ESPDL_B200_STATIC_SCRATCH_BYTES);
    // In host code the array's name is only a handle; the device address comes from cudaGetSymbolAddress, asked
    // once per device with that device current.
    static void *addr_of_device[64] = {nullptr}, *sums_of_device[64] = {nullptr};
    static std::mutex addr_mutex;
    int dev = -1;
    ESPDL_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64)
        return ESPDL_ERR_NO_DEVICE;
    void *scratch = nullptr, *sums = nullptr;
    {
        std::lock_guard<std::mutex> lock(addr_mutex);
        if (!addr_of_device[dev]) {
            void *p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_static_limb_scratch);
            if (e != cudaSuccess)
                return set_cuda_error(e, "cudaGetSymbolAddress(g_static_limb_scratch)");
            if ((e = cudaGetSymbolAddress(&sums_of_device[dev], g_static_row_sums)) != cudaSuccess)
                return set_cuda_error(e, "cudaGetSymbolAddress(g_static_row_sums)");
            addr_of_device[dev] = p;
        }
        scratch = addr_of_device[dev], sums = sums_of_device[dev];
    }
    return conv2d_tc(*desc, scratch, (size_t)ESPDL_B200_STATIC_SCRATCH_BYTES, (cudaStream_t)stream, nullptr, 0, (int *)sums);
}

#ifdef ESPDL_TC_TIMING
// Measurement builds only: copies the role cycle counters of the last gemm_tc_kernel launch (8 values per CTA).
extern "C" int espdl_b200_debug_gemm_timing(long long *out, int ctas)
{
    return cudaMemcpyFromSymbol(out, espdl::g_tc_timing, sizeof(long long) * 8 * (size_t)(ctas > 256 ? 256 : ctas)) == cudaSuccess ? 0 : -3;
}
extern "C" int espdl_b200_debug_gemm_clock(long long *out, int ctas)
{
    return cudaMemcpyFromSymbol(out, espdl::g_tc_clock, sizeof(long long) * 4 * (size_t)(ctas > 256 ? 256 : ctas)) == cudaSuccess ? 0 : -3;
}
#endif
