// Dense Conv2D (any filter size, stride 1 or 2, dilation, padding; int8, groups = 1) as an implicit GEMM on the
// tensor cores.  Replaces dl::base::conv2d<int8_t,...> (esp-dl/dl/base/dl_base_conv2d.cpp:9-163, MAC kernels
// conv2d_33cn / conv2d_hwcn) for filters larger than 1x1, with the epilogue of
// esp-dl/dl/base/dl_base_activate_buffer.hpp:27-73.
//
//   out[n, y, x, co] = epilogue( sum_{ky, kx, c} in[n, y*S + ky*D - pt, x*S + kx*D - pl, c] * w[co][ky][kx][c] + bias[co] )
//
// No im2col buffer exists anywhere.  A tile is R rows x P columns of output pixels of one image (R*P <= 128 = the
// M of a tcgen05 MMA) x up to 256 output channels.  The reduction runs over the filter taps: for tap (ky, kx) and a
// block of up to 128 input channels, ONE 4-D TMA box {channels, P, R, 1} of the NHWC input, displaced by the tap
// (and stepping S pixels per index with TMA element strides), lands in shared memory as the K-major swizzled A
// operand whose rows are the tile's pixels; coordinates outside the image are zero-filled by the TMA unit, which is
// the reference's padding rule (taps outside the image contribute nothing).  B is a 2-D box of the [Cout][KH*KW*Cin]
// filter at column (ky*KW + kx)*Cin.  KH*KW*ceil(Cin/128) such stages accumulate into one TMEM accumulator; the
// epilogue is the pointwise tile kernel's (constants of the one-add-one-shift form staged in shared memory, rows
// requantised into a shared tile and moved out by a 4-D TMA store that clips at the image border).
// Roles, barriers and bounded waits are those of gemm_tc.cu.
#include "tc_common.cuh"

#include <mutex>

namespace espdl {

__device__ int *g_conv_tc_error = nullptr; // the status word of bounded waits (common.cuh)

int bind_device_error_conv(int *word)
{
    ESPDL_CUDA_TRY(cudaMemcpyToSymbol(g_conv_tc_error, &word, sizeof(word)));
    return ESPDL_OK;
}

namespace {

using namespace tc;

constexpr int CV_THREADS = 64 + 16 * 32; // TMA warp, MMA warp, 16 epilogue warps in four groups
constexpr int CV_MAX_STAGES = 8;
constexpr int CV_MAX_ACC = 4;
constexpr size_t CV_SMEM_BUDGET = 200 * 1024;

struct ConvTcParams {
    int early; // bias, exponents and table are constants of the model: read ahead of the previous kernel's end
    int n, oh, ow, cin, cout;
    int kh, kw, S, D, pt, pl;
    int P, R;                     // tile: R rows x P columns of output pixels
    int xtiles, ytiles, n_tiles;  // tiles per image row / column, tiles along Cout
    int block_n, swz, cblocks;    // Cout per tile, bytes of Cin per stage, stages per tap
    int stages, acc_stages, tmem_cols;
    int out_pw, out_mask;         // staged epilogue: bytes per row of a group's piece (0 = direct row stores), swizzle mask
    void *out;
    long long ops;                // output pixel stride in bytes
    EpiConfig epi;
};

__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, uint32_t src, int c0, int c1, int c2, int c3)
{
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map), "r"(src), "r"(c0), "r"(c1),
                 "r"(c2), "r"(c3)
                 : "memory");
}

template <bool EVEN>
__global__ void __launch_bounds__(CV_THREADS, 1)
conv_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_out,
               const ConvTcParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int a_bytes = 128 * p.swz;
    const int b_bytes = p.block_n * p.swz;
    const int stage_bytes = a_bytes + b_bytes;
    const int n_pad = p.n_tiles * p.block_n;
    uint8_t *out_stage = smem + (size_t)p.stages * stage_bytes;
    const int out_tile_bytes = (128 * p.out_pw + 1023) & ~1023;
    uint8_t *aux = out_stage + 4 * (size_t)out_tile_bytes;
    FastParam *fast_s = (FastParam *)aux;
    uint64_t *bars = (uint64_t *)(aux + sizeof(FastParam) * (size_t)n_pad);
    uint64_t *full_bar = bars, *empty_bar = bars + CV_MAX_STAGES, *tfull_bar = bars + 2 * CV_MAX_STAGES, *tempty_bar = tfull_bar + CV_MAX_ACC;
    uint32_t *tmem_slot = (uint32_t *)(tempty_bar + CV_MAX_ACC);
    int *slow_flag = (int *)(tmem_slot + 1);
    uint8_t *lut_s = (uint8_t *)(slow_flag + 3); // the fused 8-bit table, 256 bytes, 16-byte aligned

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_per_image = p.ytiles * p.xtiles * p.n_tiles;
    const int total_tiles = p.n * tiles_per_image;
    const int parts = 4 / p.acc_stages;
    const int taps = p.kh * p.kw;
    const uint32_t a_tx = (uint32_t)(p.P * p.R * p.swz); // the A box holds P*R rows; rows up to 128 keep stale bytes

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int a = 0; a < CV_MAX_ACC; a++) {
            mbar_init(smem_u32(&tfull_bar[a]), 1);
            mbar_init(smem_u32(&tempty_bar[a]), 4 * parts);
        }
        *slow_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1)
        tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0)
        grid_dep_launch(); // set up: the next kernel's CTAs may take SMs as they become free

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one()) {
            grid_dep_wait(); // the previous kernel's output, before the first load; the other roles act on what the producer brought in
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const int nt = tile % p.n_tiles;
                const int xt = (tile / p.n_tiles) % p.xtiles;
                const int yt = (tile / (p.n_tiles * p.xtiles)) % p.ytiles;
                const int img = tile / tiles_per_image;
                const int n0 = nt * p.block_n;
                for (int tap = 0; tap < taps && ok; tap++) {
                    const int ky = tap / p.kw, kx = tap % p.kw;
                    const int ix = xt * p.P * p.S + kx * p.D - p.pl;
                    const int iy = yt * p.R * p.S + ky * p.D - p.pt;
                    for (int cb = 0; cb < p.cblocks; cb++) {
                        if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1)) {
                            ok = false;
                            break;
                        }
                        const uint32_t bar = smem_u32(&full_bar[stage]);
                        uint8_t *st = smem + (size_t)stage * stage_bytes;
                        mbar_arrive_expect_tx(bar, a_tx + (uint32_t)b_bytes);
                        tma_load_4d(smem_u32(st), &map_a, cb * p.swz, ix, iy, img, bar);
                        tma_load_2d(smem_u32(st + a_bytes), &map_b, tap * p.cin + cb * p.swz, n0, bar);
                        if (++stage == p.stages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
            if (!ok)
                report_timeout(g_conv_tc_error);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            const uint32_t idesc = idesc_i8(1, 1, 128, p.block_n);
            const int ksteps = p.swz / 32;
            const int kblocks = taps * p.cblocks;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                if (!mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1)) {
                    ok = false;
                    break;
                }
                fence_after();
                const uint32_t d0 = tmem_base + (uint32_t)(acc * p.block_n);
                for (int kb = 0; kb < kblocks; kb++) {
                    if (!mbar_wait(smem_u32(&full_bar[stage]), phase)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint32_t st = smem_u32(smem + (size_t)stage * stage_bytes);
                    const uint64_t da = smem_desc_swizzled(st, p.swz);
                    const uint64_t db = smem_desc_swizzled(st + a_bytes, p.swz);
                    for (int k = 0; k < ksteps; k++) mma_i8(d0, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb | k) != 0);
                    commit(smem_u32(&empty_bar[stage]));
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok)
                    break;
                commit(smem_u32(&tfull_bar[acc]));
                if (++acc == p.acc_stages) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            }
            if (!ok)
                report_timeout(g_conv_tc_error);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..17)
        const int ew = warp - 2;
        const int group = ew >> 2;
        const int acc = group % p.acc_stages;
        const int part = group / p.acc_stages;
        const int lane_group = warp & 3;
        const int row_in_tile = lane_group * 32 + lane;
        const int et = threadIdx.x - 64;
        if (!p.early)
            grid_dep_wait(); // bias, exponents and table may be what the previous kernel wrote
        stage_fast_params(p.epi, fast_s, p.cout, n_pad, et, 16 * 32, slow_flag);
        if (p.epi.lut)
            stage_lut(p.epi.lut, lut_s, et, 16 * 32);
        asm volatile("bar.sync 1, %0;" ::"n"(16 * 32) : "memory");
        // a fused table rides on the staged form; the direct-store form applies it in its general path
        const bool fast = !*slow_flag && !p.epi.lut_stride && (long long)p.cin * p.kh * p.kw <= 32768;
        const uint32_t fp_base = epi_param_base(fast_s);
        const int floor_q = p.epi.relu ? 0 : INT_MIN;
        const int ry = row_in_tile / p.P, rx = row_in_tile % p.P;
        uint32_t acc_phase = 0;
        bool ok = true;
        int local = 0;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, local++) {
            if (local % p.acc_stages != acc)
                continue;
            const int nt = tile % p.n_tiles;
            const int xt = (tile / p.n_tiles) % p.xtiles;
            const int yt = (tile / (p.n_tiles * p.xtiles)) % p.ytiles;
            const int img = tile / tiles_per_image;
            const int n0 = nt * p.block_n;
            if (!mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase)) {
                ok = false;
                break;
            }
            acc_phase ^= 1;
            fence_after();
            const uint32_t t0 = tmem_base + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)(acc * p.block_n);
            if (fast && p.out_pw) {
                const bool leader = (ew & 3) == 0 && lane == 0;
                const uint32_t buf = smem_u32(out_stage + (size_t)group * out_tile_bytes);
                if (leader)
                    bulk_wait_read_all();
                named_bar(2 + group, 128);
                const int col0 = part * p.out_pw;
                const uint32_t fpp = fp_base + (uint32_t)(n0 + col0) * 8u;
                if (p.epi.lut) {
                    epilogue_stage_lut<EVEN>(t0 + col0, fpp, buf, row_in_tile, p.out_pw, (uint32_t)p.out_mask, floor_q, smem_u32(lut_s));
                } else if (p.out_pw == 128)
                    epilogue_stage<128, EVEN>(t0 + col0, fpp, buf, row_in_tile, 128, floor_q);
                else if (p.out_pw == 64)
                    epilogue_stage<64, EVEN>(t0 + col0, fpp, buf, row_in_tile, 64, floor_q);
                else
                    epilogue_stage<0, EVEN>(t0 + col0, fpp, buf, row_in_tile, p.out_pw, floor_q);
                // the accumulator is free once this warp's TMEM loads are done: hand it back before the tile is stored
                fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(smem_u32(&tempty_bar[acc]));
                fence_async_smem();
                named_bar(2 + group, 128);
                if (leader) {
                    tma_store_4d(&map_out, buf, n0 + col0, xt * p.P, yt * p.R, img); // clipped at the image border and at Cout
                    bulk_commit();
                }
                continue;
            } else {
                // direct rows: any rounding mode, any shift, optional LUT, any alignment
                const int oy = yt * p.R + ry, ox = xt * p.P + rx;
                const bool row_ok = ry < p.R && oy < p.oh && ox < p.ow;
                int8_t *orow = (int8_t *)p.out + (((long long)img * p.oh + oy) * p.ow + ox) * p.ops + n0;
                const uintptr_t amix = (uintptr_t)p.ops | (((uintptr_t)p.out) + (uintptr_t)n0) | 16u;
                const int out_align = (int)(amix & (~amix + 1));
                int chunk = 0;
                for (int c0 = 0; c0 < p.block_n; c0 += 16, chunk++) {
                    if ((chunk >> 1) % parts != part)
                        continue;
                    int32_t v[16];
                    ld16(t0 + c0, v);
                    ld_wait16(v);
                    uint32_t pk[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                    if (fast) {
                        if (p.epi.relu)
                            requant16_fast<true, EVEN>(v, fast_s + n0 + c0, pk);
                        else
                            requant16_fast<false, EVEN>(v, fast_s + n0 + c0, pk);
                        if (p.epi.lut) { // a fused table on rows that leave unstaged: same lookups on the packed words
#pragma unroll
                            for (int q = 0; q < 4; q++) pk[q] = lut4(pk[q], smem_u32(lut_s));
                        }
                    } else {
                        requant16_general(v, p.epi, n0 + c0, p.cout, pk);
                    }
                    const int count = min(16, p.cout - (n0 + c0));
                    if (row_ok && count > 0)
                        store_bytes(orow + c0, pk, count, out_align);
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&tempty_bar[acc]));
        }
        if (!ok && lane == 0)
            report_timeout(g_conv_tc_error);
        if (p.out_pw && (ew & 3) == 0 && lane == 0)
            bulk_wait_all();
    }

    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        tmem_dealloc(tmem_base, p.tmem_cols);
    }
}

// ------------------------------------------------------------------------------------------ stride-1 windows from ONE patch
// The kernel above fetches every input byte once per filter tap (nine boxes of 128 pixels for a 3x3 window), and with
// 32-128 byte rows that traffic, not the MMAs, bounds it (64 -> 64 channels at 80x80: 1.8 GB through the TMA unit for a
// 0.4 GB tensor).  For stride 1, dilation 1 and one channel block the taps are shifted views of the same pixels: here a
// tile's input arrives as ONE box of PW positions by RT + KH - 1 rows whose dense shared-memory image is a run of "flat
// positions" row * PW + x, and a shift is the same run started some rows later - a descriptor start address, no data movement
// (the swizzle is a function of the absolute shared-memory address, so a start moved by whole rows stays consistent with what
// the TMA unit wrote).  The 128 rows of an MMA are 128 consecutive flat positions, of which the last `span` of every patch row
// are not outputs (their windows run into the next row); they are computed and dropped.  The whole filter stays in shared
// memory for the life of the CTA.  Borders are TMA zero fill.  Epilogue and roles as above; a tile leaves through one TMA store.
//
// A position is G pixels of an image row: an MMA row, and G * Cout accumulator columns.  Input pixel i of a position (i runs from -pl to
// G - 1 + KW - 1 - pl, pixels outside 0 .. G - 1 being those of the neighbouring positions) adds to output pixel j through tap
// kx = i + pl - j: consecutive outputs, descending taps.  With a filter row's taps stored in descending order, ONE MMA per
// input pixel and 32 channels therefore multiplies pixel i of all positions by the taps of all the outputs it belongs to,
// landing in the columns of those outputs - G + KW - 1 MMAs where G separate pixels take G * KW.  Why: an MMA reads its 128
// rows of A (4 KB) whatever its width, so that N = 64 keeps the tensor cores a third busy (51 cycles of shared-memory reads for
// 32 of math, measured); and G pixels of 128 / G channels make rows of 128 bytes, which the tensor cores read at full rate
// where 64- and 32-byte rows (and their swizzles) take 1.5 and 1.8 times as long.  Measured, 64 -> 64 channels, 3x3, 1024 images of
// 56x56: 190 us with one pixel a position, 112 with four (2.1 POPS; a large Gemm runs at 2.8); 32 -> 32, 16 images of 160x160: 26.6 -> 9.0.
// (Before, the taps of a filter row stood side by side along N and the epilogue added their columns across lanes: 238 us, bound
// by its shuffles.)
struct PatchStep {
    uint32_t ab; // offsets of A and (high half) B in 16-byte units
    uint32_t dn; // accumulator column, bit 15: the columns start from zero; high half: N
};

constexpr int PATCH_MAX_STEPS = 16;
constexpr int PATCH_THREADS = CV_THREADS + 32; // a second MMA warp

struct PatchParams {
    int early; // filter, bias, exponents and table are constants of the model: read ahead of the previous kernel's end
    int n, oh, ow, cin, cout;
    int kh, kw, pt, pl;
    int G, glo;                   // pixels per position; the first position a window reaches, relative to its own (0 or negative)
    int planes, plane_bytes;      // rows of G pixels (1), or a plane of rows per pixel of the position (G; channel slices), bytes from one plane to the next
    int PW, RT, PV;               // positions per patch row, image rows per tile, outputs per row = PW - span
    int xtiles, ytiles;
    int ncols, a_row, swz_b;      // accumulator columns = G * Cout; bytes of a row of A and of B (= their swizzle)
    int stages, acc_stages, tmem_cols;
    int issuers;                  // MMA warps that take the tiles in turn
    int patch_bytes, patch_tx;    // shared-memory stride of a stage (with slack for the last rows' overrun), bytes its boxes deliver
    int out_pw, out_mask, out_box; // columns per epilogue group, swizzle mask, channels per row of the output's box
    int dense_out;                // the output's pixels follow one another: a position's columns are consecutive bytes
    int staged;                   // the tile leaves through shared memory and TMA stores (else rows go out of registers)
    int nfirst, nrest;
    PatchStep first[PATCH_MAX_STEPS + 1], rest[PATCH_MAX_STEPS + 1]; // MMAs of the first filter row and of the others (per 32 channels)
    void *out;
    long long ops;                // output pixel stride in bytes
    EpiConfig epi;
};

__device__ __forceinline__ void tma_store_5d(const CUtensorMap *map, uint32_t src, int c0, int c1, int c2, int c3, int c4)
{
    asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];" ::"l"(map), "r"(src), "r"(c0), "r"(c1),
                 "r"(c2), "r"(c3), "r"(c4)
                 : "memory");
}

template <bool EVEN>
__global__ void __launch_bounds__(PATCH_THREADS, 1)
conv_patch_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_out,
                  const __grid_constant__ PatchParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int taps = p.kh * p.kw;
    const int b_tap = p.cout * p.swz_b;                        // one tap's filter rows: whole swizzle patterns (Cout % 16 == 0)
    uint8_t *filt_s = smem;                                    // [ky][taps of the row, descending][Cout][Cin]
    uint8_t *patch_s = smem + (((size_t)taps * b_tap + 1023) & ~(size_t)1023); // stages x patch
    uint8_t *out_stage = patch_s + (size_t)p.stages * p.patch_bytes;
    const int out_tile_bytes = p.staged ? (128 * p.out_pw + 1023) & ~1023 : 0;
    uint8_t *aux = out_stage + 4 * (size_t)out_tile_bytes;
    FastParam *fast_s = (FastParam *)aux;
    uint64_t *bars = (uint64_t *)(aux + sizeof(FastParam) * (size_t)p.ncols);
    uint64_t *full_bar = bars, *empty_bar = bars + CV_MAX_STAGES, *tfull_bar = bars + 2 * CV_MAX_STAGES, *tempty_bar = tfull_bar + CV_MAX_ACC;
    uint64_t *filt_bar = tempty_bar + CV_MAX_ACC;
    uint32_t *tmem_slot = (uint32_t *)(filt_bar + 1);
    int *slow_flag = (int *)(tmem_slot + 1);
    uint8_t *lut_s = (uint8_t *)(slow_flag + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total_tiles = p.n * p.ytiles * p.xtiles;
    const int parts = 4 / p.acc_stages;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int a = 0; a < CV_MAX_ACC; a++) {
            mbar_init(smem_u32(&tfull_bar[a]), 1);
            mbar_init(smem_u32(&tempty_bar[a]), 4 * parts);
        }
        mbar_init(smem_u32(filt_bar), 1);
        *slow_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1)
        tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0)
        grid_dep_launch(); // set up: the next kernel's CTAs may take SMs as they become free

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one()) {
            // the filter, once: one box per tap (ahead of the previous kernel's end where it is a model's constant)
            if (!p.early)
                grid_dep_wait();
            mbar_arrive_expect_tx(smem_u32(filt_bar), (uint32_t)(taps * b_tap));
            for (int ky = 0; ky < p.kh; ky++)
                for (int kx = 0; kx < p.kw; kx++)
                    tma_load_2d(smem_u32(filt_s + (size_t)(ky * p.kw + p.kw - 1 - kx) * b_tap), &map_b, (ky * p.kw + kx) * p.cin, 0, smem_u32(filt_bar));
            grid_dep_wait(); // the previous kernel's output, before the first patch; the other roles act on what the producer brought in
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            TileWalk w(blockIdx.x, gridDim.x, p.xtiles, p.ytiles);
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, w.next()) {
                if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1)) {
                    ok = false;
                    break;
                }
                const uint32_t bar = smem_u32(&full_bar[stage]);
                const uint32_t st = smem_u32(patch_s + (size_t)stage * p.patch_bytes);
                mbar_arrive_expect_tx(bar, (uint32_t)p.patch_tx);
                for (int j = 0; j < p.planes; j++)
                    tma_load_5d(st + (uint32_t)(j * p.plane_bytes), &map_a, 0, j, w.x * p.PV + p.glo, w.y * p.RT - p.pt, w.n, bar);
                if (++stage == p.stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            if (!ok)
                report_timeout(g_conv_tc_error);
        }
        __syncwarp();
    } else if (warp == 1 || warp == 18) {
        // ------------------------------------------------------------ MMA issuers
        // Two warps take the tiles in turn: one alone spent longer on a tile's waits and MMAs (some 400 cycles and 25 to 100 an MMA) than the
        // tensor cores (64 -> 64 channels, 56x56x1024: 135 us with
        // one, 115 with two).
        if (elect_one()) {
            const int second = warp == 1 ? 0 : 1;
            int stage = second, acc = second; // two stages and two accumulators at least, and an even number of these
            uint32_t phase = 0, acc_phase = 0;
            bool ok = mbar_wait(smem_u32(filt_bar), 0);
            const int ksteps = p.cin / 32;
            const uint64_t a0 = smem_desc_swizzled(smem_u32(patch_s), p.a_row), b0 = smem_desc_swizzled(smem_u32(filt_s), p.swz_b);
            const uint32_t idesc0 = idesc_i8(1, 1, 128, 0);
            const uint32_t row_a = (uint32_t)(p.PW * p.a_row) >> 4, row_b = (uint32_t)(p.kw * b_tap) >> 4, stage_a = (uint32_t)p.patch_bytes >> 4;
            for (int tile = (int)blockIdx.x + second * (int)gridDim.x; tile < total_tiles && ok && second < p.issuers; tile += p.issuers * (int)gridDim.x) {
                if (!mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1) || !mbar_wait(smem_u32(&full_bar[stage]), phase)) {
                    ok = false;
                    break;
                }
                fence_after();
                const uint32_t d0 = tmem_base + (uint32_t)(acc * p.ncols);
                const uint64_t da = a0 + (uint64_t)((uint32_t)stage * stage_a);
                auto issue = [&](uint32_t d, uint64_t x, uint64_t f, uint32_t id, uint32_t add) {
                    mma_i8(d, x, f, id, add);
                    if (ksteps > 1)
                        mma_i8(d, x + 2, f + 2, id, 1u);
                    if (ksteps > 2) {
                        mma_i8(d, x + 4, f + 4, id, 1u);
                        mma_i8(d, x + 6, f + 6, id, 1u);
                    }
                };
                PatchStep t = p.first[0];
                for (int e = 0; e < p.nfirst; e++) {
                    const PatchStep next = p.first[e + 1]; // its load in flight beside this step's MMAs
                    issue(d0 + (t.dn & 0x7fffu), da + (uint64_t)(t.ab & 0xffffu), b0 + (uint64_t)(t.ab >> 16), idesc0 + ((t.dn & 0xffff0000u) >> 2),
                          !(t.dn & 0x8000u));
                    t = next;
                }
                t = p.rest[0];
                for (int e = 0; e < p.nrest; e++) {
                    const PatchStep next = p.rest[e + 1];
                    const uint32_t d = d0 + (t.dn & 0x7fffu), id = idesc0 + ((t.dn & 0xffff0000u) >> 2);
                    uint64_t x = da + (uint64_t)(t.ab & 0xffffu), f = b0 + (uint64_t)(t.ab >> 16);
                    for (int ky = 1; ky < p.kh; ky++) {
                        x += row_a, f += row_b;
                        issue(d, x, f, id, 1u);
                    }
                    t = next;
                }
                commit(smem_u32(&empty_bar[stage]));
                commit(smem_u32(&tfull_bar[acc]));
                if ((stage += p.issuers) >= p.stages) {
                    stage -= p.stages;
                    phase ^= 1;
                }
                if ((acc += p.issuers) >= p.acc_stages) {
                    acc -= p.acc_stages;
                    acc_phase ^= 1;
                }
            }
            if (!ok)
                report_timeout(g_conv_tc_error);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..17)
        const int ew = warp - 2;
        const int group = ew >> 2;
        const int acc = group % p.acc_stages;
        const int part = group / p.acc_stages;
        const int lane_group = warp & 3;
        const int row_in_tile = lane_group * 32 + lane;
        const int et = threadIdx.x - 64;
        if (!p.early)
            grid_dep_wait(); // bias, exponents and table may be what the previous kernel wrote
        for (int j = 0; j < p.G; j++) stage_fast_params(p.epi, fast_s + j * p.cout, p.cout, p.cout, et, 16 * 32, slow_flag);
        if (p.epi.lut)
            stage_lut(p.epi.lut, lut_s, et, 16 * 32);
        asm volatile("bar.sync 1, %0;" ::"n"(16 * 32) : "memory");
        const bool fast = !*slow_flag && !p.epi.lut_stride && (long long)p.cin * p.kh * p.kw <= 32768;
        const uint32_t fp_base = epi_param_base(fast_s);
        const int floor_q = p.epi.relu ? 0 : INT_MIN;
        const int r = row_in_tile / p.PW, xx = row_in_tile - r * p.PW; // this thread's image row and position of a tile
        const bool counts = xx < p.PV && r < p.RT;
        const int row = r * p.PV + xx;                                // its row of the staging tile, which holds outputs only
        const int col0 = part * p.out_pw;
        const uint32_t fpp = fp_base + (uint32_t)col0 * 8u;
        const uint32_t tbl = p.epi.lut ? smem_u32(lut_s) : 0u;
        uint32_t acc_phase = 0;
        bool ok = true;
        const int first = (int)blockIdx.x + acc * (int)gridDim.x, step = p.acc_stages * (int)gridDim.x; // an accumulator takes every acc_stages-th tile
        TileWalk w(first, step, p.xtiles, p.ytiles);
        for (int tile = first; tile < total_tiles && ok; tile += step, w.next()) {
            if (!mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase)) {
                ok = false;
                break;
            }
            acc_phase ^= 1;
            fence_after();
            const uint32_t t0 = tmem_base + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)(acc * p.ncols);
            if (!fast || !p.staged) {
                // rows out of registers: no room for staging tiles next to a large resident filter, or any rounding, shift and table
                const int oy = w.y * p.RT + r, ox = (w.x * p.PV + xx) * p.G;
                int8_t *orow = (int8_t *)p.out + (((long long)w.n * p.oh + oy) * p.ow + ox) * p.ops;
                const bool row_ok = counts && oy < p.oh && ox < p.ow;
                int j = col0 / p.cout, ch = col0 - j * p.cout; // output pixel and channel of the column
                for (int c = 0; c < p.out_pw; c += 16) {
                    int32_t v[16];
                    uint32_t pk[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                    ld16(t0 + col0 + c, v);
                    ld_wait16(v);
                    if (fast) {
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            pk[q] = requant4_floor<EVEN>(v + 4 * q, fpp + (uint32_t)(c + 4 * q) * 8u, floor_q);
                            if (tbl)
                                pk[q] = lut4(pk[q], tbl);
                        }
                    } else {
                        requant16_general(v, p.epi, ch, p.cout, pk);
                    }
                    if (row_ok)
                        *(uint4 *)(orow + j * p.ops + ch) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    if ((ch += 16) == p.cout)
                        ch = 0, j++;
                }
                fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(smem_u32(&tempty_bar[acc]));
                continue;
            }
            const bool leader = (ew & 3) == 0 && lane == 0;
            const uint32_t buf = smem_u32(out_stage + (size_t)group * out_tile_bytes);
            if (leader)
                bulk_wait_read_all();
            named_bar(2 + group, 128);
            const uint32_t rb = buf + (uint32_t)(row * p.out_pw), rx = (((uint32_t)(row * p.out_pw) >> 7) & (uint32_t)p.out_mask) << 4;
            if (p.epi.lut)
                epilogue_stage_lut<EVEN>(t0 + col0, fpp, buf, row, p.out_pw, (uint32_t)p.out_mask, floor_q, tbl, counts);
            else if (p.out_pw == 128)
                epilogue_stage_at<128, EVEN>(t0 + col0, fpp, rb, rx, 128, floor_q, counts);
            else if (p.out_pw == 64)
                epilogue_stage_at<64, EVEN>(t0 + col0, fpp, rb, rx, 64, floor_q, counts);
            else
                epilogue_stage_at<0, EVEN>(t0 + col0, fpp, rb, rx, p.out_pw, floor_q, counts);
            fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&tempty_bar[acc]));
            fence_async_smem();
            named_bar(2 + group, 128);
            if (leader) {
                // rows and positions outside the image are clipped
                if (p.dense_out)
                    tma_store_5d(&map_out, buf, col0, 0, w.x * p.PV, w.y * p.RT, w.n);
                else
                    tma_store_5d(&map_out, buf, col0 % p.cout, col0 / p.cout, w.x * p.PV, w.y * p.RT, w.n);
                bulk_commit();
            }
        }
        if (!ok && lane == 0)
            report_timeout(g_conv_tc_error);
        if ((ew & 3) == 0 && lane == 0)
            bulk_wait_all();
    }

    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        tmem_dealloc(tmem_base, p.tmem_cols);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn conv_encode()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

CUtensorMapSwizzle swizzle_of(int bytes)
{
    return bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
        : (bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : (bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE));
}

size_t conv_aux_bytes(const ConvTcParams &p) { return sizeof(FastParam) * (size_t)p.n_tiles * p.block_n + (2 * CV_MAX_STAGES + 2 * CV_MAX_ACC) * 8 + 32 + 256; }

bool conv_plan(const espdl_conv_desc &d, ConvTcParams &p)
{
    p.n = d.n, p.oh = d.out_h, p.ow = d.out_w, p.cin = d.in_c, p.cout = d.out_c;
    p.kh = d.kh, p.kw = d.kw, p.S = d.stride_h, p.D = d.dilation_h, p.pt = d.pad_top, p.pl = d.pad_left;
    // tile shape: the R x P (R*P <= 128) that wastes the fewest accumulator rows on this image
    double best = -1;
    p.P = 1, p.R = 1;
    for (int P = 1; P <= 128 && P <= d.out_w && P * p.S <= 256; P++) {
        const int R = min(128 / P, min(d.out_h, 256 / p.S));
        if (R < 1)
            continue;
        const double eff = ((double)d.out_w / (((d.out_w + P - 1) / P) * P)) * ((double)d.out_h / (((d.out_h + R - 1) / R) * R)) * (P * R / 128.0);
        if (eff > best + 1e-9) {
            best = eff;
            p.P = P, p.R = R;
        }
    }
    p.xtiles = (d.out_w + p.P - 1) / p.P, p.ytiles = (d.out_h + p.R - 1) / p.R;
    p.n_tiles = (p.cout + 255) / 256;
    p.block_n = (((p.cout + p.n_tiles - 1) / p.n_tiles) + 15) / 16 * 16;
    if (p.block_n > 128)
        p.block_n = (p.block_n + 31) / 32 * 32;
    p.n_tiles = (p.cout + p.block_n - 1) / p.block_n;
    p.swz = p.cin >= 96 ? 128 : (p.cin > 32 ? 64 : 32);
    p.cblocks = (p.cin + p.swz - 1) / p.swz;
    p.acc_stages = 4 * p.block_n <= 512 ? 4 : 2;
    int pow2 = 32;
    while (pow2 < p.acc_stages * p.block_n) pow2 *= 2;
    if (pow2 > 512)
        return false;
    p.tmem_cols = pow2;
    const long long ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.out_pw = 0, p.out_mask = 0;
    if (ops % 16 == 0 && d.out_c % 16 == 0 && ((uintptr_t)d.output % 16) == 0 && !getenv("ESPDL_B200_DIRECT_STORES")) { // (a TMA store clips rows in units of 16 bytes)
        const int parts = 4 / p.acc_stages;
        if (p.block_n % (16 * parts) == 0 && p.block_n / parts <= 128) {
            p.out_pw = p.block_n / parts;
            p.out_mask = p.out_pw == 128 ? 7 : (p.out_pw == 64 ? 3 : 0);
        }
    }
    const size_t stage_bytes = (size_t)(128 + p.block_n) * p.swz;
    size_t out_bytes = 4 * (size_t)((128 * p.out_pw + 1023) & ~1023);
    long long stages = ((long long)CV_SMEM_BUDGET - (long long)conv_aux_bytes(p) - (long long)out_bytes - 1024) / (long long)stage_bytes;
    if (p.out_pw && stages < 4) { // a long reduction needs the deep load pipeline more than the output needs staging
        p.out_pw = 0, p.out_mask = 0, out_bytes = 0;
        stages = ((long long)CV_SMEM_BUDGET - (long long)conv_aux_bytes(p) - 1024) / (long long)stage_bytes;
    }
    if (stages < 2)
        return false;
    p.stages = stages > CV_MAX_STAGES ? CV_MAX_STAGES : (int)stages;
    return true;
}

// The one-patch kernel may use all of an SM's shared memory (227 KB per CTA): a resident 3x3 filter over 128 -> 128
// channels is 144 KB, and what is left decides between two and three patches in flight.
constexpr size_t PATCH_SMEM_BUDGET = 226 * 1024;

size_t patch_aux_bytes(const PatchParams &p) { return sizeof(FastParam) * (size_t)p.ncols + (2 * CV_MAX_STAGES + 2 * CV_MAX_ACC + 1) * 8 + 32 + 256; }

size_t patch_filter_bytes(const PatchParams &p) { return ((size_t)p.kh * p.kw * p.cout * p.swz_b + 1023) & ~(size_t)1023; }

int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// The MMAs of a filter row with G pixels a position (see the kernel); returns their time in cycles, 0 where the list is too long.  An MMA of N
// columns: 32 + N / 4 cycles of shared-memory reads with 128-byte rows (1.5 and 1.8 times that with 64 and 32), N / 2 of math.
double patch_steps(PatchParams &p)
{
    const double narrow = p.a_row == 128 ? 1.0 : (p.a_row == 64 ? 1.5 : 1.8);
    double cycles = 0;
    p.nfirst = p.nrest = 0;
    unsigned covered = 0;
    auto add = [&](PatchStep *list, int &count, int i, int lo, int hi, bool start) {
        if (count == PATCH_MAX_STEPS)
            return false;
        const int q = floor_div(i, p.G), pixel = i - q * p.G, slot = p.kw - 1 - (i + p.pl - lo), n = (hi - lo + 1) * p.cout;
        PatchStep &t = list[count++];
        const int per_row = p.a_row / p.cin, at = (pixel / per_row * p.plane_bytes + pixel % per_row * p.cin + (q - p.glo) * p.a_row) / 16;
        t.ab = (uint32_t)at | (uint32_t)(slot * p.cout * p.swz_b / 16) << 16;
        t.dn = (uint32_t)(lo * p.cout) | (start ? 0x8000u : 0u) | (uint32_t)n << 16;
        return true;
    };
    auto range = [&](int i, int &lo, int &hi) { lo = max(0, i + p.pl - p.kw + 1), hi = min(p.G - 1, i + p.pl); };
    for (int width = p.G; width > 0; width--) // widest first: fewest pieces that start accumulator columns
        for (int i = -p.pl; i <= p.G + p.kw - 2 - p.pl; i++) {
            int lo, hi;
            range(i, lo, hi);
            if (hi - lo + 1 != width)
                continue;
            cycles += p.cin / 32 * (max(width * p.cout / 2.0, narrow * (32 + width * p.cout / 4.0)) + 4);
            if (!add(p.rest, p.nrest, i, lo, hi, false))
                return 0;
            for (int from = lo; from <= hi;) {
                const bool start = !(covered >> from & 1);
                int to = from;
                while (to < hi && !(covered >> (to + 1) & 1) == start) to++;
                if (!add(p.first, p.nfirst, i, from, to, start))
                    return 0;
                for (int j = from; j <= to; j++) covered |= 1u << j;
                from = to + 1;
            }
        }
    return cycles;
}

// The one-patch form: stride 1, dilation 1, Cin = 32, 64 or 128 (one swizzle row per pixel), Cout <= 256 in one tile, the
// filter small enough to stay in shared memory next to two or more patches, and the staged epilogue's alignment.
bool patch_plan(const espdl_conv_desc &d, PatchParams &best)
{
    if (getenv("ESPDL_B200_NO_CONV_PATCH"))
        return false;
    if (d.stride_h != 1 || d.stride_w != 1 || d.dilation_h != 1 || d.dilation_w != 1 || (d.in_c != 32 && d.in_c != 64 && d.in_c != 128))
        return false;
    if (d.out_c > 256 || d.out_c % 16 != 0 || d.kw > 8 || d.kh > 8 || d.kh * d.kw < 2)
        return false;
    const long long ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c, ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    if (ops % 16 != 0 || ((uintptr_t)d.output % 16) != 0)
        return false;
    const bool single = getenv("ESPDL_B200_NO_TAP_STACK") != nullptr; // one pixel a position
    PatchParams p;
    p.n = d.n, p.oh = d.out_h, p.ow = d.out_w, p.cin = d.in_c, p.cout = d.out_c;
    p.kh = d.kh, p.kw = d.kw, p.pt = d.pad_top, p.pl = d.pad_left;
    double least = -1;
    for (int G : {1, 2, 4}) {
        if (G > 1 && (single || d.in_w % G || d.out_w % G || G * d.out_c > 256))
            break;
        p.G = G, p.ncols = G * d.out_c;
        p.a_row = ips == d.in_c ? min(128, G * d.in_c) : d.in_c;
        p.planes = G * d.in_c / p.a_row;
        p.acc_stages = 4 * p.ncols <= 512 ? 4 : 2;
        const int parts = 4 / p.acc_stages;
        if (p.ncols % (16 * parts) != 0 || p.ncols / parts > 128)
            continue;
        p.tmem_cols = 32;
        while (p.tmem_cols < p.acc_stages * p.ncols) p.tmem_cols *= 2;
        p.out_pw = p.ncols / parts;
        p.dense_out = G == 1 || ops == d.out_c;
        p.out_box = p.dense_out ? p.out_pw : d.out_c;
        if (p.out_pw % p.out_box)
            continue;
        p.out_mask = p.out_box == 128 ? 7 : (p.out_box == 64 ? 3 : 0);
        p.glo = floor_div(-p.pl, G);
        const int span = floor_div(G - 1 - p.pl + p.kw - 1, G) - p.glo;
        p.plane_bytes = 0;
        const double mma = p.kh * patch_steps(p);
        if (mma == 0)
            continue;
        // positions per patch row: the narrowest that cut an image row into so many tiles.  The time of a tile is its MMAs, its loads (32 bytes
        // a cycle) or its requantisation (3.6 instructions a column and warp), whichever is longest
        const int positions = d.out_w / G, fewest = (positions + 128 - span - 1) / (128 - span);
        for (p.xtiles = fewest; p.xtiles < fewest + 6 && p.xtiles <= positions; p.xtiles++) {
            p.PV = (positions + p.xtiles - 1) / p.xtiles, p.PW = p.PV + span, p.RT = min(128 / p.PW, d.out_h);
            p.ytiles = (d.out_h + p.RT - 1) / p.RT;
            const int rows = (p.RT + p.kh - 1) * p.PW;
            // the last rows of A (dropped positions) reach past the patch
            p.plane_bytes = (max(rows, 128 + (p.kh - 1) * p.PW + span) * p.a_row + 1023) & ~1023;
            p.patch_bytes = p.planes * p.plane_bytes, p.patch_tx = p.planes * rows * p.a_row;
            const double tile = max(max(mma, p.patch_tx / 32.0), p.ncols * 3.6) + 200;
            const double waves = (double)(((long long)p.n * p.xtiles * p.ytiles + num_sms() - 1) / num_sms());
            // the first tile's way through the pipeline: the filter (below: in the wider form only where many tiles follow), its loads, its MMAs
            const double cost = waves * tile + (p.kh * p.kw * p.cout * p.cin + p.patch_tx) / 32.0 + mma;
            if (least >= 0 && cost >= least * 0.999)
                continue;
            const long long out_bytes = 4 * (long long)((128 * p.out_pw + 1023) & ~1023);
            // filter rows of 128 bytes (the bytes behind Cin are not read; a longer start, shorter MMAs), then of Cin, then without staging tiles: rows go out of registers (long
            // reductions, the epilogue is a small part)
            long long stages = 0;
            for (int form = waves < 12 ? 1 : 0; form < 3 && stages < 2; form++) {
                p.swz_b = form == 0 ? 128 : d.in_c, p.staged = form < 2;
                stages = ((long long)PATCH_SMEM_BUDGET - (long long)patch_filter_bytes(p) - (long long)patch_aux_bytes(p) - 1024 - (p.staged ? out_bytes : 0)) / p.patch_bytes;
            }
            if (stages < 2)
                continue;
            p.stages = stages > 4 ? 4 : (int)stages;
            p.issuers = p.acc_stages == 4 && p.stages == 4 ? 2 : 1; // with two of either both tiles would be multiplied, and then both be drained, at once
            best = p, least = cost;
            patch_steps(best); // the planes' distance is known now
        }
    }
    return least >= 0;
}

int launch_patch(const espdl_conv_desc &d, PatchParams &p, cudaStream_t s)
{
    EncodeTiledFn enc = conv_encode();
    if (!enc)
        return set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled entry point not found");
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    p.out = d.output;
    p.ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.epi.bias = d.bias, p.epi.ew = d.filter_exponents, p.epi.lut = d.lut, p.epi.lut_stride = d.lut_channel_stride;
    p.epi.e_shift_base = d.out_exponent - d.in_exponent;
    p.epi.ew_scalar = d.filter_exponent, p.epi.per_channel = d.per_channel;
    p.epi.relu = d.activation == ESPDL_ACT_RELU, p.epi.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    p.epi.acc_bound = min(d.in_c * d.kh * d.kw, 65536) << 14;
    const cuuint64_t G = (cuuint64_t)p.G, w = (cuuint64_t)d.in_w, ow = (cuuint64_t)d.out_w, out_stride = (cuuint64_t)p.ops, in_stride = (cuuint64_t)ips;
    CUtensorMap ma, mb, mo;
    {
        // {channels of a row of A, pixels of a position, positions of an image row, rows, images}
        cuuint64_t dims[5] = {(cuuint64_t)p.a_row, (cuuint64_t)p.planes, w / G, (cuuint64_t)d.in_h, (cuuint64_t)d.n};
        cuuint64_t strides[4] = {p.planes == p.G ? in_stride : (cuuint64_t)p.a_row, G * in_stride, w * in_stride, w * in_stride * d.in_h};
        cuuint32_t box[5] = {(cuuint32_t)p.a_row, 1, (cuuint32_t)p.PW, (cuuint32_t)(p.RT + d.kh - 1), 1};
        cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        if (enc(&ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, const_cast<void *>(d.input), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle_of(p.a_row), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled(conv patch input)");
    }
    {
        const cuuint64_t krow = (cuuint64_t)d.kh * d.kw * d.in_c;
        cuuint64_t dims[2] = {krow, (cuuint64_t)d.out_c};
        cuuint64_t strides[1] = {krow};
        cuuint32_t box[2] = {(cuuint32_t)p.swz_b, (cuuint32_t)p.cout};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(d.filter), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle_of(p.swz_b), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled(conv patch filter)");
    }
    {
        cuuint64_t dims[5] = {(cuuint64_t)(p.dense_out ? p.ncols : p.cout), p.dense_out ? 1 : G, ow / G, (cuuint64_t)d.out_h, (cuuint64_t)d.n};
        cuuint64_t strides[4] = {out_stride, G * out_stride, ow * out_stride, ow * out_stride * d.out_h};
        cuuint32_t box[5] = {(cuuint32_t)p.out_box, (cuuint32_t)(p.out_pw / p.out_box), (cuuint32_t)p.PV, (cuuint32_t)p.RT, 1};
        cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        if (enc(&mo, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, d.output, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle_of(p.out_mask ? p.out_box : 0), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled(conv patch output)");
    }
    size_t smem = 1024 + patch_filter_bytes(p) + (size_t)p.stages * p.patch_bytes +
        (p.staged ? 4 * (size_t)((128 * p.out_pw + 1023) & ~1023) : 0) + patch_aux_bytes(p);
    if (smem < 120 * 1024)
        smem = 120 * 1024;
    static std::once_flag attr_once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(attr_once, [] {
        attr_err = cudaFuncSetAttribute(conv_patch_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(PATCH_SMEM_BUDGET + 1024));
        if (attr_err == cudaSuccess)
            attr_err = cudaFuncSetAttribute(conv_patch_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(PATCH_SMEM_BUDGET + 1024));
    });
    if (attr_err != cudaSuccess)
        return set_cuda_error(attr_err, "cudaFuncSetAttribute(conv_patch_kernel)");
    const long long total = (long long)p.n * p.ytiles * p.xtiles;
    if (total > 0x7fffffffll)
        return ESPDL_ERR_TOO_LARGE;
    const auto kernel = p.epi.half_even ? conv_patch_kernel<true> : conv_patch_kernel<false>;
    launch_overlapped(kernel, dim3((int)min(total, (long long)num_sms())), dim3(PATCH_THREADS), smem, s, ma, mb, mo, p);
    count_launch();
    return check_launch("conv_patch");
}

} // namespace

bool conv2d_conv_tc_supported(const espdl_conv_desc &d)
{
    if (d.dtype != ESPDL_DTYPE_INT8 || d.group != 1 || d.n <= 0)
        return false;
    if (d.kh < 1 || d.kw < 1 || d.kh * d.kw > 49 || (d.kh == 1 && d.kw == 1 && d.stride_h == 1))
        return false; // 1x1 stride 1 is the pointwise tile kernel's
    if (d.stride_h != d.stride_w || (d.stride_h != 1 && d.stride_h != 2) || d.dilation_h != d.dilation_w || d.dilation_h < 1 || d.dilation_h > 8)
        return false;
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    if (d.in_c % 16 || ips % 16 || ((uintptr_t)d.input % 16) || ((uintptr_t)d.filter % 16) || d.out_c > 8192)
        return false;
    if (d.pad_top < 0 || d.pad_left < 0 || d.in_w > (1 << 20) || d.in_h > (1 << 20))
        return false;
    ConvTcParams p;
    return conv_plan(d, p);
}

int conv2d_conv_tc(const espdl_conv_desc &d, cudaStream_t s)
{
    ConvTcParams p;
    if (!conv2d_conv_tc_supported(d) || !conv_plan(d, p))
        return ESPDL_ERR_UNSUPPORTED;
    {
        PatchParams pp;
        memset(&pp, 0, sizeof(pp));
        pp.early = in_model_scope();
        if (patch_plan(d, pp))
            return launch_patch(d, pp, s);
    }
    EncodeTiledFn enc = conv_encode();
    if (!enc)
        return set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled entry point not found");
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    p.early = in_model_scope();
    p.out = d.output;
    p.ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.epi.bias = d.bias, p.epi.ew = d.filter_exponents, p.epi.lut = d.lut, p.epi.lut_stride = d.lut_channel_stride;
    p.epi.e_shift_base = d.out_exponent - d.in_exponent;
    p.epi.ew_scalar = d.filter_exponent, p.epi.per_channel = d.per_channel;
    p.epi.relu = d.activation == ESPDL_ACT_RELU, p.epi.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    p.epi.acc_bound = min(d.in_c * d.kh * d.kw, 65536) << 14;

    CUtensorMap ma, mb, mo;
    {
        cuuint64_t dims[4] = {(cuuint64_t)d.in_c, (cuuint64_t)d.in_w, (cuuint64_t)d.in_h, (cuuint64_t)d.n};
        cuuint64_t strides[3] = {(cuuint64_t)ips, (cuuint64_t)ips * d.in_w, (cuuint64_t)ips * d.in_w * d.in_h};
        cuuint32_t box[4] = {(cuuint32_t)p.swz, (cuuint32_t)(p.P * p.S), (cuuint32_t)(p.R * p.S), 1};
        cuuint32_t estr[4] = {1, (cuuint32_t)p.S, (cuuint32_t)p.S, 1};
        if (enc(&ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void *>(d.input), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle_of(p.swz), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled(conv input)");
    }
    {
        const cuuint64_t krow = (cuuint64_t)d.kh * d.kw * d.in_c;
        cuuint64_t dims[2] = {krow, (cuuint64_t)d.out_c};
        cuuint64_t strides[1] = {krow};
        cuuint32_t box[2] = {(cuuint32_t)p.swz, (cuuint32_t)p.block_n};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(d.filter), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle_of(p.swz), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled(conv filter)");
    }
    mo = ma;
    if (p.out_pw) {
        cuuint64_t dims[4] = {(cuuint64_t)d.out_c, (cuuint64_t)d.out_w, (cuuint64_t)d.out_h, (cuuint64_t)d.n};
        cuuint64_t strides[3] = {(cuuint64_t)p.ops, (cuuint64_t)p.ops * d.out_w, (cuuint64_t)p.ops * d.out_w * d.out_h};
        cuuint32_t box[4] = {(cuuint32_t)p.out_pw, (cuuint32_t)p.P, (cuuint32_t)p.R, 1};
        cuuint32_t estr[4] = {1, 1, 1, 1};
        if (enc(&mo, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, d.output, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle_of(p.out_pw == 128 ? 128 : (p.out_pw == 64 ? 64 : 0)), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled(conv output)");
    }
    const size_t stage_bytes = (size_t)(128 + p.block_n) * p.swz;
    size_t smem = 1024 + (size_t)p.stages * stage_bytes + 4 * (size_t)((128 * p.out_pw + 1023) & ~1023) + conv_aux_bytes(p);
    if (smem < 120 * 1024)
        smem = 120 * 1024; // one CTA per SM, so that TMEM allocation never waits on a neighbour
    static std::once_flag attr_once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(attr_once, [] {
        attr_err = cudaFuncSetAttribute(conv_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(CV_SMEM_BUDGET + 2048));
        if (attr_err == cudaSuccess)
            attr_err = cudaFuncSetAttribute(conv_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(CV_SMEM_BUDGET + 2048));
    });
    if (attr_err != cudaSuccess)
        return set_cuda_error(attr_err, "cudaFuncSetAttribute(conv_tc_kernel)");
    const long long total = (long long)p.n * p.ytiles * p.xtiles * p.n_tiles;
    if (total > 0x7fffffffll)
        return ESPDL_ERR_TOO_LARGE;
    const int grid = (int)min(total, (long long)num_sms());
    const auto kernel = p.epi.half_even ? conv_tc_kernel<true> : conv_tc_kernel<false>;
    launch_overlapped(kernel, dim3(grid), dim3(CV_THREADS), smem, s, ma, mb, mo, p);
    count_launch();
    return check_launch("conv_tc");
}

} // namespace espdl
