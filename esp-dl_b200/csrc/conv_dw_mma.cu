// 3x3 DepthwiseConv2D, int8, stride 1, on the warp-level matrix instruction, fed by TMA: large NHWC tensors whose channel count is a multiple of 16 (which of them: dwm_pays).
// Replaces dl::base::depthwise_conv2d<int8_t,...> (esp-dl/dl/base/dl_base_depthwise_conv2d.cpp:47-66, shell
// esp-dl/dl/base/dl_base.hpp:1209-2107): out[y,x,c] = sat8(act(rnd((sum_{ky,kx} in[y+ky-pt, x+kx-pl, c] * w[ky,kx,c] + bias[c]) >> shift[c]))),
// taps outside the image contribute nothing.
//
// The op moves two bytes per output and needs nine MACs for them: it is bound by HBM if and only if the arithmetic keeps
// up.  On dp4a (dw3x3_dp4a_kernel, conv_dw.cu) it takes eleven instructions per output, because the four bytes of an operand have to be
// taps of one channel and NHWC bytes are channels.  The warp-level matrix instruction takes the bytes as they lie: in mma.sync m16n8k32 a
// column of B is a position, its 32 bytes four neighbouring pixels of eight channels (a lane's 16-byte load is the operand of
// two instructions, no byte is moved), and a row of A one output whose weights stand at the bytes of its own channel, zero elsewhere.  Nine tenths of
// the products are with zeros, but an SM finishes 128 outputs in three instructions of two cycles each, 21 outputs a cycle where HBM
// delivers for twelve, and a thread issues seven instructions per output.  (With positions as rows of A every operand had to be put together from
// two loads' registers: sixteen.)
// A position is two neighbouring output pixels (input pixels 2p .. 2p + 3), the 16 rows are 2 pixels x 8 channels.  At stride 2 the four pixels are one
// output's, half the rows stay empty and nothing is gained over dp4a (56x56x144: 128 us, 104 there; 112x112x96 266 / 254), which keeps it.
// A warp walks down its band an input row a step: the row goes into the sums of the three output rows that read it, which are independent
// instructions, and completes the first of them.
// Sums start from the bias and the rounding's half; results become pixels of 16 channels by a transposing stmatrix.
// One persistent CTA per SM splits the roles:
//   last warp   producer: one TMA box per tile brings the input patch (NB images x IH rows x IW columns x CB
//               channels, zero-filled outside the image, so padding needs no code) into a ring of shared-memory stages, and one stores each finished
//               output tile (clipped at the image border, so ragged tiles need no code either).  A load takes some 4500 cycles,
//               longer than a tile, so there is one in flight beside those being computed at the least.  Rows whose pixels lie side by side in memory
//               (all channels in the block) move as runs of whole rows: the unit takes 3.5 cycles for a run, whatever its length;
//   the others  consumers, in teams that take the tiles in turn: a warp owns 16 channels and walks groups of 8 positions down a band of rows, writing the
//               requantised words into an output tile in shared memory.
// Bound by the latency of a warp's walk, some 260 cycles a row with three or four warps a scheduler (1024 of 28x28x192: matrix pipe 43 %, issue slots 45 % busy); loads and
// stores alone run at the copy bandwidth.  1024 images, dp4a before and now, us: 112x112x32 207 -> 165, 28x28x192 83 -> 75, 14x14x384 54 -> 41,
// 14x14x576 75 -> 60, 7x7x960 44 -> 30.  Where tiles' channel blocks share lines of memory they follow one another (fetched twice otherwise: 28x28x192
// could not be below 78), and with two stages a tile waited half its time for its load.
// A fragment load is 16 bytes of 6 pixels to a quarter warp: without bank conflicts where CB / 16 is odd, two-way for 32 and 96,
// and never a multiple of 128 (dwm_search).
// Every mbarrier wait is bounded; a wait that expires records ESPDL_ERR_TIMEOUT and raises a CTA-wide flag, every role leaves at the flag or at its own
// limit, and the producer waits for the copies in flight.
#include "dw_mma_plan.cuh"
#include "tc_common.cuh"

#include <climits>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>

namespace espdl {

__device__ int *g_dwm_error = nullptr; // the status word of bounded waits (common.cuh)

int bind_device_error_dw_mma(int *word)
{
    ESPDL_CUDA_TRY(cudaMemcpyToSymbol(g_dwm_error, &word, sizeof(word)));
    return ESPDL_OK;
}

namespace {

using namespace tc;

__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, uint32_t src, int c0, int c1, int c2, int c3)
{
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map), "r"(src), "r"(c0), "r"(c1),
                 "r"(c2), "r"(c3)
                 : "memory");
}

__device__ __forceinline__ void mma_s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const int (&c)[4])
{
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}

enum class DwmForm { Linear, Relu, General }; // of the requantisation: one-add-one-shift without and with ReLU, or any

// What a lane (g, t) keeps of its 16 channels: fragments of A for both pairs of words of a load, constants of the channels whose sums
// it receives.  Rows g and g + 8 are neighbouring channels of one pixel: channels 2 (g & 3) and the next of a pair's eight, of pixel g / 4.
struct DwmConsts {
    static constexpr int QUADS = 2; // results: two channels of two positions each
    uint32_t a[3][2][4];
    int start[QUADS][4], shift[QUADS][2];
    DwmForm form;
};

// Channel of row g + 8h of an accumulator, from the block's first.
__device__ __forceinline__ int dwm_channel(int g, int quad, int h) { return 8 * quad + 2 * (g & 3) + h; }

template <bool EVEN>
__device__ __forceinline__ void dwm_load_consts(DwmConsts &k, const DwmSource &p, int c0, int g, int t)
{
    const int kx = t - (g >> 2);
#pragma unroll
    for (int ky = 0; ky < 3; ky++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const bool mine = kx >= 0 && kx < 3, second = g & 2;
            const uint32_t f = mine ? __ldg((const uint32_t *)(p.w + (long long)(ky * 3 + kx) * p.C + c0 + 8 * j + (second ? 4 : 0))) : 0u;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t v = f & (0xffu << (8 * (2 * (g & 1) + h)));
                k.a[ky][j][h] = second ? 0u : v, k.a[ky][j][2 + h] = second ? v : 0u;
            }
        }
    bool fast = true;
#pragma unroll
    for (int q = 0; q < DwmConsts::QUADS; q++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int c = c0 + dwm_channel(g, q, h);
            int start, shift;
            fast = fast_constants(p.bias ? __ldg(p.bias + c) : 0, p.e_shift_base - (p.per_channel ? __ldg(p.ew + c) : p.ew_scalar), 9 << 14, EVEN, start, shift) && fast;
            k.start[q][2 * h] = k.start[q][2 * h + 1] = start;
            k.shift[q][h] = shift - (p.relu && !EVEN ? 1 : 0); // what dwm_pack shifts by
        }
    k.form = !__all_sync(0xffffffffu, fast) ? DwmForm::General : (p.relu ? DwmForm::Relu : DwmForm::Linear);
}

// A lane's share of a group with channels outside the one-add-one-shift form (a shift below 1, a huge bias): `pixels` output pixels of its position, four channels from `c` on, `rows` rows, by plain loops and the general requantisation.
__device__ __noinline__ void dwm_walk_general(const DwmSource &p, const int8_t *ip, int8_t *op, int in_row, int out_row, int CB, int rows, int pixels, int c)
{
    for (int y = 0; y < rows; y++)
        for (int x = 0; x < pixels; x++)
            for (int i = 0; i < 4; i++) {
                int32_t acc = 0;
                for (int ky = 0; ky < 3; ky++)
                    for (int kx = 0; kx < 3; kx++) acc += (int)ip[(y + ky) * in_row + (x + kx) * CB + i] * (int)p.w[(ky * 3 + kx) * p.C + c + i];
                const int shift = max(-31, min(32, p.e_shift_base - (p.per_channel ? p.ew[c + i] : p.ew_scalar)));
                op[y * out_row + x * CB + i] = (int8_t)requant8(acc, p.bias ? p.bias[c + i] : 0, shift, p.relu, p.half_even);
            }
}

// Two channels of two positions: bytes (position, channel).
template <bool EVEN, bool RELU>
__device__ __forceinline__ uint32_t dwm_pack(const int (&acc)[4], const int (&shift)[2])
{
    int q[4];
    uint32_t hi, w;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int s = shift[i >> 1], v = EVEN && RELU ? max(acc[i], 0) : acc[i];
        // half to even: acc + bias + 2^(s-1) - 1 = v, quotient (v + bit s of v) >> s (derived beside shift_fast in tc_common.cuh)
        q[i] = EVEN ? (v + ((v >> s) & 1)) >> s : v >> s;
    }
    if constexpr (RELU && !EVEN) {
        // The staged shifts are one less than the real ones; packing with saturation to [0, 255] clamps below at zero, halving every byte
        // completes the shift and turns the upper clamp into 127 - a shift and a mask per word instead of a max per output.
        asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(q[3]), "r"(q[1]));
        asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q[2]), "r"(q[0]), "r"(hi));
        return (w >> 1) & 0x7f7f7f7fu;
    }
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(q[3]), "r"(q[1]));
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q[2]), "r"(q[0]), "r"(hi));
    return w;
}

// An output row's sums, requantised and stored: `at` is where the lane's row of the store goes (a position's 16 channels).
template <bool EVEN, bool RELU>
__device__ __forceinline__ void dwm_store(const int (&acc)[2][4], const DwmConsts &k, uint32_t at, int g)
{
    const uint32_t w0 = dwm_pack<EVEN, RELU>(acc[0], k.shift[0]), w1 = dwm_pack<EVEN, RELU>(acc[1], k.shift[1]);
    // lanes of pixel 0 have all of its channels, lanes of pixel 1 theirs: after the exchange either half has eight channels of both
    const bool first = g < 4;
    const uint32_t got = __shfl_xor_sync(0xffffffffu, first ? w1 : w0, 16);
    asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1, %2};" ::"r"(at), "r"(first ? w0 : got), "r"(first ? got : w1) : "memory");
}

// One filter row's products with one input row.
__device__ __forceinline__ void dwm_row(int (&acc)[2][4], const DwmConsts &k, int ky, const uint4 &r)
{
    mma_s8(acc[0], k.a[ky][0], r.x, r.y, acc[0]);
    mma_s8(acc[1], k.a[ky][1], r.z, r.w, acc[1]);
}

__device__ __forceinline__ void dwm_first_row(int (&acc)[2][4], const DwmConsts &k, const uint4 &r)
{
    mma_s8(acc[0], k.a[0][0], r.x, r.y, k.start[0]);
    mma_s8(acc[1], k.a[0][1], r.z, r.w, k.start[1]);
}

// A group's walk down its band: `rows` output rows from the lane's load address `in`, to its store address `out`.  The loop has no test within a
// turn of the accumulators, so the last row's products for rows beyond the band and one load (in shared memory still, see dwm_shape) are made for nothing.
template <bool EVEN, bool RELU>
__device__ __forceinline__ void dwm_walk(const DwmConsts &k, uint32_t in, uint32_t out, int in_row, int out_row, int rows, int g)
{
    auto load = [&](uint4 &r) {
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(in) : "memory");
        in += (uint32_t)in_row;
    };
    auto store = [&](const int(&acc)[2][4]) {
        dwm_store<EVEN, RELU>(acc, k, out, g);
        out += (uint32_t)out_row;
    };
    int a[2][4], b[2][4], c[2][4];
    uint4 r, r1;
    load(r);
    load(r1);
    dwm_first_row(a, k, r);
    load(r);
    dwm_row(a, k, 1, r1);
    dwm_first_row(b, k, r1);
    // `done` gets its last row, `half` its second, `fresh` its first; the next row arrives while the sums are requantised
    auto step = [&](int(&done)[2][4], int(&half)[2][4], int(&fresh)[2][4]) {
        dwm_row(done, k, 2, r);
        dwm_row(half, k, 1, r);
        dwm_first_row(fresh, k, r);
        load(r);
        store(done);
    };
    int left = rows;
    for (; left >= 3; left -= 3) {
        step(a, b, c);
        step(b, c, a);
        step(c, a, b);
    }
    if (left > 0) {
        dwm_row(a, k, 2, r);
        dwm_row(b, k, 1, r);
        load(r);
        store(a);
    }
    if (left > 1) {
        dwm_row(b, k, 2, r);
        store(b);
    }
}

template <bool EVEN>
__global__ void __launch_bounds__(DWM_MAX_THREADS, 1)
dw3x3_mma_kernel(const __grid_constant__ CUtensorMap map_in, const __grid_constant__ CUtensorMap map_out, const __grid_constant__ DwmParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // 128-byte aligned start, found by offset so that every pointer below is still known to be shared memory
    uint8_t *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    const int NS = p.stages, NO = 2 * p.teams;
    uint8_t *patch0 = smem, *out0 = patch0 + (size_t)NS * p.stage_bytes;
    uint64_t *bars = (uint64_t *)(out0 + (size_t)NO * p.out_bytes);
    // a patch is there; all of a team have computed their part of an output tile; it has left
    uint64_t *full_bar = bars, *done_bar = full_bar + DWM_MAX_STAGES, *free_bar = done_bar + 2 * DWM_MAX_TEAMS;
    volatile int *abort_flag = (volatile int *)(free_bar + 2 * DWM_MAX_TEAMS);
    volatile int *block_ring = abort_flag + 1; // DWM_RING tiles' channel blocks, -1 behind the last, producer -> consumers (published by the "full" arrive)
    volatile int *tile_ring = block_ring + DWM_RING; // and their numbers, for the producer's stores
    int2 *position = (int2 *)((uint8_t *)bars + DWM_BARRIER_BYTES); // of every position: bytes into the patch, and into the output tile (-1: padding, odd: one pixel)
    uint8_t *nowhere = out0 + (size_t)NO * p.out_bytes - 16; // results of padding

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31; // the same for all of a warp, as the compiler can see
    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; s++) mbar_init(smem_u32(&full_bar[s]), 1);
        for (int s = 0; s < NO; s++) {
            mbar_init(smem_u32(&done_bar[s]), p.nw);
            mbar_init(smem_u32(&free_bar[s]), 1);
        }
        *abort_flag = 0;
        for (int i = 0; i < DWM_RING; i++) block_ring[i] = 0; // never negative before the producer says so
        fence_barrier_init();
    }
    if (threadIdx.x == 32) {
        prefetch_tensormap(&map_in);
        prefetch_tensormap(&map_out);
    }
    for (int q = threadIdx.x; q < 8 * p.groups; q += blockDim.x) {
        const int row = q / p.PX, px = q - row * p.PX, nb = row / p.nbands, band = row - nb * p.nbands;
        const bool real = q < p.Q;
        position[q] = make_int2(real ? ((nb * p.IH + band * p.RB) * p.IW + 2 * px) * p.CB : 0,
                                real ? ((nb * p.TH + band * p.RB) * p.TW + 2 * px) * p.CB + (2 * px + 1 >= p.TW ? 1 : 0) : -1);
    }
    __syncthreads();
    const int CB = p.CB;
    if (threadIdx.x == 0)
        grid_dep_launch(); // set up: the next kernel's CTAs may take SMs as they become free

    if (warp == p.nw * p.teams) {
        grid_dep_wait(); // the previous kernel's output (and its use of the tile counter) before the first load
        // ------------------------------------------------------------ producer: the warp walks the tiles, lane 0 issues
        // Tiles below p.static_tiles go round the CTAs in the fixed order; the rest is handed out by a global counter, one
        // number per tile and asked for one tile ahead, so that an SM that runs slower than the others ends with fewer tiles.
        bool handed = false, ok = true;
        auto after = [&](int cur) {
            if (!handed && cur + (int)gridDim.x < p.static_tiles)
                return cur + (int)gridDim.x;
            if (!p.sched)
                return handed || cur + (int)gridDim.x >= p.total_tiles ? p.total_tiles : cur + (int)gridDim.x;
            handed = true;
            int v = 0;
            if (lane == 0)
                v = p.static_tiles + (int)atomicAdd(p.sched, 1u);
            return __shfl_sync(0xffffffffu, v, 0);
        };
        struct Place {
            int cb, x, y, n;
        };
        auto place = [&](int t) {
            const int t_in_cb = t / p.cblocks, xt = t_in_cb % p.xtiles, r = t_in_cb / p.xtiles;
            return Place{t - t_in_cb * p.cblocks, xt * p.TW, r % p.ytiles * p.TH, r / p.ytiles * p.NB};
        };
        int next = blockIdx.x, loaded = 0, ends = 0;
        Place next_at = place(next);
        auto load = [&](int i) { // the next tile as the CTA's i-th, or word to a team that there is none
            const int s = i % NS;
            const bool more = next < p.total_tiles;
            if (elect_one()) {
                const uint32_t bar = smem_u32(&full_bar[s]), to = smem_u32(patch0 + (size_t)s * p.stage_bytes);
                block_ring[i & (DWM_RING - 1)] = more ? next_at.cb : -1, tile_ring[i & (DWM_RING - 1)] = next;
                if (more) {
                    mbar_arrive_expect_tx(bar, (uint32_t)p.tx_bytes);
                    if (p.flat)
                        tma_load_3d(to, &map_in, (next_at.x - p.pl) * (CB / 8), next_at.y - p.pt, next_at.n, bar);
                    else
                        tma_load_4d(to, &map_in, next_at.cb * CB, next_at.x - p.pl, next_at.y - p.pt, next_at.n, bar);
                } else {
                    mbar_arrive(bar);
                }
            }
            __syncwarp();
            loaded += more, ends += !more;
        };
        auto advance = [&] {
            if (next < p.total_tiles) {
                next = after(next);
                next_at = place(next);
            }
        };
        for (int i = 0; i < NS && ends < p.teams; i++) {
            load(i);
            advance();
        }
        int i = 0;
        for (; i < loaded; i++) {
            const int s = i % NO;
            const Place at = place(tile_ring[i & (DWM_RING - 1)]);
            if (i > 0 && elect_one()) { // the same lane each time: a thread waits for its own stores
                bulk_wait_read_all();
                mbar_arrive(smem_u32(&free_bar[(i - 1) % NO]));
            }
            __syncwarp();
            ok = !*abort_flag && mbar_wait(smem_u32(&done_bar[s]), (i / NO) & 1, p.wait_limit);
            if (!ok) {
                *abort_flag = 1;
                if (lane == 0)
                    report_timeout(g_dwm_error);
                break;
            }
            if (elect_one()) { // the store ahead of the next load: the unit takes them in order
                const uint32_t from = smem_u32(out0 + (size_t)s * p.out_bytes);
                if (p.flat)
                    tma_store_3d(&map_out, from, at.x * (CB / 8), at.y, at.n);
                else
                    tma_store_4d(&map_out, from, at.cb * CB, at.x, at.y, at.n);
                bulk_commit();
            }
            __syncwarp();
            if (ends < p.teams)
                load(i + NS);
            advance();
        }
        if (!ok) // the loads on their way land before shared memory is given back
            for (; i < loaded; i++) mbar_wait(smem_u32(&full_bar[i % NS]), (i / NS) & 1, p.wait_limit);
        if (elect_one())
            bulk_wait_all(); // shared memory stays allocated until the last store has left it
        __syncwarp();
        if (p.sched && lane == 0) {
            // the last CTA's producer leaves the counters as it found them (it is also the thread that asked for tiles)
            __threadfence();
            if (atomicAdd(p.sched + 1, 1u) == gridDim.x - 1) {
                p.sched[0] = 0;
                p.sched[1] = 0;
            }
        }
        __syncwarp();
        return;
    }

    // ---------------------------------------------------------------- consumers
    // A warp goes through its team's tiles at its own pace.
    const int g = lane >> 2, t4 = lane & 3;
    const int team = warp / p.nw, member = warp - team * p.nw, cb16 = member % p.ncb, sub = member / p.ncb;
    const int in_row = p.IW * CB, out_row = p.TW * CB;
    const int in_lane = t4 * CB + 16 * cb16; // a lane's bytes within the position it loads
    const int pixel = (lane >> 3) & 1;          // of the position whose row it addresses in a store

    DwmConsts k;
    int have_cb = -1;
    for (int i = team;; i += p.teams) {
        const int s = i % NS, o = i % NO;
        // The output tile first: tile i - NO has left it, so the producer has seen the end of every tile up to that one, tile i - NS among them
        // (NS >= NO), and the stage's barrier is at most one phase behind.  The other way round, a load of another team's tile i - NS still on its
        // way would leave the parity as it is after tile i.
        if (!mbar_wait(smem_u32(&free_bar[o]), (i / NO & 1) ^ 1, p.wait_limit) || !mbar_wait(smem_u32(&full_bar[s]), (i / NS) & 1, p.wait_limit)) {
            *abort_flag = 1; // the tile before never left, or the patch never came
            if (lane == 0)
                report_timeout(g_dwm_error);
        }
        const int cb = block_ring[i & (DWM_RING - 1)];
        if (*abort_flag || cb < 0)
            break;
        const int c0 = cb * CB + 16 * cb16;
        if (cb != have_cb) {
            dwm_load_consts<EVEN>(k, p.src, c0, g, t4);
            have_cb = cb;
        }
        const uint32_t patch = smem_u32(patch0 + (size_t)s * p.stage_bytes), obuf = smem_u32(out0 + (size_t)o * p.out_bytes);
        for (int grp = sub; grp < p.groups; grp += p.wpc) {
            const int from = position[8 * grp + g].x, to = position[8 * grp + (lane & 7)].y;
            const bool real = to >= 0 && !((to & 1) && pixel);
            const uint32_t in = patch + (uint32_t)(from + in_lane), out = real ? obuf + (uint32_t)((to & ~1) + pixel * CB + 16 * cb16) : smem_u32(nowhere);
            const int step = real ? out_row : 0;
            if (k.form == DwmForm::Relu) {
                dwm_walk<EVEN, true>(k, in, out, in_row, step, p.RB, g);
            } else if (k.form == DwmForm::Linear) {
                dwm_walk<EVEN, false>(k, in, out, in_row, step, p.RB, g);
            } else if (const int own = position[8 * grp + g].y; own >= 0) {
                const int ch = 16 * cb16 + 4 * t4;
                dwm_walk_general(p.src, (const int8_t *)patch0 + (size_t)s * p.stage_bytes + from + ch, (int8_t *)out0 + (size_t)o * p.out_bytes + (own & ~1) + ch,
                                 in_row, out_row, CB, p.RB, own & 1 ? 1 : 2, cb * CB + ch);
            }
        }
        fence_async_smem(); // the output words are visible to the TMA unit
        __syncwarp();
        if (lane == 0 && !(p.withhold_arrive && warp == 0))
            mbar_arrive(smem_u32(&done_bar[o]));
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn dwm_encode()
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

bool dwm_flat(const espdl_conv_desc &d)
{
    return (d.in_pixel_stride == 0 || d.in_pixel_stride == d.in_c) && (d.out_pixel_stride == 0 || d.out_pixel_stride == d.out_c);
}

// The plan of a layer (dwm_search), kept for the calls that follow.
bool dwm_plan(const espdl_conv_desc &d, DwmParams &p)
{
    static std::mutex mu;
    static std::map<std::tuple<int, int, int, int, bool>, DwmParams> memo;
    const bool dense = dwm_flat(d);
    const auto key = std::make_tuple(d.in_c, d.out_h, d.out_w, d.n, dense);
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = memo.find(key);
        if (it != memo.end()) {
            p = it->second;
            return p.nw > 0;
        }
    }
    p = dwm_search(d.in_c, d.out_h, d.out_w, d.n, dense, num_sms());
    {
        std::lock_guard<std::mutex> lock(mu);
        if (memo.size() >= 4096)
            memo.clear();
        memo[key] = p;
    }
    return p.nw > 0;
}

int dwm_launch(const CUtensorMap &mi, const CUtensorMap &mo, const DwmParams &p, size_t smem, int grid, cudaStream_t s)
{
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] {
        attr_err = cudaFuncSetAttribute(dw3x3_mma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DWM_SMEM_BUDGET);
        if (attr_err == cudaSuccess)
            attr_err = cudaFuncSetAttribute(dw3x3_mma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DWM_SMEM_BUDGET);
    });
    if (attr_err != cudaSuccess)
        return set_cuda_error(attr_err, "cudaFuncSetAttribute(dw3x3_mma_kernel)");
    launch_overlapped(p.src.half_even ? dw3x3_mma_kernel<true> : dw3x3_mma_kernel<false>, dim3(grid), dim3((p.nw * p.teams + 1) * 32), smem, s, mi, mo, p);
    count_launch();
    return check_launch("dw3x3_mma");
}

} // namespace

bool conv2d_dw_mma_supported(const espdl_conv_desc &d)
{
    if (d.dtype != ESPDL_DTYPE_INT8 || d.group == 1 || d.kh != 3 || d.kw != 3 || d.dilation_h != 1 || d.dilation_w != 1)
        return false;
    if (d.stride_h != 1 || d.stride_w != 1 || d.lut) // a table would be the general form's, whose loops have more threads on dp4a
        return false;
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c, ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    if (d.in_c % 16 || ips % 16 || ops % 16 || ((uintptr_t)d.input % 16) || ((uintptr_t)d.output % 16) || ((uintptr_t)d.filter % 4))
        return false;
    if (d.pad_top > 255 || d.pad_left > 255)
        return false;
    DwmParams p;
    return dwm_plan(d, p);
}

bool conv2d_dw_mma_pays(const espdl_conv_desc &d)
{
    // the size before the search for a plan
    if (!dwm_large(d.in_c, (long long)d.n * d.out_h * d.out_w * d.in_c) || !conv2d_dw_mma_supported(d))
        return false;
    DwmParams p;
    auto pays = [&](bool whole) { return dwm_pays(p, d.in_c, d.out_h, d.out_w, d.n, d.round_mode == ESPDL_ROUND_HALF_EVEN, whole, num_sms()); };
    return dwm_plan(d, p) && (pays(true) || (pays(false) && !conv2d_dw_tma_whole(d))); // dp4a's plan only where it decides
}

int conv2d_dw_mma(const espdl_conv_desc &d, cudaStream_t s)
{
    DwmParams p;
    if (!conv2d_dw_mma_supported(d) || !dwm_plan(d, p))
        return ESPDL_ERR_UNSUPPORTED;
    EncodeTiledFn enc = dwm_encode();
    if (!enc)
        return set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled entry point not found");
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c, ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.pt = d.pad_top, p.pl = d.pad_left;
    // ESPDL_B200_DEBUG_WAIT_EXPIRY=<milliseconds> (with ESPDL_B200_DW_MMA=always), the test of the bounded waits: one arrival is withheld and the limit that
    // short, so the producer's wait runs out and every role leaves; espdl_b200_stream_sync then reports ESPDL_ERR_TIMEOUT.
    const char *expiry = getenv("ESPDL_B200_DEBUG_WAIT_EXPIRY");
    p.withhold_arrive = expiry && atoi(expiry) > 0 ? 1 : 0;
    p.wait_limit = p.withhold_arrive ? (long long)atoi(expiry) * 2000000ll : WAIT_LIMIT_CYCLES;
    p.src.C = d.in_c;
    p.src.w = (const int8_t *)d.filter, p.src.bias = (const int32_t *)d.bias, p.src.ew = d.filter_exponents;
    p.src.e_shift_base = d.out_exponent - d.in_exponent;
    p.src.ew_scalar = d.filter_exponent, p.src.per_channel = d.per_channel;
    p.src.relu = d.activation == ESPDL_ACT_RELU, p.src.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    // A map of {channels, width, height, images}, or of {bytes of a row as 8-byte words, height, images}
    auto encode = [&](CUtensorMap *m, void *base, int w, int h, int stride, int box_w, int box_h) {
        const cuuint64_t row = (cuuint64_t)stride * w, dims4[4] = {(cuuint64_t)d.in_c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)d.n}, strides4[3] = {(cuuint64_t)stride, row, row * h};
        const cuuint64_t dims3[3] = {row / 8, (cuuint64_t)h, (cuuint64_t)d.n}, strides3[2] = {row, row * h};
        const cuuint32_t box4[4] = {(cuuint32_t)p.CB, (cuuint32_t)box_w, (cuuint32_t)box_h, (cuuint32_t)p.NB}, box3[3] = {(cuuint32_t)(box_w * p.CB / 8), (cuuint32_t)box_h, (cuuint32_t)p.NB};
        const cuuint32_t ones[4] = {1, 1, 1, 1};
        return enc(m, p.flat ? CU_TENSOR_MAP_DATA_TYPE_INT64 : CU_TENSOR_MAP_DATA_TYPE_UINT8, p.flat ? 3 : 4, base, p.flat ? dims3 : dims4, p.flat ? strides3 : strides4,
                   p.flat ? box3 : box4, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    CUtensorMap mi, mo;
    if (!encode(&mi, const_cast<void *>(d.input), d.in_w, d.in_h, ips, p.IW, p.IH) || !encode(&mo, d.output, d.out_w, d.out_h, ops, p.TW, p.TH))
        return set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled(depthwise)");
    const size_t smem = dwm_smem_bytes(p);
    const int grid = dwm_grid(p, num_sms());
    // three quarters of the tiles in the fixed order, the last quarter to whichever SM is free; with several channel blocks a tile handed out would mostly be
    // another block's, whose constants take longer to load than the slow SMs lose (7x7x960 32.8 us, 29.9 in the fixed order)
    p.sched = p.total_tiles >= 4 * grid && p.cblocks == 1 ? sched_counters(s) : nullptr;
    p.static_tiles = p.sched ? (int)((long long)p.total_tiles * 3 / 4 / grid) * grid : p.total_tiles;
    return dwm_launch(mi, mo, p, smem, grid, s);
}

} // namespace espdl
