// How dw3x3_mma_kernel (conv_dw_mma.cu) cuts a layer into tiles, teams of warps and stages of its ring.  Plain C++.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>

namespace espdl {

constexpr int DWM_MAX_CONSUMER_WARPS = 15; // with the producer's four warps a scheduler: 128 registers
constexpr int DWM_MAX_THREADS = (DWM_MAX_CONSUMER_WARPS + 1) * 32;
constexpr int DWM_MAX_STAGES = 8, DWM_MAX_TEAMS = 7;
constexpr int DWM_RING = 16; // tile numbers on their way from the producer to the consumers (more than stages and teams together)
constexpr int DWM_BARRIER_BYTES = 8 * (DWM_MAX_STAGES + 4 * DWM_MAX_TEAMS) + 4 + 8 * DWM_RING + 12;
constexpr int DWM_POSITION_BYTES = 8; // an entry of the table of positions
constexpr size_t DWM_SMEM_BUDGET = 220 * 1024;

// Where the filter and the requantisation constants come from.
struct DwmSource {
    const int8_t *w;          // [3][3][C]
    const int32_t *bias, *ew; // int32[C] or null
    int C, e_shift_base, ew_scalar, per_channel, relu, half_even;
};

struct DwmParams {
    int CB, NB, TH, TW, IH, IW;
    int RB, nbands, PX, Q, groups; // rows of a band; positions of a row, of a tile, and in eights
    int ncb, wpc, nw;              // 16-channel blocks, warps of each, warps of a team
    int teams, stages;             // consumer teams, each with two output tiles; patches in the ring, two a team at the least (dwm_shape)
    int flat;                      // rows of the tensors are runs of bytes without gaps
    int cblocks, nblocks, ytiles, xtiles, total_tiles; // tiles of neighbouring channel blocks, which share lines of memory, follow one another
    int pt, pl;
    int stage_bytes, out_bytes, tx_bytes; // patch stride in the ring, output tile size, bytes one patch load delivers
    unsigned *sched;                      // {next tile, CTAs done}: the tiles from static_tiles on are handed out by this counter; null = fixed walk
    int static_tiles;                     // tiles walked in the fixed order (a multiple of the grid size)
    long long wait_limit;                 // cycles a wait may take (WAIT_LIMIT_CYCLES; shorter only in the expiry test)
    int withhold_arrive;                  // expiry test: consumer warp 0 never reports its part of a tile, so the producer's wait runs out
    DwmSource src;
};

inline size_t dwm_smem_bytes(const DwmParams &p)
{
    return 128 + (size_t)p.stages * p.stage_bytes + 2 * (size_t)p.teams * p.out_bytes + DWM_BARRIER_BYTES + (size_t)p.groups * 8 * DWM_POSITION_BYTES;
}

// The plan of a tile shape: warps, teams, stages; its time per tile and SM in cycles, 0 if it does not fit.  A tile takes as long as the
// slowest of: the consumers' instructions (56 a row and group, 2.4 a cycle and SM over all warps), one team's walk over the teams (230 cycles a row),
// the matrix instructions (one per two cycles), the bytes (22 a cycle and SM, halos at half: neighbours' come from L2), the TMA unit's runs
// (3.5 cycles each) and the latency of a load (4500 cycles) over the stages that no team is computing.
inline double dwm_shape(DwmParams &q, int CB, int NB, int TW, int RB, int nbands, bool flat)
{
    q.CB = CB, q.NB = NB, q.TW = TW, q.RB = RB, q.nbands = nbands, q.flat = flat;
    q.TH = RB * nbands, q.IH = q.TH + 2;
    q.PX = (TW + 1) / 2, q.IW = 2 * q.PX + 2;
    if (q.IH > 256 || (flat ? q.IW * CB > 2048 : q.IW > 256))
        return 0;
    q.tx_bytes = NB * q.IH * q.IW * CB;
    q.stage_bytes = (q.tx_bytes + 127) & ~127;
    // 16 for what goes nowhere; two tiles no less than the row that is read behind a patch
    q.out_bytes = (std::max(NB * q.TH * TW * CB + 16, q.IW * CB / 2 + 16) + 127) & ~127;
    q.Q = NB * nbands * q.PX, q.groups = (q.Q + 7) / 8;
    q.ncb = CB / 16, q.wpc = std::min(DWM_MAX_CONSUMER_WARPS / q.ncb, q.groups), q.nw = q.ncb * q.wpc;
    for (q.teams = std::min(DWM_MAX_TEAMS, DWM_MAX_CONSUMER_WARPS / q.nw);; q.teams--) {
        if (q.teams == 0)
            return 0;
        q.stages = 0;
        const size_t rest = dwm_smem_bytes(q);
        q.stages = rest < DWM_SMEM_BUDGET ? (int)std::min((size_t)DWM_MAX_STAGES, (DWM_SMEM_BUDGET - rest) / q.stage_bytes) : 0;
        // A team that waits for tile i by the parity of its stage has to know that tile i - stages has landed, another team's mostly.  It waits
        // for its output tile first, whose last store, tile i - 2 teams, was behind the end of all tiles up to that one: enough if stages >= 2 teams.
        if (q.stages >= 2 * q.teams)
            break;
    }
    const int rounds = (q.groups + q.wpc - 1) / q.wpc;
    const double walks = (double)q.groups * q.ncb, in = q.tx_bytes, out = (double)NB * q.TH * TW * CB;
    const double issue = walks * (RB * 56.0 + 150.0) / 2.4, chain = rounds * (RB * 230.0 + 600.0) / q.teams, mma = walks * RB * 12.0;
    const double bytes = (0.5 * in + 1.5 * out) / 22.0;
    const int run = (CB + 127) / 128;
    const double runs = 3.5 * NB * (flat ? q.IH * ((q.IW * CB + 127) / 128) + q.TH * ((TW * CB + 127) / 128) : (q.IH * q.IW + q.TH * TW) * run);
    return std::max(std::max(std::max(issue, chain), std::max(mma, bytes)), std::max(runs, 4500.0 / (q.stages - q.teams))) + 100.0;
}

// Tile shape: channel block CB, NB images of TH x TW output pixels cut into bands - the one with the least estimated time over all tiles.  nw is 0
// where no tile fits.
inline DwmParams dwm_search(int C, int out_h, int out_w, int n, bool dense, int sms)
{
    DwmParams best{};
    double best_time = 1e300;
    for (int CB = 16; CB <= DWM_MAX_CONSUMER_WARPS * 16 && CB <= C; CB += 16) {
        if (C % CB || CB % 128 == 0)
            continue;
        for (int xt = 1; xt <= 16 && xt <= out_w; xt++) {
            int TW = (out_w + xt - 1) / xt;
            if (xt > 1)
                TW = (TW + 1) & ~1;
            for (int yt = 1; yt <= 16 && yt <= out_h; yt++)
                for (int nbands = 1; nbands <= 8; nbands++) {
                    const int RB = ((out_h + yt - 1) / yt + nbands - 1) / nbands;
                    if (nbands > 1 && RB < 2)
                        break;
                    for (int NB = 1; NB <= (xt == 1 && yt == 1 ? 16 : 1) && NB <= n; NB++) {
                        DwmParams q{};
                        const double tile = dwm_shape(q, CB, NB, TW, RB, nbands, dense && CB == C && (TW + 3) * CB <= 2048);
                        if (tile == 0)
                            break;
                        const long long xtiles = (out_w + TW - 1) / TW, ytiles = (out_h + q.TH - 1) / q.TH, nblocks = (n + NB - 1) / NB;
                        const long long tiles = xtiles * ytiles * nblocks * (C / CB);
                        if (tiles > 0x7fffffffll)
                            continue;
                        const double waves = (double)tiles / sms, time = (tiles >= 4 * sms ? waves + 0.5 : ceil(waves)) * tile;
                        if (time < best_time * (1.0 - 1e-9)) {
                            best_time = time;
                            q.cblocks = C / CB, q.nblocks = (int)nblocks, q.ytiles = (int)ytiles, q.xtiles = (int)xtiles, q.total_tiles = (int)tiles;
                            best = q;
                        }
                    }
                }
        }
    }
    return best;
}

// CTAs of a launch: a CTA keeps to one channel block and its constants.
inline int dwm_grid(const DwmParams &p, int sms)
{
    return std::min(p.total_tiles, sms >= 2 * p.cblocks ? sms / p.cblocks * p.cblocks : sms);
}

// What a launch takes, us.  Beside the terms of dwm_shape there are the producer's turn (1700 cycles a tile: the wait for a tile's end, its store, the next
// load, one after the other), the hand-over, the constants where a CTA's next tile is another block's, and the SMs that whole channel blocks leave idle;
// the norm stands for terms that meet.  Fitted to 2000 layers of 16 to 6000 channels, which it meets to within 5 % (standard deviation) from 32 M
// outputs on; of smaller ones the previous kernel hides up to 4 us.
inline double dwm_estimate_us(const DwmParams &p, int sms)
{
    const int rounds = (p.groups + p.wpc - 1) / p.wpc, run = (p.CB + 127) / 128, ctas = dwm_grid(p, sms);
    const double walks = (double)p.groups * p.ncb, in = p.tx_bytes, out = (double)p.NB * p.TH * p.TW * p.CB;
    const double runs = p.NB * (p.flat ? p.IH * ((p.IW * p.CB + 127) / 128) + p.TH * ((p.TW * p.CB + 127) / 128) : (p.IH * p.IW + p.TH * p.TW) * run);
    double sum = 0;
    for (double x : {walks * (p.RB * 57.0 + 50.0) / 2.4, rounds * (p.RB * 250.0 + 285.0) / p.teams, walks * p.RB * 12.0, 0.026 * in + 0.067 * out, 3.5 * runs,
                     3400.0 / (p.stages - p.teams), 1700.0}) {
        x *= x, x *= x, x *= x;
        sum += x * x;
    }
    const double tile = sqrt(sqrt(sqrt(sqrt(sum)))) + 400.0 + (ctas % p.cblocks ? 900.0 : 0.0);
    return 6.7 + ((double)p.total_tiles / ctas + 0.5) * tile / 1965.0;
}

// Large enough to be planned at all: below some 32 M outputs the ring's start costs what the walk saves (64 of 57x58x96 15.6 / 13.8, 256 of 7x7x960
// 15.8 / 14.6; 1024 of them 33.8 / 44), except in narrow tensors, whose rows are few runs here and which dp4a reads straight from global memory.
inline bool dwm_large(int C, long long outputs) { return C < 64 || outputs >= 32ll << 20; }

// The planned launch against dp4a.  In a tile of 64 channels the pixels' banks collide (300 of 20x20x256: 26.5 us, 21.0 on dp4a), and narrower ones that are not
// dense rows are the TMA unit's short runs.  For the others dp4a's time, from 2200 layers half up and 1400 half to even, which takes 1.22 of the estimate here:
// 0.45 / 0.59 ps an output for 96 channels, 0.49 / 0.54 for 144 (widths that dp4a has forms of its own for) and 0.53 / 0.66 for others that its tile takes
// whole (`dp4a_whole`), a quarter more for images below 200 pixels; 0.7 / 0.83 and more where it cuts pixels up; 0.49 / 0.57 for narrow tensors, more for small images and for 16 channels
// (0.6 to 0.9, never less than here).  us here / there: 619 of 20x20x144 28.6 / 22.6, 928 of 20x20x96 29.8 / 22.1, 650 of 28x28x144 45.3 / 41.1, 1024 of
// 80x80x48 201 / 170, 104 of 28x27x4000 231 / 219; 1024 of 112x112x32 171 / 207, 3715 of 14x14x144 60.8 / 67.0; half to even 160 of 57x56x144 55.9 / 50.3,
// 836 of 28x28x112 45.7 / 56.2.  Narrow tensors below 64 M outputs stay here, whichever way the estimate falls (mostly 0.7 to 1.0 of dp4a's time, in
// eight of 155 layers 1.05 to 1.24).
inline bool dwm_pays(const DwmParams &p, int C, int out_h, int out_w, int n, bool half_even, bool dp4a_whole, int sms)
{
    const double outputs = (double)n * out_h * out_w * C, pixels = (double)out_h * out_w;
    if (p.nw == 0 || p.CB % 64 == 0 || (C < 64 ? !p.flat : p.CB < 80))
        return false;
    const double us = dwm_estimate_us(p, sms) * (half_even ? 1.22 : 1.0);
    if (C < 64)
        return C == 16 || pixels <= 200 || outputs < (64 << 20) || us < 8.0 + (half_even ? 0.57e-6 : 0.49e-6) * outputs;
    if (dp4a_whole) {
        const double each = half_even ? (C == 96 ? 0.59e-6 : C == 144 ? 0.54e-6 : 0.66e-6) : (C == 96 ? 0.45e-6 : C == 144 ? 0.49e-6 : 0.53e-6);
        return us < (half_even ? 7.5 : 6.5) + each * (pixels <= 200 ? 1.25 : 1.0) * outputs;
    }
    return us < 8.0 + (half_even ? 0.83e-6 : 0.7e-6) * (pixels <= 200 ? 1.12 : 1.0) * outputs;
}

} // namespace espdl
