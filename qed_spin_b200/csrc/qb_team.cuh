// =============================================================================
// qb_team.cuh -- the team walk: a team of lanes per row, for blocks of vectors and for one vector on a small sector.
// Compiled for 32-bit states (team32.cu), 64-bit ones (team64.cu) and 64-bit ones of sectors with row pairs
// (team64_pairs.cu).
// =============================================================================
#pragma once

#include "qb_walk.cuh"

namespace qb {
namespace {

// Team kernel: kTeam lanes per row (4, 8, 16 or 32), kCpl columns per lane (k <= kTeam kCpl vectors). Every column
// adds its row's entries in group order whatever kTeam is, so the team size changes only the time.
// What bounds it: instruction issue (canonicalisation, then eight FP64 operations an element and target) and the latency of
// the loads between. 32-bit states when every state fits. Registers: the compiler's own count (60 to 64 for up to five
// columns of 32-bit states) with no bound on the blocks an SM. A bound of one block an SM gave one column 128 registers:
// 2% faster on the 9,252 rows of chain-20 alone (25.0 against 25.6 us), 1.2 to 1.7x slower from 20 k rows, where a launch is
// more than two blocks an SM (one vector, chain-24 at 8 spins up 52.8 against 39.0 us; 6x5 at 7 spins up 400 against 274).
// A bound of four blocks spills in 64-bit states (one vector, 36 sites at 5 spins up 69.7 against 64.3 us) and from five
// columns on (chain-24, 40 FP64 vectors 203 against 188 us, FP32 159 against 155). Two columns of 32-bit states in teams of 32
// are the exception: there the compiler's count spills (64 FP64 vectors, chiral-24 at 9 spins up 248 against 232 us).
template <class State, int kTeam, int kCpl>
constexpr int kTeamBlocks = sizeof(State) == 4 && kTeam == 32 && kCpl == 2 ? 4 : 0;   // 0: no bound
template <class State, int kTeam, int kCpl, bool kF32, bool kOutF32, bool kSame, int kCand>
__global__ void __launch_bounds__(256, kTeamBlocks<State, kTeam, kCpl>) walk_team(DSector row, DSector col, DProgram P,
                                                 bool prog_in_smem, const void* in_v, void* out_v, int k) {
    extern __shared__ __align__(16) unsigned char smem[];
    using St = Store<kF32>;
    using So = Store<kOutF32>;
    using T = typename St::T;
    const T* in = static_cast<const T*>(in_v);
    typename So::T* out = static_cast<typename So::T*>(out_v);
    const SmemProgram sp = stage(P, col, smem, prog_in_smem);
    const int lane = threadIdx.x & 31;
    const int team = lane / kTeam, tl = lane % kTeam;
    const unsigned team_mask = kTeam == 32 ? 0xffffffffu : ((1u << kTeam) - 1u) << (team * kTeam);
    const std::uint64_t warp = (static_cast<std::uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const std::uint64_t r = warp * (32 / kTeam) + team;
    const bool live = r < row.dim;
    const State s = live ? static_cast<State>(__ldg(row.reps + r)) : State(0);
    const double w = live ? __ldg(row.inv_norms + r) : 0.0;
    cplx acc[kCpl];
#pragma unroll
    for (int c = 0; c < kCpl; ++c) acc[c] = {0.0, 0.0};
    const int c0 = tl * kCpl;
    for (u32 g0 = 0; g0 < sp.P.n_groups; g0 += kTeam) {
        const u32 g = g0 + tl;
        State t = 0;
        cplx h{0.0, 0.0};
        long long j = -1;
        cplx cv{0.0, 0.0};
        bool act = live && g < sp.P.n_groups && connection<State>(sp.P, s, g, t, h);
        if (act) act = entry<kSame, State, kCand>(col, sp.T, s, static_cast<long long>(r), w, t, h, j, cv);
        unsigned acting = __ballot_sync(0xffffffffu, act) & team_mask;
        while (acting) {
            const int src = __ffs(acting) - 1;
            acting &= acting - 1;
            const long long jj = __shfl_sync(team_mask, j, src);
            const double cre = __shfl_sync(team_mask, cv.re, src);
            const double cim = __shfl_sync(team_mask, cv.im, src);
            const std::size_t base = static_cast<std::size_t>(jj) * k;
#pragma unroll
            for (int c = 0; c < kCpl; ++c)
                if (c0 + c < k) acc[c] = cadd(acc[c], cmul({cre, cim}, St::load(in, base + c0 + c)));
        }
    }
    if (!live) return;
#pragma unroll
    for (int c = 0; c < kCpl; ++c)
        if (c0 + c < k) So::store(out, static_cast<std::size_t>(r) * k + c0 + c, acc[c]);
}

template <class State, int kCand, int kTeam, int kCpl, bool kF32, bool kOutF32>
void team_launch(const qb_sector* row, const qb_sector* col, const qb_program* P, const void* in, void* out, int k,
                 cudaStream_t st) {
    bool in_smem = false;
    const std::size_t smem = smem_for(P, col, in_smem, kCand == kRowPairs);
    constexpr int kRowsPerWarp = 32 / kTeam;
    const std::uint64_t warps = (row->dim + kRowsPerWarp - 1) / kRowsPerWarp;
    const unsigned blocks = static_cast<unsigned>((warps * 32 + 255) / 256);
    auto go = [&](auto kk) {
        set_smem(kk, smem);
        kk<<<blocks, 256, smem, st>>>(row->view(), col->view(kCand == kRowPairs), P->view, in_smem, in, out, k);
    };
    if (row == col)
        go(walk_team<State, kTeam, kCpl, kF32, kOutF32, true, kCand>);
    else
        go(walk_team<State, kTeam, kCpl, kF32, kOutF32, false, kCand>);
    cuda_check(cudaGetLastError(), "walk_team launch");
}

// The columns per lane: the least of 1, 2, 4, 5 and 8 that covers k; a team that covers the 64 vectors of a block walk
// with fewer has no kernel of the larger ones.
template <class State, int kCand, int kTeam, bool kF32, bool kOutF32>
void team_cols(const qb_sector* row, const qb_sector* col, const qb_program* P, const void* in, void* out, int k,
               cudaStream_t st) {
    const int cpl = (k + kTeam - 1) / kTeam;
    if (cpl <= 1) return team_launch<State, kCand, kTeam, 1, kF32, kOutF32>(row, col, P, in, out, k, st);
    if (cpl <= 2) return team_launch<State, kCand, kTeam, 2, kF32, kOutF32>(row, col, P, in, out, k, st);
    if constexpr (kTeam < 32)
        if (cpl <= 4) return team_launch<State, kCand, kTeam, 4, kF32, kOutF32>(row, col, P, in, out, k, st);
    if constexpr (kTeam < 16) {
        if (cpl <= 5) return team_launch<State, kCand, kTeam, 5, kF32, kOutF32>(row, col, P, in, out, k, st);
        if (cpl <= 8) return team_launch<State, kCand, kTeam, 8, kF32, kOutF32>(row, col, P, in, out, k, st);
    }
    throw Error(QB_EUNSUPPORTED, "block matvec: at most 64 vectors");
}

template <class State, int kCand, bool kF32, bool kOutF32>
void team_shape(int shape, const qb_sector* row, const qb_sector* col, const qb_program* P, const void* in, void* out,
                int k, cudaStream_t st) {
    if (shape == 0)
        team_cols<State, kCand, 8, kF32, kOutF32>(row, col, P, in, out, k, st);
    else if (shape == 1)
        team_cols<State, kCand, 16, kF32, kOutF32>(row, col, P, in, out, k, st);
    else if (shape == 2)
        team_cols<State, kCand, 32, kF32, kOutF32>(row, col, P, in, out, k, st);
    else
        team_cols<State, kCand, 4, kF32, kOutF32>(row, col, P, in, out, k, st);
}

template <class State, int kCand>
void launch_walk_team(int shape, bool in32, bool out32, const qb_sector* row, const qb_sector* col, const qb_program* P,
                      const void* in, void* out, int k, cudaStream_t st) {
    if (in32 && out32)
        team_shape<State, kCand, true, true>(shape, row, col, P, in, out, k, st);
    else if (in32)
        team_shape<State, kCand, true, false>(shape, row, col, P, in, out, k, st);
    else if (out32)
        team_shape<State, kCand, false, true>(shape, row, col, P, in, out, k, st);
    else
        team_shape<State, kCand, false, false>(shape, row, col, P, in, out, k, st);
}

}  // namespace
}  // namespace qb
