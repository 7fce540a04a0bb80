// =============================================================================
// start.cu -- the lanes' staged Gaussian start drawn on the device.
//
// The stream of the reference's staged_seed (src/engine/block_solve.cpp:263-277): std::mt19937_64(seed) through
// std::normal_distribution<double>, entry i = (re, im) with im drawn first. As in staged_seed_into (qb_krylov.cuh),
// which draws it on the host bit for bit: two raw outputs make a polar attempt, the accepted attempts in order make the
// entries, entry = (x m, y m), m = sqrt(-2 log(r2) / r2). Here the acceptance is decided with the same arithmetic, so
// every entry comes from its own attempt; the entries themselves differ from the host's by the last bit of log.
//
// What bounds it: the generator is a serial chain of 312-word blocks. One CTA twists a block per step from shared memory,
// a barrier a block, 0.18 us; the attempts are then counted, their places summed and the entries written by the whole
// chip. chain-32 (4.7 M entries, 12 M words): 7 ms, where the host's draw on 16 cores and its upload took about 28
// (E0 of that sector, FP32 storage and refinement: 81 -> 57 ms); below 2^20 entries the host draws with one thread.
// =============================================================================
#include <algorithm>
#include <cstdint>
#include <random>
#include <vector>

#include "qb_internal.cuh"

namespace qb {
namespace {

// MT19937-64 (M. Matsumoto and T. Nishimura, 2000; the parameters of std::mt19937_64).
constexpr int kN = 312, kM = 156;
constexpr int kGenThreads = 160;

__device__ __forceinline__ u64 twist(u64 a, u64 b, u64 c) {
    const u64 x = (a & 0xFFFFFFFF80000000ULL) | (b & 0x7FFFFFFFULL);
    return c ^ (x >> 1) ^ ((0ULL - (x & 1ULL)) & 0xB5026F5AA96619E9ULL);
}
__device__ __forceinline__ u64 temper(u64 y) {
    y ^= (y >> 29) & 0x5555555555555555ULL;
    y ^= (y << 17) & 0x71D67FFFEDA60000ULL;
    y ^= (y << 37) & 0xFFF7EEE000000000ULL;
    return y ^ (y >> 43);
}

// `blocks` blocks of state words into out (their readers temper them), from the seed (first) or from the state left by the launch before. Thread t makes
// words t and t + 156 of each block: word t + 156 needs the new word t, its own, and the last one the new word 0,
// which its thread forms again; so a block needs only the old state, and one barrier.
__global__ void __launch_bounds__(kGenThreads) k_mt64(u64 seed, int first, u64 blocks, u64* state, u64* out) {
    __shared__ u64 mt[2][kN];
    const int t = threadIdx.x;
    if (first) {
        if (t == 0) {
            u64 x = seed;
            mt[0][0] = x;
            for (int i = 1; i < kN; ++i) {
                x = 6364136223846793005ULL * (x ^ (x >> 62)) + static_cast<u64>(i);
                mt[0][i] = x;
            }
        }
    } else {
        for (int i = t; i < kN; i += kGenThreads) mt[0][i] = state[i];
    }
    __syncthreads();
    int cur = 0;
    for (u64 b = 0; b < blocks; ++b) {
        const u64* o = mt[cur];
        u64* w = mt[cur ^ 1];
        if (t < kM) {
            const u64 lo = twist(o[t], o[t + 1], o[t + kM]);
            const u64 next = t + 1 < kM ? o[t + kM + 1] : twist(o[0], o[1], o[kM]);
            const u64 hi = twist(o[t + kM], next, lo);
            w[t] = lo;
            w[t + kM] = hi;
            out[b * kN + t] = lo;
            out[b * kN + kM + t] = hi;
        }
        __syncthreads();
        cur ^= 1;
    }
    for (int i = t; i < kN; i += kGenThreads) state[i] = mt[cur][i];
}

// generate_canonical's value of a state word's output u: u / 2^64, the largest double below 1 when that rounds to 1.
__device__ __forceinline__ double canonical(u64 u) {
    const double r = __dmul_rn(__ull2double_rn(temper(u)), 0x1.0p-64);
    return r >= 1.0 ? 0x1.fffffffffffffp-1 : r;
}
// A polar attempt: x, y and r2, or a negative value when rejected.
__device__ __forceinline__ double polar(const ulonglong2 u, double& x, double& y) {
    x = __dsub_rn(__dmul_rn(2.0, canonical(u.x)), 1.0);
    y = __dsub_rn(__dmul_rn(2.0, canonical(u.y)), 1.0);
    const double r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
    return (r2 > 1.0 || r2 == 0.0) ? -1.0 : r2;
}

constexpr int kPolarThreads = 256;
constexpr int kPolarEach = 4;                           // attempts a thread, in order
constexpr int kPolarBlock = kPolarThreads * kPolarEach;   // attempts a block

// The accepted attempts of each block of kPolarBlock.
__global__ void __launch_bounds__(kPolarThreads) k_polar_count(const ulonglong2* raw, u64 attempts, u32* counts) {
    __shared__ u32 sm[kPolarThreads / 32];
    u32 c = 0;
    for (int q = 0; q < kPolarEach; ++q) {
        const u64 a = static_cast<u64>(blockIdx.x) * kPolarBlock + static_cast<u64>(q) * kPolarThreads + threadIdx.x;
        double x, y;
        if (a < attempts && polar(__ldg(raw + a), x, y) >= 0.0) ++c;
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        u32 s = 0;
        for (int w = 0; w < kPolarThreads / 32; ++w) s += sm[w];
        counts[blockIdx.x] = s;
    }
}

// offs[b] = *base + the counts before block b; *base advances by their sum. One CTA of 1024 threads.
__global__ void __launch_bounds__(1024) k_polar_offsets(const u32* counts, int n, u64* offs, u64* base) {
    __shared__ u32 wsum[32];
    __shared__ u64 run;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) run = *base;
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += 1024) {
        const int i = i0 + static_cast<int>(threadIdx.x);
        const u32 c = i < n ? counts[i] : 0;
        u32 incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const u32 v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        u32 before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < wid) before += wsum[w];
            all += wsum[w];
        }
        if (i < n) offs[i] = run + before + incl - c;
        __syncthreads();
        if (threadIdx.x == 0) run += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *base = run;
}

// The entries of the accepted attempts, at their places below n.
__global__ void __launch_bounds__(kPolarThreads) k_polar_write(const ulonglong2* raw, u64 attempts, const u64* offs, u64 n,
                                                               double2* out) {
    __shared__ u32 wsum[kPolarThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    u64 at = offs[blockIdx.x];
    for (int q = 0; q < kPolarEach; ++q) {
        const u64 a = static_cast<u64>(blockIdx.x) * kPolarBlock + static_cast<u64>(q) * kPolarThreads + threadIdx.x;
        double x = 0.0, y = 0.0;
        const double r2 = a < attempts ? polar(__ldg(raw + a), x, y) : -1.0;
        const unsigned bal = __ballot_sync(0xffffffffu, r2 >= 0.0);
        if (lane == 0) wsum[wid] = __popc(bal);
        __syncthreads();
        u32 before = 0, all = 0;
        for (int w = 0; w < kPolarThreads / 32; ++w) {
            if (w < wid) before += wsum[w];
            all += wsum[w];
        }
        const u64 i = at + before + __popc(bal & ((1u << lane) - 1u));
        if (r2 >= 0.0 && i < n) {
            const double m = sqrt(__ddiv_rn(__dmul_rn(-2.0, log(r2)), r2));
            out[i] = make_double2(__dmul_rn(x, m), __dmul_rn(y, m));
        }
        at += all;
        __syncthreads();
    }
}

// Up to this many entries the host draws them: the device's four launches and its wait take about 60 us whatever the number,
// the host 0.06 us an entry (the lowest level of 8 states: 1.08 ms with the host's draw, 1.13 with the device's).
constexpr std::uint64_t kHostEntries = 512;

// A pass of the draw: at most 1 M attempts, 16 MB of raw outputs.
constexpr u64 kPassBlocks = (u64{1} << 20) / (kN / 2);

}  // namespace

// out[0, n): the staged start of the seed, queued on st; returns when it is complete.
void staged_start_device(double2* out, std::uint64_t n, std::uint64_t seed, cudaStream_t st) {
    if (n == 0) return;
    if (n <= kHostEntries) {
        std::vector<double2> v(n);
        std::mt19937_64 gen(seed);
        std::normal_distribution<double> normal(0.0, 1.0);
        for (double2& z : v) {
            z.y = normal(gen);   // the imaginary part is drawn first
            z.x = normal(gen);
        }
        upload_host(out, v.data(), n * 16, st);
        return;
    }
    // pi/4 of the attempts are accepted: the expected number and a margin, in whole generator blocks of 156 attempts
    auto blocks_for = [](u64 left) {
        const u64 a = left + left / 4 + left / 32 + 1024;
        return std::min<u64>(kPassBlocks, (a + kN / 2 - 1) / (kN / 2));
    };
    const u64 most = blocks_for(n);
    const u64 most_polar = (most * (kN / 2) + kPolarBlock - 1) / kPolarBlock;
    DevBuf<u64> raw(most * kN), state(kN), offs(most_polar), base(1);
    DevBuf<u32> counts(most_polar);
    cuda_check(cudaMemsetAsync(base.p, 0, 8, st), "start clear");
    u64 done = 0;
    for (int pass = 0; done < n; ++pass) {
        const u64 blocks = std::min(most, blocks_for(n - done));
        const u64 attempts = blocks * (kN / 2);
        const unsigned pb = static_cast<unsigned>((attempts + kPolarBlock - 1) / kPolarBlock);
        k_mt64<<<1, kGenThreads, 0, st>>>(seed, pass == 0, blocks, state.p, raw.p);
        k_polar_count<<<pb, kPolarThreads, 0, st>>>(reinterpret_cast<const ulonglong2*>(raw.p), attempts, counts.p);
        k_polar_offsets<<<1, 1024, 0, st>>>(counts.p, static_cast<int>(pb), offs.p, base.p);
        k_polar_write<<<pb, kPolarThreads, 0, st>>>(reinterpret_cast<const ulonglong2*>(raw.p), attempts, offs.p, n, out);
        cuda_check(cudaGetLastError(), "staged start");
        cuda_check(cudaMemcpyAsync(&done, base.p, 8, cudaMemcpyDeviceToHost, st), "staged start");
        cuda_check(cudaStreamSynchronize(st), "staged start");
    }
}

}  // namespace qb
