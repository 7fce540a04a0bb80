// =============================================================================
// dense.cu -- the dense tail on the device: the full spectra of many small blocks at once.
//
// The reference solves blocks up to dense_max_dim exactly (include/ed/sectors/thermal.h:35) through a pool of
// cusolverDnXsyevd streams (src/gpu/little_group.cu:185-188). Here every block is assembled on the device from
// its row walk in one launch (k_assemble) into one column-major buffer of all blocks, and one launch reduces them
// all, a CTA per block (largest first):
//   - Householder reflections to a Hermitian tridiagonal: for each column k, v = x - alpha e1 (alpha = -x0 /
//     |x0| ||x||) normalised, p = A22 v, w = p - (v^H p) v, A22 -= 2 (v w^H + w v^H). One pass over A22 a step:
//     the previous step's update is applied to column k alone, which fixes v, and the pass that applies it to
//     the rest forms p from the updated elements as it stores them (p_j = sum_i conj(a_ij) v_i, A22 being
//     Hermitian), a warp per pair of columns, v and w in shared memory;
//   - the moduli of the off-diagonal make a real symmetric tridiagonal with the same spectrum;
//   - every eigenvalue by Sturm-count bisection to full precision, the threads taking the indices in turn, so
//     the levels come out ascending.
// Blocks above kDenseDeviceMax states keep the host reduction (lanes.cu).
// =============================================================================
#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include "qb_krylov.cuh"
#include "qb_walk.cuh"

namespace qb {

const qb_csr* csr_lane(const qb_sector* row, const qb_sector* col, const qb_program* P);

namespace {

constexpr int kDenseDeviceMax = 1024;   // four vectors of 16-byte elements in shared memory, a row a thread
constexpr int kDenseThreads = 1024;
static_assert(kDenseThreads >= kDenseDeviceMax, "a thread holds at most one row of a column");
// Launches whose largest block has at most this many states: 256 threads, whose barriers and sums of the warps' sums are
// shorter (one block, us, 1,024 against 256 threads: 12 states 188 / 165, 28 338 / 279, 56 828 / 727; 126 states 1,548 / 1,421,
// 210 3,478 / 3,489).
constexpr int kDenseFew = 64, kDenseFewThreads = 256;

struct DenseBlock {
    unsigned long long a_off;   // the block's matrix at A + a_off (column-major, n x n)
    unsigned long long v_off;   // its levels at values + v_off
    int n;
};

// A block to assemble, and its matrix at A + a_off.
struct AsmItem {
    DSector sec;
    DProgram prog;
    unsigned long long a_off;
    int in_smem;
};
struct AsmTile {
    int item;
    u32 row0;
};

// The matrices of all blocks, cleared before: a thread per row walks its row and adds each entry into its column in
// group order, the sums of the block matvec on identity columns. A tile of 256 rows a CTA; every block's tiles run
// side by side. (The identity matvecs took two small kernels and a walk per 64 columns, one after another: on the
// 238 dense blocks of a 16-site chain 8 ms of kernels in 1,700 launches, against one of 0.09 ms.)
constexpr int kAsmRows = 256;
template <class ST>
__global__ void __launch_bounds__(kAsmRows) k_assemble(const AsmItem* items, const AsmTile* tiles, double2* A_all) {
    extern __shared__ __align__(16) unsigned char smem[];
    const AsmItem& I = items[tiles[blockIdx.x].item];
    const SmemProgram sp = stage(I.prog, I.sec, smem, I.in_smem != 0);
    const std::uint64_t n = I.sec.dim, r = tiles[blockIdx.x].row0 + threadIdx.x;
    if (r >= n) return;
    double2* A = A_all + I.a_off;
    const ST s = static_cast<ST>(__ldg(I.sec.reps + r));
    const double w = __ldg(I.sec.inv_norms + r);
    for (u32 g = 0; g < sp.P.n_groups; ++g) {
        ST t;
        cplx h, c;
        long long j;
        if (!connection<ST>(sp.P, s, g, t, h)) continue;
        if (!entry<true, ST>(I.sec, sp.T, s, static_cast<long long>(r), w, t, h, j, c)) continue;
        double2& a = A[static_cast<std::size_t>(j) * n + r];
        const cplx sum = cadd({a.x, a.y}, c);
        a = make_double2(sum.re, sum.im);
    }
}

// A block with an attached CSR: its stored rows instead of the walk, a thread per row.
__global__ void k_assemble_csr(std::uint64_t n, const unsigned long long* row_ptr, const u32* col,
                               const unsigned char* ids, int id_bytes, const double2* vals, double2* A) {
    const std::uint64_t r = static_cast<std::uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= n) return;
    for (unsigned long long e = row_ptr[r]; e < row_ptr[r + 1]; ++e) {
        const u64 id = id_bytes == 1 ? ids[e] : id_bytes == 2 ? reinterpret_cast<const u16*>(ids)[e] : e;
        const double2 v = vals[id];
        double2& a = A[static_cast<std::size_t>(col[e]) * n + r];
        const cplx sum = cadd({a.x, a.y}, {v.x, v.y});
        a = make_double2(sum.re, sum.im);
    }
}

__device__ __forceinline__ double block_sum(double v, double* sm) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    double s = 0.0;
    for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) s += sm[i];   // the same order in every thread
    return s;
}

__device__ int sturm_below(const double* d, const double* e, int n, double x) {
    int c = 0;
    double q = d[0] - x;
    if (q < 0.0) ++c;
    for (int i = 1; i < n; ++i) {
        const double qq = q != 0.0 ? q : 2.2250738585072014e-308;
        q = d[i] - x - e[i - 1] * e[i - 1] / qq;
        if (q < 0.0) ++c;
    }
    return c;
}

// What bounds it: the matrix streams through one SM's path to L2, 32 bytes an element and step (read and written
// once), about n^3 / 3 elements in all; then the latency of a step's sums. A warp takes two columns at a time, so
// that one read of v_i, w_i and the new v_i from shared memory serves two elements, and each lane keeps several
// elements in flight. The 238 dense blocks of a 16-site chain (64 of about 500 states, side by side): 23 ms, where two
// passes over A22 a step (p, then the update), 256 threads and a thread per row of p took 145 ms.
constexpr std::size_t kDenseSmem = (4 * static_cast<std::size_t>(kDenseDeviceMax) * 16) + 64 * 8;
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 1) k_dense_levels(const DenseBlock* blocks, double2* A_all,
                                                                   double* values) {
    extern __shared__ __align__(16) unsigned char smem[];
    double2* v = reinterpret_cast<double2*>(smem);       // the pending update A22 -= 2 (v w^H + w v^H)
    double2* w = v + kDenseDeviceMax;
    double2* vn = w + kDenseDeviceMax;                   // this step's reflection
    double2* p = vn + kDenseDeviceMax;
    double* sm = reinterpret_cast<double*>(p + kDenseDeviceMax);
    __shared__ double d[kDenseDeviceMax], e[kDenseDeviceMax];
    __shared__ double s_lo, s_hi;
    const DenseBlock B = blocks[blockIdx.x];
    const int n = B.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarps = kThreads / 32;
    double2* A = A_all + B.a_off;
    auto col = [&](int c) { return A + static_cast<std::size_t>(c) * n; };
    // a - 2 (vi conj(wj) + wi conj(vj))
    auto updated = [](double2 a, double2 vi, double2 wi, double2 vj, double2 wj) {
        a.x -= 2.0 * ((vi.x * wj.x + vi.y * wj.y) + (wi.x * vj.x + wi.y * vj.y));
        a.y -= 2.0 * ((vi.y * wj.x - vi.x * wj.y) + (wi.y * vj.x - wi.x * vj.y));
        return a;
    };
    for (int i = threadIdx.x; i < n; i += kThreads) v[i] = w[i] = make_double2(0.0, 0.0);
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        // column k with the pending update; a thread keeps its row's element (n is at most the threads)
        const int i0 = k + threadIdx.x;
        double2 x = make_double2(0.0, 0.0);
        if (i0 < n) x = updated(col(k)[i0], v[i0], w[i0], v[k], w[k]);
        if (threadIdx.x == 0) {
            d[k] = x.x;
            x = make_double2(0.0, 0.0);
        }
        if (k + 1 >= n) {
            if (threadIdx.x == 0) e[k] = 0.0;
            break;
        }
        const double xn = sqrt(block_sum(x.x * x.x + x.y * x.y, sm));
        if (threadIdx.x == 0) e[k] = xn;   // |alpha|, the modulus the reflection leaves below the diagonal
        if (k + 2 >= n) {
            __syncthreads();
            continue;
        }
        if (threadIdx.x == 1) {            // v = x - alpha e1, alpha = -(x0 / |x0|) ||x||: x0 grows by ||x|| along itself
            const double ax0 = sqrt(x.x * x.x + x.y * x.y);
            const double2 ph = ax0 > 0.0 ? make_double2(x.x / ax0, x.y / ax0) : make_double2(1.0, 0.0);
            x.x += ph.x * xn;
            x.y += ph.y * xn;
        }
        const double len = sqrt(block_sum(x.x * x.x + x.y * x.y, sm));
        const double inv = len > 0.0 ? 1.0 / len : 0.0;   // a zero column: no reflection, the pending update alone
        if (i0 < n && threadIdx.x > 0) vn[i0] = make_double2(x.x * inv, x.y * inv);
        __syncthreads();
        // the pass: two columns a warp
        for (int j = k + 1 + 2 * warp; j < n; j += 2 * kWarps) {
            const bool two = j + 1 < n;
            const int j1 = two ? j + 1 : j;
            double2* c0 = col(j);
            double2* c1 = col(j1);
            const double2 vj0 = v[j], wj0 = w[j], vj1 = v[j1], wj1 = w[j1];
            double r0 = 0.0, s0 = 0.0, r1 = 0.0, s1 = 0.0;
            int i = k + 1 + lane;
            constexpr int U = 2;
            for (; i + 32 * (U - 1) < n; i += 32 * U) {
                double2 a0[U], a1[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    a0[u] = c0[i + 32 * u];
                    a1[u] = c1[i + 32 * u];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const double2 vi = v[i + 32 * u], wi = w[i + 32 * u], z = vn[i + 32 * u];
                    const double2 y0 = updated(a0[u], vi, wi, vj0, wj0), y1 = updated(a1[u], vi, wi, vj1, wj1);
                    c0[i + 32 * u] = y0;
                    if (two) c1[i + 32 * u] = y1;
                    r0 += y0.x * z.x + y0.y * z.y;
                    s0 += y0.x * z.y - y0.y * z.x;
                    r1 += y1.x * z.x + y1.y * z.y;
                    s1 += y1.x * z.y - y1.y * z.x;
                }
            }
            for (; i < n; i += 32) {
                const double2 vi = v[i], wi = w[i], z = vn[i];
                const double2 y0 = updated(c0[i], vi, wi, vj0, wj0), y1 = updated(c1[i], vi, wi, vj1, wj1);
                c0[i] = y0;
                if (two) c1[i] = y1;
                r0 += y0.x * z.x + y0.y * z.y;
                s0 += y0.x * z.y - y0.y * z.x;
                r1 += y1.x * z.x + y1.y * z.y;
                s1 += y1.x * z.y - y1.y * z.x;
            }
            for (int o = 16; o > 0; o >>= 1) {
                r0 += __shfl_xor_sync(0xffffffffu, r0, o);
                s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                r1 += __shfl_xor_sync(0xffffffffu, r1, o);
                s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            }
            if (lane == 0) {
                p[j] = make_double2(r0, s0);
                if (two) p[j1] = make_double2(r1, s1);
            }
        }
        __syncthreads();
        // K = v^H p (real), w = p - K v: the next pending update
        double2 z = make_double2(0.0, 0.0), pi = z;
        if (i0 < n && threadIdx.x > 0) {
            z = vn[i0];
            pi = p[i0];
        }
        const double K = block_sum(z.x * pi.x + z.y * pi.y, sm);
        if (i0 < n && threadIdx.x > 0) {
            v[i0] = z;
            w[i0] = make_double2(pi.x - K * z.x, pi.y - K * z.y);
        }
        __syncthreads();
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // Gershgorin bounds
        double lo = 1e300, hi = -1e300;
        for (int i = lane; i < n; i += 32) {
            const double r = (i > 0 ? e[i - 1] : 0.0) + (i + 1 < n ? e[i] : 0.0);
            lo = fmin(lo, d[i] - r);
            hi = fmax(hi, d[i] + r);
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        const double pad = 1e-12 * fmax(fabs(lo), fabs(hi)) + 1e-300;
        s_lo = lo - pad;
        s_hi = hi + pad;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < n; q += kThreads) {
        double lo = s_lo, hi = s_hi;
        for (int it = 0; it < 200; ++it) {
            const double mid = 0.5 * (lo + hi);
            if (mid <= lo || mid >= hi) break;
            if (sturm_below(d, e, n, mid) > q)
                hi = mid;
            else
                lo = mid;
        }
        values[B.v_off + q] = 0.5 * (lo + hi);
    }
}

// Launches k_assemble over the blocks of `set`.
template <class ST>
void assemble(const std::vector<int>& set, const qb_sector* const* secs, const qb_program* const* progs,
              const std::vector<std::uint64_t>& a_off, double2* A, DevBuf<AsmItem>& d_items, DevBuf<AsmTile>& d_tiles,
              QueuedUploads& up) {
    if (set.empty()) return;
    std::vector<AsmItem> items;
    std::vector<AsmTile> tiles;
    std::size_t smem = 0;
    for (int b : set) {
        bool in_smem = false;
        smem = std::max(smem, smem_for(progs[b], secs[b], in_smem));
        for (std::uint64_t r = 0; r < secs[b]->dim; r += kAsmRows)
            tiles.push_back(AsmTile{static_cast<int>(items.size()), static_cast<u32>(r)});
        items.push_back(AsmItem{secs[b]->view(), progs[b]->view, a_off[b], in_smem ? 1 : 0});
    }
    const unsigned n_tiles = static_cast<unsigned>(tiles.size());
    up.add(d_items, std::move(items));
    up.add(d_tiles, std::move(tiles));
    set_smem(k_assemble<ST>, smem);
    k_assemble<ST><<<n_tiles, kAsmRows, smem, cudaStreamPerThread>>>(d_items.p, d_tiles.p, A);
    cuda_check(cudaGetLastError(), "dense assembly");
}

}  // namespace

// The spectra of blocks of at most kDenseDeviceMax states, all on the device: block b's levels, ascending, at
// values[off[b] ...] (host). Returns false (nothing done) when a block is larger.
bool dense_levels_device(const qb_sector* const* secs, const qb_program* const* progs, int n_blocks,
                         const std::vector<std::size_t>& off, double* values) {
    std::uint64_t a_tot = 0, v_tot = 0;
    std::vector<DenseBlock> desc;
    std::vector<std::uint64_t> a_off(n_blocks, 0);
    std::vector<int> walk_set[2];   // 32-bit and 64-bit states
    for (int b = 0; b < n_blocks; ++b) {
        const std::uint64_t n = secs[b]->dim;
        if (n > static_cast<std::uint64_t>(kDenseDeviceMax)) return false;
        if (n == 0) continue;
        desc.push_back(DenseBlock{a_tot, off[b], static_cast<int>(n)});
        a_off[b] = a_tot;
        a_tot += n * n;
        v_tot = std::max<std::uint64_t>(v_tot, off[b] + n);
        if (!csr_lane(secs[b], secs[b], progs[b])) walk_set[secs[b]->N <= 32 ? 0 : 1].push_back(b);
    }
    if (desc.empty()) return true;
    DevBuf<double2> A(a_tot);
    cuda_check(cudaMemsetAsync(A.p, 0, a_tot * 16, cudaStreamPerThread), "dense clear");
    DevBuf<AsmItem> d_items[2];
    DevBuf<AsmTile> d_tiles[2];
    QueuedUploads up;
    assemble<u32>(walk_set[0], secs, progs, a_off, A.p, d_items[0], d_tiles[0], up);
    assemble<u64>(walk_set[1], secs, progs, a_off, A.p, d_items[1], d_tiles[1], up);
    for (int b = 0; b < n_blocks; ++b)
        if (const qb_csr* C = secs[b]->dim ? csr_lane(secs[b], secs[b], progs[b]) : nullptr)
            k_assemble_csr<<<static_cast<unsigned>((C->rows + 127) / 128), 128, 0, cudaStreamPerThread>>>(
                C->rows, C->row_ptr.p, C->col_idx.p, C->ids.p, C->id_bytes, C->vals.p, A.p + a_off[b]);
    cuda_check(cudaGetLastError(), "dense assembly");
    std::vector<int> order(desc.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return desc[a].n > desc[c].n; });
    std::vector<DenseBlock> sorted(desc.size());
    for (std::size_t i = 0; i < order.size(); ++i) sorted[i] = desc[order[i]];
    DevBuf<DenseBlock> dd;
    const unsigned n_desc = static_cast<unsigned>(sorted.size());
    const int most = sorted.front().n;
    up.add(dd, std::move(sorted));
    DevBuf<double> dv(v_tot);
    auto go = [&](auto kernel, int threads) {
        set_smem(kernel, kDenseSmem);
        kernel<<<n_desc, threads, kDenseSmem, cudaStreamPerThread>>>(dd.p, A.p, dv.p);
    };
    if (most <= kDenseFew)
        go(k_dense_levels<kDenseFewThreads>, kDenseFewThreads);
    else
        go(k_dense_levels<kDenseThreads>, kDenseThreads);
    cuda_check(cudaGetLastError(), "dense levels");
    std::vector<double> hv(v_tot);
    cuda_check(cudaMemcpy(hv.data(), dv.p, v_tot * 8, cudaMemcpyDeviceToHost), "dense levels");
    up.finish();
    for (const auto& d : desc) std::copy(hv.begin() + d.v_off, hv.begin() + d.v_off + d.n, values + d.v_off);
    return true;
}

}  // namespace qb
