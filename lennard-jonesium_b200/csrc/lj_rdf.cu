// lj_rdf.cu -- radial distribution histogram (new: the reference has no RDF).
//
// Ordered pairs (i != j) at minimum-image distance r < rmax are counted in bin
// floor(sqrt(r^2) * (nbins / rmax)).  The separation, r^2 and the bin follow
// exactly the arithmetic of the CPU oracle (dd - image * L with image from
// dd > L/2, fma-ordered r^2, IEEE sqrt), so histograms agree bit-for-bit.
//
// Boxes with at least 3 cells of edge >= rmax per axis use a cell list over half a
// stencil (counting sort into an RDF grid, positions copied in that order; each
// unordered pair evaluated once and counted twice); smaller boxes use all pairs.
// Where the bins are wide against FP32 rounding of the box coordinates, the cells are
// half as large and a pair is tested, and its bin found, in FP32 -- unless its
// distance lies so near a bin's edge that the rounding could matter, when the
// exact arithmetic above decides.  Each block accumulates a shared-memory
// histogram and adds it to the global 64-bit histogram once.

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "lj_mixed.cuh"

namespace ljb {

namespace {

__device__ __forceinline__ double min_image(double dd, double L, double halfL) {
    double img = dd > halfL ? 1.0 : (dd < -halfL ? -1.0 : 0.0);
    return __dsub_rn(dd, __dmul_rn(img, L));
}

template <unsigned INC>
__device__ __forceinline__ void rdf_count(const double4& xi, const double4& xj, const PairParams& pp,
                                          double rmax2, double inv_dr, int nbins, unsigned* sh) {
    double sx = min_image(__dsub_rn(xi.x, xj.x), pp.L[0], pp.halfL[0]);
    double sy = min_image(__dsub_rn(xi.y, xj.y), pp.L[1], pp.halfL[1]);
    double sz = min_image(__dsub_rn(xi.z, xj.z), pp.L[2], pp.halfL[2]);
    double r2 = norm2(sx, sy, sz);
    if (r2 < rmax2) {
        int b = (int)__dmul_rn(__dsqrt_rn(r2), inv_dr);
        if (b < nbins) atomicAdd(&sh[b], INC);
    }
}

// Add the block's counts to the histogram; they start from zero again.
__device__ __forceinline__ void flush(unsigned* sh, int nbins, unsigned long long* hist) {
    __syncthreads();
    for (int b = threadIdx.x; b < nbins; b += blockDim.x)
        if (sh[b]) {
            atomicAdd(&hist[b], (unsigned long long)sh[b]);
            sh[b] = 0;
        }
    __syncthreads();
}

// All pairs: block (x, y) takes 128 atoms i against the y-th slice of the j > i.
__global__ void __launch_bounds__(kThreads)
rdf_all_pairs_kernel(int N, const double4* __restrict__ pos, PairParams pp, double rmax2, double inv_dr,
                     int nbins, unsigned long long* __restrict__ hist) {
    extern __shared__ unsigned sh[];
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) sh[b] = 0;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, per = (N + gridDim.y - 1) / gridDim.y;
    const int j0 = blockIdx.y * per, j1 = min(N, j0 + per);
    if (i < N) {
        double4 xi = pos[i];
        for (int j = max(j0, i + 1); j < j1; ++j) rdf_count<2u>(xi, pos[j], pp, rmax2, inv_dr, nbins, sh);
    }
    flush(sh, nbins, hist);
}

__global__ void __launch_bounds__(kThreads)
rdf_cells_kernel(int N, const double4* __restrict__ sorted, Grid g, const int* __restrict__ start,
                 PairParams pp, double rmax2, double inv_dr, int nbins, unsigned long long* __restrict__ hist) {
    extern __shared__ unsigned sh[];
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) sh[b] = 0;
    __syncthreads();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) {
        double4 xi = sorted[i];
        int ci[3] = {cell_coord(xi.x, g.ratio[0], g.n[0]), cell_coord(xi.y, g.ratio[1], g.n[1]),
                     cell_coord(xi.z, g.ratio[2], g.n[2])};
        // half shell: the own cell's later atoms and the 13 stencil cells after
        // the own cell in (a, b, c) order; each unordered pair is met once and
        // counts for both ordered pairs (the separation of (j, i) is exactly the
        // negated one of (i, j), so both fall in the same bin)
        for (int j = i + 1; j < start[g.flat(ci[0], ci[1], ci[2]) + 1]; ++j)
            rdf_count<2u>(xi, sorted[j], pp, rmax2, inv_dr, nbins, sh);
        for (int s = 14; s < 27; ++s) {
            int a = s / 9 - 1, b = (s / 3) % 3 - 1, c = s % 3 - 1;
            int cell = g.flat((ci[0] + a + g.n[0]) % g.n[0], (ci[1] + b + g.n[1]) % g.n[1],
                              (ci[2] + c + g.n[2]) % g.n[2]);
            for (int j = start[cell]; j < start[cell + 1]; ++j)
                rdf_count<2u>(xi, sorted[j], pp, rmax2, inv_dr, nbins, sh);
        }
    }
    flush(sh, nbins, hist);
}

constexpr int kStep = 4;  // candidates a lane takes at a time
constexpr unsigned kAll = (1u << kStep) - 1u;

// What the FP32 test of a pair needs: E bounds the error of the FP32 distance.
struct RdfFast {
    float outer2;       // (rmax + E)^2: no pair beyond counts
    float inv_dr;
    float half;         // a bin is certain within this of its middle, in bins,
    float end;          // and below 2^23 + nbins
    float3 Lf;
};

// Half the stencil of +-2 cells of edge >= rmax / 2 (>= 5 per axis): the atom's later
// column mates up to two cells above, then the columns after its own in (a, b)
// order, each a run of slots (two where it wraps in z).  One atom per thread, the
// columns dealt to the grid's y blocks; four candidates at a time from a 16-byte
// boundary, one load an axis, tested two per
// instruction with packed FP32 arithmetic (PosNeg: negated, by component); the lanes
// of a warp are neighbours in a column and read the same candidates.  A candidate
// whose bin is certain is counted at once, one whose is not is left to the exact
// arithmetic after the block.  The counts are added up after every `rounds` rounds of
// atoms, before 32 bits could wrap (rdf_rounds).  Bound by issue (70 %, 19 of 32 lanes
// active in the branch of a hit).  Measured at 100 003 atoms, rho 0.8442, 200 bins to 4.0: a whole
// sample 355 -> 98 us, this kernel 82; the exact form tests 729 candidates an atom in
// FP64, one thread per atom.
__global__ void __launch_bounds__(kThreads, 6)
rdf_fast_kernel(int N, const double4* __restrict__ sorted, PosNeg posn, Grid g, const int* __restrict__ start,
                PairParams pp, double rmax2, double inv_dr, int nbins, RdfFast f, int rounds,
                unsigned long long* __restrict__ hist) {
    extern __shared__ unsigned sh[];
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) sh[b] = 0;
    __syncthreads();
    const float* const px = posn.p;
    const float* const py = px + posn.np;
    const float* const pz = py + posn.np;
    const int nz = g.n[2];
    int round = 0;
    for (int i0 = blockIdx.x * blockDim.x; i0 < N; i0 += gridDim.x * blockDim.x, ++round) {
        if (round == rounds) {
            flush(sh, nbins, hist);
            round = 0;
        }
        const int i = i0 + threadIdx.x;
        if (i >= N) continue;  // (the last round of all)
        const double4 xd = sorted[i];
        const float xi = (float)xd.x, yi = (float)xd.y, zi = (float)xd.z;
        const int ca = cell_coord(xd.x, g.ratio[0], g.n[0]), cb = cell_coord(xd.y, g.ratio[1], g.n[1]),
                  cc = cell_coord(xd.z, g.ratio[2], g.n[2]);
#pragma unroll 1
        for (int col = blockIdx.y; col < 13; col += gridDim.y) {  // (0, 0), (0, 1), (0, 2), (1, -2) ... (2, 2)
            const int a = col < 3 ? 0 : 1 + (col - 3) / 5, b = col < 3 ? col : (col - 3) % 5 - 2;
            int na = ca + a, nb = cb + b;
            const int ia = na >= g.n[0] ? 1 : 0, ib = nb < 0 ? -1 : (nb >= g.n[1] ? 1 : 0);
            na -= ia * g.n[0];
            nb -= ib * g.n[1];
            const int c0 = g.flat(na, nb, 0);
            const float2 sx = make_float2(xi - ia * f.Lf.x, xi - ia * f.Lf.x), sy = make_float2(yi - ib * f.Lf.y, yi - ib * f.Lf.y);
            // the cells below the wrap, those in place, those above the wrap
#pragma unroll 1
            for (int part = col > 0 && cc < 2 ? -1 : 0; part <= (cc + 2 >= nz ? 1 : 0); ++part) {
                const int z0 = part < 0 ? nz + cc - 2 : (part > 0 ? 0 : (col > 0 ? max(cc - 2, 0) : cc));
                const int z1 = part < 0 ? nz - 1 : (part > 0 ? cc + 2 - nz : min(cc + 2, nz - 1));
                const int js = col == 0 && part == 0 ? i + 1 : start[c0 + z0], je = start[c0 + z1 + 1];
                const float2 sz = make_float2(zi - part * f.Lf.z, zi - part * f.Lf.z);
                unsigned valid = kAll << (js & 3);  // candidates of the block, first lowest
                for (int j0 = js & ~3; j0 < je; j0 += kStep) {
                    if (je - j0 < kStep) valid &= (1u << (je - j0)) - 1u;
                    unsigned exact = 0;
                    auto pair = [&](int t, float r2) {
                        if (r2 < f.outer2 && (valid & (1u << t)) != 0) {
                            float r;
                            asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(r2));
                            const float x = r * f.inv_dr;
                            const float big = __fadd_rd(x, 8388608.0f);           // 2^23 + floor(x)
                            const float off = fabsf(x - (big - 8388607.5f));      // from the bin's middle
                            if (off < f.half && big < f.end)
                                atomicAdd(sh + (__float_as_uint(big) & 0x7fffffu), 2u);
                            else
                                exact |= 1u << t;
                        }
                    };
#pragma unroll
                    for (int t = 0; t < kStep; t += 4) {
                        const float4 qx = ld_four<true>(px + j0 + t), qy = ld_four<true>(py + j0 + t), qz = ld_four<true>(pz + j0 + t);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float2 dx = __fadd2_rn(sx, h ? make_float2(qx.z, qx.w) : make_float2(qx.x, qx.y));
                            const float2 dy = __fadd2_rn(sy, h ? make_float2(qy.z, qy.w) : make_float2(qy.x, qy.y));
                            const float2 dz = __fadd2_rn(sz, h ? make_float2(qz.z, qz.w) : make_float2(qz.x, qz.y));
                            const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                            pair(t + 2 * h, r2.x);
                            pair(t + 2 * h + 1, r2.y);
                        }
                    }
                    valid = kAll;
                    while (exact) {
                        const int t = __ffs(exact) - 1;
                        exact &= exact - 1;
                        rdf_count<2u>(xd, sorted[j0 + t], pp, rmax2, inv_dr, nbins, sh);
                    }
                }
            }
        }
    }
    flush(sh, nbins, hist);
}

// A position outside the box, wrapped into it.
__device__ __noinline__ double4 wrapped(double4 x, double3 L) {
    return make_double4(wrap(x.x, L.x), wrap(x.y, L.y), wrap(x.z, L.z), 0.0);
}

// Cell of each atom and its arrival rank (`count` is zero before and, after the
// scan, again); `clear` (may be null): a histogram to start from zero.  Cells, images
// and the FP32 test's error bound are those of positions in [0, L], but a caller's may lie
// outside: those are binned where they wrap to, and their cell is left complemented
// for rdf_place_kernel.  (Every atom compared with the box in both kernels: 1.2 us more
// at 100 003 atoms.)
__global__ void rdf_bin_kernel(int N, const double4* __restrict__ pos, double3 L, Grid g, int* __restrict__ cell_of,
                               int* __restrict__ rank, int* __restrict__ count, unsigned long long* clear, int nbins) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (clear)
        for (int b = i; b < nbins; b += gridDim.x * blockDim.x) clear[b] = 0ull;
    if (i >= N) return;
    double4 x = pos[i];
    const double fx = floor(__dmul_rn(x.x, g.ratio[0])), fy = floor(__dmul_rn(x.y, g.ratio[1])),
                 fz = floor(__dmul_rn(x.z, g.ratio[2]));
    int ca = (int)fx, cb = (int)fy, cc = (int)fz;
    bool out = false;
    if ((unsigned)ca >= (unsigned)g.n[0] || (unsigned)cb >= (unsigned)g.n[1] || (unsigned)cc >= (unsigned)g.n[2]) {
        // (a coordinate of L exactly belongs to the last cell)
        out = fx < 0.0 || fy < 0.0 || fz < 0.0 || x.x > L.x || x.y > L.y || x.z > L.z;
        if (out) x = wrapped(x, L);
        ca = cell_coord(x.x, g.ratio[0], g.n[0]);
        cb = cell_coord(x.y, g.ratio[1], g.n[1]);
        cc = cell_coord(x.z, g.ratio[2], g.n[2]);
    }
    const int c = g.flat(ca, cb, cc);
    cell_of[i] = out ? ~c : c;
    rank[i] = atomicAdd(&count[c], 1);
}

// Exclusive scan of up to a few tiles of counts by one block, which leaves them zero.
constexpr int kOneBlockCells = 8 * kScanTile;

__global__ void __launch_bounds__(1024)
rdf_scan_kernel(int* __restrict__ count, int n, int* __restrict__ start) {
    __shared__ int tot;
    int base = 0;
    for (int t0 = 0; t0 < n; t0 += kScanTile) {
        const int idx = t0 + 4 * threadIdx.x;
        int c[4], sum = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            c[q] = idx + q < n ? count[idx + q] : 0;
            sum += c[q];
        }
        int ex = block_exclusive_scan<1024>(sum, &tot) + base;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (idx + q < n) {
                start[idx + q] = ex;
                count[idx + q] = 0;
            }
            ex += c[q];
        }
        base += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) start[n] = base;
}

__global__ void rdf_place_kernel(int N, const double4* __restrict__ pos, double3 L, const int* __restrict__ cell_of,
                                 const int* __restrict__ rank, const int* __restrict__ start,
                                 double4* __restrict__ sorted, PosNeg posn) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    int c = cell_of[i];
    double4 x = pos[i];
    if (c < 0) {
        c = ~c;
        x = wrapped(x, L);
    }
    const int k = start[c] + rank[i];
    sorted[k] = x;
    if (posn.p) posn.set(k, x);
}

constexpr int kRdfRounds = 4;  // blocks, in times what the GPU holds

// Rounds of atoms after which a block's 32-bit counts are added up: an atom counts each
// of the others once, by two (beyond 2^24 atoms every round, as the blocks of the other
// forms, which have one).
int rdf_rounds(int N) {
    const double most = 4294967295.0 / (2.0 * kThreads * (double)N);
    return most < 1.0 ? 1 : (int)std::min(most, 1e9);
}

// Error bound of the FP32 distance of two atoms in box L: coordinates and box edges
// rounded (2^-24 L each), the image shift's subtraction (2^-24 2 L), over three
// axes, and the evaluation of r itself.
double rdf_error(const double L[3], double rmax) {
    const double Lmax = std::max(L[0], std::max(L[1], L[2]));
    return std::ldexp(12.0 * Lmax + 16.0 * rmax, -24);
}

}  // namespace

Grid rdf_grid(const double L[3], double rmax, long long max_cells) {
    // floor(L / rmax) in double: a tiny rmax gives a huge count, not an int overflow
    double n[3];
    for (int k = 0; k < 3; ++k) n[k] = std::max(1.0, std::floor(L[k] / rmax));
    double prod = n[0] * n[1] * n[2];
    if (prod > (double)max_cells) {
        double f = std::cbrt((double)max_cells / prod);
        for (int k = 0; k < 3; ++k) n[k] = std::max(1.0, std::floor(n[k] * f));
        while (n[0] * n[1] * n[2] > (double)max_cells) {
            int k = n[0] >= n[1] ? (n[0] >= n[2] ? 0 : 2) : (n[1] >= n[2] ? 1 : 2);
            n[k] -= 1.0;
        }
    }
    Grid g;
    for (int k = 0; k < 3; ++k) {
        g.n[k] = (int)n[k];
        g.ratio[k] = (double)g.n[k] / L[k];
    }
    return g;
}

RdfPlan rdf_plan(const double L[3], int nbins, double rmax, long long max_cells) {
    RdfPlan p;
    p.g = rdf_grid(L, rmax, max_cells);
    p.cells = p.g.n[0] >= 3 && p.g.n[1] >= 3 && p.g.n[2] >= 3;
    // bins at least 20 error bounds wide (the exact arithmetic decides one pair in ten
    // there), and a stencil of +-2 cells of half the edge
    if (p.cells && rdf_error(L, rmax) * nbins <= 0.05 * rmax) {
        const Grid h = rdf_grid(L, 0.5 * rmax, max_cells);
        p.fast = h.n[0] >= 5 && h.n[1] >= 5 && h.n[2] >= 5;
        if (p.fast) p.g = h;
    }
    return p;
}

int rdf_enqueue(int N, const double4* pos, const PairParams& pp, const RdfPlan& plan, int nbins, double rmax,
                const RdfScratch& s, unsigned long long* hist, bool clear, cudaStream_t stream, long long* launches) {
    double rmax2 = rmax * rmax, inv_dr = (double)nbins / rmax;
    size_t shm = sizeof(unsigned) * nbins;
    int blocks = (N + kThreads - 1) / kThreads;
    const Grid& g = plan.g;
    if (!plan.cells) {
        if (clear && cudaMemsetAsync(hist, 0, sizeof(unsigned long long) * nbins, stream) != cudaSuccess) return 2;
        // slices until the GPU has a few blocks per SM
        const dim3 grid(blocks, std::max(1, std::min(64, 1024 / blocks)));
        rdf_all_pairs_kernel<<<grid, kThreads, shm, stream>>>(N, pos, pp, rmax2, inv_dr, nbins, hist);
        ++*launches;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }
    int nc = g.ncell();
    const double3 L = make_double3(pp.L[0], pp.L[1], pp.L[2]);
    Gate open{};
    open.always = 1;
    rdf_bin_kernel<<<blocks, kThreads, 0, stream>>>(N, pos, L, g, s.cell_of, s.rank, s.count, clear ? hist : nullptr, nbins);
    if (nc <= kOneBlockCells) {
        rdf_scan_kernel<<<1, 1024, 0, stream>>>(s.count, nc, s.start);
        *launches += 4;
    } else {
        int ntiles = (nc + kScanTile - 1) / kScanTile;
        scan_reduce_kernel<false><<<ntiles, 1024, 0, stream>>>(s.count, nc, s.tiles, open);
        scan_tiles_kernel<false><<<1, 1024, 0, stream>>>(s.tiles, ntiles, open);
        scan_apply_kernel<false><<<ntiles, 1024, 0, stream>>>(s.count, nc, s.tiles, s.start, open);
        *launches += 6;
    }
    const PosNeg posn{plan.fast ? s.posn : nullptr, PosNeg::stride(N)};
    rdf_place_kernel<<<blocks, kThreads, 0, stream>>>(N, pos, L, s.cell_of, s.rank, s.start, s.sorted, posn);
    if (plan.fast) {
        const double E = rdf_error(pp.L, rmax), d = E * inv_dr;
        RdfFast f;
        f.outer2 = (float)((rmax + E) * (rmax + E) * (1.0 + 1e-6));
        f.inv_dr = (float)inv_dr;
        f.half = (float)(0.5 - d);
        f.end = 8388608.0f + (float)nbins;
        f.Lf = make_float3((float)pp.L[0], (float)pp.L[1], (float)pp.L[2]);
        // small systems: an atom's columns on several threads, until the GPU is full a few
        // times over; large ones: blocks stay for several rounds of atoms, so that the
        // histograms are added up once each
        const int most = kRdfRounds * 148 * 6, slices = std::max(1, std::min(13, most / blocks));
        rdf_fast_kernel<<<dim3(std::min(blocks, most / slices), slices), kThreads, shm, stream>>>(
            N, s.sorted, posn, g, s.start, pp, rmax2, inv_dr, nbins, f, rdf_rounds(N), hist);
    } else {
        rdf_cells_kernel<<<blocks, kThreads, shm, stream>>>(N, s.sorted, g, s.start, pp, rmax2, inv_dr, nbins, hist);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int rdf_set_smem(int nbins) {
    size_t shm = sizeof(unsigned) * nbins;
    if (shm <= 48 * 1024) return 0;
    if (cudaFuncSetAttribute(rdf_fast_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm) != cudaSuccess ||
        cudaFuncSetAttribute(rdf_cells_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm) != cudaSuccess ||
        cudaFuncSetAttribute(rdf_all_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm) !=
            cudaSuccess)
        return 2;
    return 0;
}

int rdf_reserve(RdfScratch& s, int N, int ncell, int nbins) {
    if (N > s.atoms) {
        cudaFree(s.cell_of);
        cudaFree(s.rank);
        cudaFree(s.sorted);
        cudaFree(s.posn);
        s.cell_of = s.rank = nullptr;
        s.sorted = nullptr;
        s.posn = nullptr;
        s.atoms = 0;
        if (cudaMalloc(&s.cell_of, sizeof(int) * N) != cudaSuccess ||
            cudaMalloc(&s.rank, sizeof(int) * N) != cudaSuccess ||
            cudaMalloc(&s.sorted, sizeof(double4) * N) != cudaSuccess ||
            cudaMalloc(&s.posn, sizeof(float) * 3 * (size_t)PosNeg::stride(N)) != cudaSuccess ||
            cudaMemset(s.posn, 0, sizeof(float) * 3 * (size_t)PosNeg::stride(N)) != cudaSuccess ||
            cudaStreamSynchronize(nullptr) != cudaSuccess)
            return 2;
        s.atoms = N;
    }
    if (ncell > s.cells) {
        cudaFree(s.count);
        cudaFree(s.start);
        s.count = s.start = nullptr;
        s.cells = 0;
        // the counts are zero between samples
        if (cudaMalloc(&s.count, sizeof(int) * ncell) != cudaSuccess ||
            cudaMalloc(&s.start, sizeof(int) * (ncell + 1)) != cudaSuccess ||
            cudaMemset(s.count, 0, sizeof(int) * ncell) != cudaSuccess || cudaStreamSynchronize(nullptr) != cudaSuccess)
            return 2;
        s.cells = ncell;
    }
    if (!s.tiles && cudaMalloc(&s.tiles, sizeof(int) * kMaxScanTiles) != cudaSuccess) return 2;
    if (nbins > s.bins) {
        unsigned long long* h = nullptr;
        if (cudaMalloc(&h, sizeof(unsigned long long) * 2 * (size_t)nbins) != cudaSuccess) return 2;
        // a running accumulation moves to the new buffer (rare: a larger
        // single sample taken in the middle of an accumulation)
        // (the samples were enqueued on a non-blocking stream: wait for the device first)
        if (s.samples > 0 &&
            (cudaDeviceSynchronize() != cudaSuccess ||
             cudaMemcpy(h, s.hist, sizeof(unsigned long long) * s.acc_bins, cudaMemcpyDeviceToDevice) != cudaSuccess)) {
            cudaFree(h);
            return 2;
        }
        cudaFree(s.hist);
        s.hist = h;
        s.bins = nbins;
    }
    return 0;
}

void rdf_release(RdfScratch& s) {
    void* ptrs[] = {s.cell_of, s.rank, s.count, s.start, s.tiles, s.sorted, s.posn, s.hist};
    for (void* q : ptrs)
        if (q) cudaFree(q);
    s = RdfScratch{};
}

}  // namespace ljb

namespace ljb {

// ---------------------------------------------------------------------------
// Allocation-free RDF entry point.
//
// For callers that may not call cudaMalloc: an application whose GPU memory is
// owned by its own pool allocator (a deep-learning framework, for instance,
// whose caching allocator must see every allocation), or a per-step analysis
// hook in a time-critical loop, where cudaMalloc's latency and the implicit
// device-wide synchronisation that cudaMalloc/cudaFree can cause are not
// acceptable.  They pass device buffers they already own for the positions and
// the histogram; the cell-list scratch comes from the fixed device array below.
//
// The array is a file-scope __device__ variable: every GPU that loads this
// library holds it (about 6.9 MB) until the process exits.  All calls on a
// device share it and it keeps the last call's contents; each call leaves the cell
// counts at zero, as it found them, and clears the output histogram on its stream.
// (Calls that overlapped do so too, once all are done: each call's scan clears every
// count that its binning, before it, can have touched.  One whose launches fail between
// the two does not: the next call clears them first, which on every call would cost
// 3.4 us, 98.5 -> 101.9 us at 100 003 atoms.)
// Calls whose work overlaps on the GPU (different streams, or several host
// threads) race on the shared array: serialise them.
// ---------------------------------------------------------------------------

namespace {

constexpr int kNoAllocMaxAtoms = 131072;
constexpr int kNoAllocMaxCells = 32768;
constexpr int kNoAllocMaxBins = 12288;  // 48 KB shared-memory histogram, no attribute change needed
constexpr size_t kOffSorted = 0;
constexpr size_t kOffCellOf = kOffSorted + sizeof(double4) * kNoAllocMaxAtoms;
constexpr size_t kOffRank = kOffCellOf + sizeof(int) * kNoAllocMaxAtoms;
constexpr size_t kOffCount = kOffRank + sizeof(int) * kNoAllocMaxAtoms;
constexpr size_t kOffStart = kOffCount + sizeof(int) * kNoAllocMaxCells;
constexpr size_t kOffTiles = kOffStart + sizeof(int) * (kNoAllocMaxCells + 256);
constexpr size_t kOffPosn = kOffTiles + sizeof(int) * kMaxScanTiles;
constexpr size_t kNoAllocBytes = kOffPosn + sizeof(float) * 3 * (kNoAllocMaxAtoms + 2 * kPosPad);
static_assert(kOffCellOf % 256 == 0 && kOffRank % 256 == 0 && kOffCount % 256 == 0 &&
              kOffStart % 256 == 0 && kOffTiles % 256 == 0 && kOffPosn % 256 == 0, "scratch sub-buffers must stay aligned");

__device__ __align__(256) unsigned char g_rdf_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
std::atomic<unsigned char*> g_scratch_addr[kMaxDevices];
std::atomic<bool> g_scratch_unclean[kMaxDevices];  // a call's launches failed: the counts may not be zero

// Device address of g_rdf_scratch on the current device, looked up on the
// first call on each device and cached for the life of the process.  A
// cudaDeviceReset (or anything else that destroys and recreates the device's
// primary context) reloads the module and may move the array: the cached
// address is then stale, so a process that resets a device must not call
// lj_gpu_rdf_noalloc on it afterwards.
int scratch_address(unsigned char** out, int& dev) {
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 2;
    unsigned char* p = g_scratch_addr[dev].load();
    if (!p) {
        void* q = nullptr;
        if (cudaGetSymbolAddress(&q, g_rdf_scratch) != cudaSuccess || !q) return 2;
        p = static_cast<unsigned char*>(q);
        g_scratch_addr[dev].store(p);
    }
    *out = p;
    return 0;
}

}  // namespace

}  // namespace ljb

extern "C" int lj_gpu_rdf_noalloc(const double* pos, int N, const double* box, int nbins, double rmax,
                                  unsigned long long* hist, void* stream_handle) {
    using namespace ljb;
    if (!pos || !box || !hist || N < 1 || nbins < 1 || !(rmax > 0)) return 1;  // LJ_ERR_ARG
    if (N > kNoAllocMaxAtoms || nbins > kNoAllocMaxBins) return 1;
    // double4 position loads need 16-byte alignment, the 64-bit histogram atomics 8
    if ((reinterpret_cast<uintptr_t>(pos) & 15) != 0 || (reinterpret_cast<uintptr_t>(hist) & 7) != 0) return 1;
    PairParams pp{};
    for (int k = 0; k < 3; ++k) {
        if (!(box[k] > 0) || !std::isfinite(box[k]) || rmax > 0.5 * box[k]) return 1;
        pp.L[k] = box[k];
        pp.halfL[k] = 0.5 * box[k];
    }
    // cells of edge >= rmax, coarser where the box holds more than the array's
    // kNoAllocMaxCells of them (the histogram does not depend on the cell size)
    const RdfPlan plan = rdf_plan(pp.L, nbins, rmax, kNoAllocMaxCells);
    unsigned char* base = nullptr;
    int dev = 0;
    if (scratch_address(&base, dev)) return 2;  // LJ_ERR_CUDA
    RdfScratch sc{};
    sc.sorted = reinterpret_cast<double4*>(base + kOffSorted);
    sc.cell_of = reinterpret_cast<int*>(base + kOffCellOf);
    sc.rank = reinterpret_cast<int*>(base + kOffRank);
    sc.count = reinterpret_cast<int*>(base + kOffCount);
    sc.start = reinterpret_cast<int*>(base + kOffStart);
    sc.tiles = reinterpret_cast<int*>(base + kOffTiles);
    sc.posn = reinterpret_cast<float*>(base + kOffPosn);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_handle);
    long long launches = 0;
    std::atomic<bool>& unclean = g_scratch_unclean[dev];
    if (unclean.load()) {
        if (cudaMemsetAsync(sc.count, 0, sizeof(int) * kNoAllocMaxCells, stream) != cudaSuccess) return 2;
        unclean.store(false);
    }
    const int rc = rdf_enqueue(N, reinterpret_cast<const double4*>(pos), pp, plan, nbins, rmax, sc, hist, true, stream,
                               &launches);
    if (rc) unclean.store(true);
    return rc;
}
