// lj_kernels.cuh -- kernels of the single-system engine (FP64 drop-in path and
// the shared binning / neighbour-list machinery).
//
// Device layout (HBM), all in cell-sorted slot order and re-sorted at every
// neighbour-list build:
//   pos   double4[N]       x, y, z, 0 -- gathered by neighbours, one 32-byte sector each
//   soa   double[9][N]     vx vy vz | dx dy dz (displacement) | fx fy fz, coalesced per atom
//   ids   int[N]           slot -> atom id (the reference's column index)
//   bd    double[3][N]     displacement at the last list build (skin criterion)
//   nbr   uint32[cap][N]   neighbour list, transposed so entry k of all atoms is contiguous;
//                          slot << 6 | code (the list kernels below)
//   cnt   int[N]           neighbour count
#pragma once

#include <cuda.h>

#include "lj_common.cuh"

namespace ljb {

enum SoaField { VX = 0, VY, VZ, DX, DY, DZ, FX, FY, FZ, SOA_FIELDS };

struct Soa {
    double* p;
    int N;
    __device__ __forceinline__ double& at(int f, int i) const { return p[(size_t)f * N + i]; }
};

// FP32 copy of the positions for the list builds, negated and by component, so
// that four candidates are one 16-byte load per axis and go into packed
// arithmetic as they come.  Components are `np` floats apart: the slots and some
// padding, which may be read but never counts.
constexpr int kPosPad = 32;

struct PosNeg {
    float* p;
    int np;
    __host__ __device__ static int stride(int n) { return (n + 2 * kPosPad) & ~(kPosPad - 1); }
    __device__ __forceinline__ void set(int i, const double4& x) const {
        p[i] = -(float)x.x;
        p[np + i] = -(float)x.y;
        p[2 * (size_t)np + i] = -(float)x.z;
    }
    __device__ __forceinline__ float3 at(int i) const { return make_float3(p[i], p[np + i], p[2 * (size_t)np + i]); }
};

// Rebuild gate: evaluated identically by every kernel of the rebuild chain.
struct Gate {
    const Scalars* sc;
    double thresh2;  // rebuild when max |d - d_build|^2 exceeds this
    int always;      // small-box / zero-skin mode: rebuild every step
    __device__ __forceinline__ bool open() const {
        if (always || sc->need_rebuild) return true;
        return __longlong_as_double((long long)sc->max_disp2) > thresh2;
    }
};

// ---------------------------------------------------------------------------
// Integration: integrator.cpp:62-88, first half (kick, drift, displacement, wrap)
// ---------------------------------------------------------------------------
template <bool PERIODIC, bool TRACK, bool LOCAL>
static __global__ void __launch_bounds__(kThreads)
kick_drift_kernel(int N, const double4* pos, double4* pos_out, Soa s, const double* __restrict__ bd,
                  const double* __restrict__ bx, float4* __restrict__ posl, PairParams pp, Scalars* sc) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double m = 0.0;
    if (i < N) {
        double4 x = pos[i];
        double xs[3] = {x.x, x.y, x.z};
        float l[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double v = kick(s.at(VX + k, i), s.at(FX + k, i), pp.dt);
            double inc = __dmul_rn(v, pp.dt);
            double xn = __dadd_rn(xs[k], inc);
            double dn = __dadd_rn(s.at(DX + k, i), inc);
            if (PERIODIC) xn = wrap(xn, pp.L[k]);
            s.at(VX + k, i) = v;
            s.at(DX + k, i) = dn;
            xs[k] = xn;
            if (TRACK || LOCAL) {
                double e = dn - bd[(size_t)k * N + i];
                m = fma(e, e, m);
                // mixed path: cell-local FP32 coordinate xl = bx + (d - d_build)
                if (LOCAL) l[k] = (float)(bx[(size_t)k * N + i] + e);
            }
        }
        pos_out[i] = make_double4(xs[0], xs[1], xs[2], 0.0);
        if (LOCAL) posl[i] = make_float4(l[0], l[1], l[2], 0.f);
    }
    if (TRACK) {
        m = warp_max(m);
        if ((threadIdx.x & 31) == 0 && m > 0.0)
            atomicMax(&sc->max_disp2, (unsigned long long)__double_as_longlong(m));
    }
}

// Second half kick without a force calculation (LJ_FORCE_NONE), with the
// measurement partial sums.
static __global__ void __launch_bounds__(kThreads)
kick_measure_kernel(int N, Soa s, double dt, int do_kick, double* __restrict__ partials) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[4] = {0, 0, 0, 0};
    if (i < N) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double v = s.at(VX + k, i);
            if (do_kick) {
                v = kick(v, s.at(FX + k, i), dt);
                s.at(VX + k, i) = v;
            }
            acc[0] = fma(v, v, acc[0]);
            double d = s.at(DX + k, i);
            acc[3] = fma(d, d, acc[3]);
        }
    }
    block_sum<4, kThreads>(acc);
    if (threadIdx.x == 0)
        for (int q = 0; q < 4; ++q) partials[(size_t)blockIdx.x * 4 + q] = acc[q];
}

// ---------------------------------------------------------------------------
// Cell binning (counting sort): particle_pair_filter.cpp:141-154
// ---------------------------------------------------------------------------
template <bool GATED>
static __global__ void __launch_bounds__(kThreads)
bin_count_kernel(int N, const double4* __restrict__ pos, Grid g, int* __restrict__ cell_of,
                 int* __restrict__ rank, int* __restrict__ count, Gate gate) {
    if (GATED && !gate.open()) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    double4 x = pos[i];
    int c = g.flat(cell_coord(x.x, g.ratio[0], g.n[0]), cell_coord(x.y, g.ratio[1], g.n[1]),
                   cell_coord(x.z, g.ratio[2], g.n[2]));
    cell_of[i] = c;
    rank[i] = atomicAdd(&count[c], 1);
}

// Exclusive scan of count[0..n) into start[0..n]: tile sums, scan of tile sums, apply.
template <bool GATED>
static __global__ void __launch_bounds__(1024)
scan_reduce_kernel(const int* __restrict__ count, int n, int* __restrict__ tile_sums, Gate gate) {
    if (GATED && !gate.open()) return;
    int base = blockIdx.x * kScanTile + threadIdx.x * 4;
    int s = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) s += base + q < n ? count[base + q] : 0;
    __shared__ int tot;
    block_exclusive_scan<1024>(s, &tot);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

template <bool GATED>
static __global__ void __launch_bounds__(1024)
scan_tiles_kernel(int* __restrict__ tile_sums, int ntiles, Gate gate) {
    if (GATED && !gate.open()) return;
    int x = threadIdx.x < ntiles ? tile_sums[threadIdx.x] : 0;
    __shared__ int tot;
    int ex = block_exclusive_scan<1024>(x, &tot);
    if (threadIdx.x < ntiles) tile_sums[threadIdx.x] = ex;
}

template <bool GATED>
static __global__ void __launch_bounds__(1024)
scan_apply_kernel(int* __restrict__ count, int n, const int* __restrict__ tile_sums,
                  int* __restrict__ start, Gate gate) {
    if (GATED && !gate.open()) return;
    int base = blockIdx.x * kScanTile + threadIdx.x * 4;
    int c[4];
    int s = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        c[q] = base + q < n ? count[base + q] : 0;
        s += c[q];
    }
    __shared__ int tot;
    int ex = block_exclusive_scan<1024>(s, &tot) + tile_sums[blockIdx.x];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (base + q < n) {
            start[base + q] = ex;
            count[base + q] = 0;  // ready for the next binning
        }
        ex += c[q];
    }
    if (base < n && base + 4 >= n) start[n] = ex;
}

template <bool GATED>
static __global__ void __launch_bounds__(kThreads)
scatter_kernel(int N, const int* __restrict__ cell_of, const int* __restrict__ rank,
               const int* __restrict__ start, int* __restrict__ order, Gate gate) {
    if (GATED && !gate.open()) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    order[start[cell_of[i]] + rank[i]] = i;
}

// Order each cell's members by their previous slot.  Slots come from the last
// sort, so the order is a fixed function of the trajectory and every run is
// bit-reproducible without reading atom ids.  (The reference's own cell
// contents, ascending atom id, are produced by lj_gpu_debug_cells.)
// One warp per cell: cells of up to 32 atoms are sorted in registers by a
// bitonic network over warp shuffles; larger cells (rare) by one lane.
constexpr int kSortWarps = 4;

template <bool GATED>
static __global__ void __launch_bounds__(32 * kSortWarps)
cell_sort_kernel(int ncell, const int* __restrict__ start, int* __restrict__ order, Gate gate) {
    if (GATED && !gate.open()) return;
    int lane = threadIdx.x & 31;
    int c = blockIdx.x * kSortWarps + (threadIdx.x >> 5);
    if (c >= ncell) return;
    int b = start[c], e = start[c + 1], n = e - b;
    if (n <= 1) return;
    if (n <= 32) {
        int v = lane < n ? order[b + lane] : 0x7fffffff;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                int o = __shfl_xor_sync(0xffffffffu, v, j);
                bool up = (lane & k) == 0, lower = (lane & j) == 0;
                v = (lower == up) ? min(v, o) : max(v, o);
            }
        if (lane < n) order[b + lane] = v;
        return;
    }
    if (lane == 0)
        for (int k = b + 1; k < e; ++k) {
            int v = order[k], q = k - 1;
            while (q >= b && order[q] > v) {
                order[q + 1] = order[q];
                --q;
            }
            order[q + 1] = v;
        }
}

// Gather the state into sorted order (into the scratch copies).  The forces move only
// when asked: within a step they have been used up before the rebuild and are
// about to be computed anew.
template <bool FORCES>
static __global__ void __launch_bounds__(kThreads)
gather_kernel(int N, const int* __restrict__ order, const double4* __restrict__ pos,
              double4* __restrict__ pos_out, Soa s, Soa s_out, const int* __restrict__ ids,
              int* __restrict__ ids_out, double* __restrict__ bd, Gate gate) {
    if (!gate.open()) return;
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    int o = order[k];
    pos_out[k] = pos[o];
#pragma unroll
    for (int f = 0; f < (FORCES ? SOA_FIELDS : FX); ++f) {
        const double v = s.at(f, o);
        s_out.at(f, k) = v;
        if (f >= DX && f < DX + 3) bd[(size_t)(f - DX) * N + k] = v;
    }
    ids_out[k] = ids[o];
}

// Copy the sorted state back and write the FP32 position copy used by the list build
// and, for the mixed path (LOCAL), the position relative to the atom's list cell.
template <bool FORCES, bool LOCAL>
static __global__ void __launch_bounds__(kThreads)
copy_back_kernel(int N, const double4* __restrict__ pos_in, double4* __restrict__ pos, Soa s_in,
                 Soa s, const int* __restrict__ ids_in, int* __restrict__ ids, PosNeg posn, Grid g,
                 double* __restrict__ bx, float4* __restrict__ posl, Gate gate) {
    if (!gate.open()) return;
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    double4 x = pos_in[k];
    pos[k] = x;
    posn.set(k, x);
#pragma unroll
    for (int f = 0; f < (FORCES ? SOA_FIELDS : FX); ++f) s.at(f, k) = s_in.at(f, k);
    ids[k] = ids_in[k];
    if (LOCAL) {
        const double xs[3] = {x.x, x.y, x.z};
        float l[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int c = cell_coord(xs[q], g.ratio[q], g.n[q]);
            const double o = (double)c * (1.0 / g.ratio[q]);
            const double b = xs[q] - o;
            bx[(size_t)q * N + k] = b;
            l[q] = (float)b;
        }
        posl[k] = make_float4(l[0], l[1], l[2], 0.f);
    }
}

// Neighbour list over the 27-cell stencil of the list grid.
//
// Layout: groups of 4 entries, group g of atom i at nbr4[g * N + i] (one 16-byte
// load per group, coalesced across a warp); the tail of the last group is
// padded with the ghost slot N, which sits far outside every box.  An entry is
// slot << 6 | code, the code the lattice image in boxes under 3 cells per axis
// (SMALL, rebuilt every step), otherwise the stencil offset (the pair kernels
// recompute the minimum image each step).
//
// The candidate test runs in FP32 on box coordinates against a radius widened
// by 8 * L * 2^-24, so the list is a superset of the FP64 pair set; the pair
// kernels apply the exact test.
//
// This kernel builds the lists of boxes under 3 cells per axis.
static __global__ void __launch_bounds__(kThreads)
build_small_list_kernel(int N, const double4* __restrict__ pos, PosNeg posn, Grid g, const int* __restrict__ start,
                        float3 Lf, float cut2, int cap, uint4* __restrict__ nbr4, int* __restrict__ cnt, Scalars* sc,
                        Gate gate) {
    if (!gate.open()) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = 0;
    unsigned* nbr = reinterpret_cast<unsigned*>(nbr4);
    if (i < N) {
        const float3 xi = posn.at(i);  // negated, as the candidates
        // the home cell comes from the FP64 position, exactly as the binning placed the atom
        double4 xd = pos[i];
        int ci[3] = {cell_coord(xd.x, g.ratio[0], g.n[0]), cell_coord(xd.y, g.ratio[1], g.n[1]),
                     cell_coord(xd.z, g.ratio[2], g.n[2])};
        for (int a = -1; a <= 1; ++a) {
            int na = ci[0] + a, ia = na < 0 ? -1 : (na >= g.n[0] ? 1 : 0);
            na -= ia * g.n[0];
            for (int b = -1; b <= 1; ++b) {
                int nb = ci[1] + b, ib = nb < 0 ? -1 : (nb >= g.n[1] ? 1 : 0);
                nb -= ib * g.n[1];
                for (int c = -1; c <= 1; ++c) {
                    int nc = ci[2] + c, ic = nc < 0 ? -1 : (nc >= g.n[2] ? 1 : 0);
                    nc -= ic * g.n[2];
                    int cell = g.flat(na, nb, nc);
                    float sx = ia * Lf.x, sy = ib * Lf.y, sz = ic * Lf.z;
                    unsigned code = offset_code(ia, ib, ic);
                    int e = start[cell + 1];
                    for (int j = start[cell]; j < e; ++j) {
                        const float3 xj = posn.at(j);
                        float dx = (xj.x - xi.x) - sx;
                        float dy = (xj.y - xi.y) - sy;
                        float dz = (xj.z - xi.z) - sz;
                        if (fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < cut2 && j != i) {
                            if (n < cap) nbr[((size_t)(n >> 2) * N + i) * 4 + (n & 3)] = make_entry((unsigned)j, code);
                            ++n;
                        }
                    }
                }
            }
        }
        int m = n < cap ? n : cap;
        cnt[i] = m;
        for (int k = m; k < ((m + 3) & ~3); ++k)  // ghost padding (no image, no offset)
            nbr[((size_t)(k >> 2) * N + i) * 4 + (k & 3)] = make_entry((unsigned)N, kGhostCode);
    }
    // block max of n -> sc->max_count; overflow flag
    int m = n;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&sc->max_count, m);
        if (m > cap) atomicExch(&sc->overflow, 1);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd((unsigned long long*)&sc->builds, 1ull);
}

template <bool NC>
__device__ __forceinline__ float4 ld_four(const float* p) {
    float4 r;
    if (NC)
        r = __ldg(reinterpret_cast<const float4*>(p));
    else
        asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
    return r;
}

// Lists on grids of >= 3 cells per axis (the minimum-image form) are built a warp
// per cell (build_cell_lists) or, where a cell would leave most of a warp's lanes
// without an atom, an atom per lane (build_atom_lists); entries and order (stencil
// cell, then slot) are the same.
//
// In both, every candidate's entry is stored to shared memory under a predicate
// and the store's address stepped under the same: no lane waits for another's
// hits, and an entry costs two instructions of every lane, hit or not, where a
// loop over the hits took 25 to 35 per round and as many rounds as the busiest lane
// has hits.  When a lane has no room for another block of candidates, all lanes
// send their whole groups to memory, 16 bytes a lane.
//
// Bound by issue (75 %) and by shared memory (77 % of the L1 data pipe: broadcast
// reads of candidates, predicated stores of entries).  Measured at 256 000 atoms,
// rho 0.8442, a list build by a warp per cell 153 -> 133 us, by an atom per lane 155
// us; a whole rebuild at 1 048 576 atoms 701 -> 610 us.  Thin systems gain most: the
// lists of 23 328 atoms at rho 0.46, beside 63 other systems in the resident launch,
// 967 -> 243 us.  The line between the two, kFullCell, is where their times in that
// launch cross (rho 0.46: 257 against 370 us per cell; rho 0.73: 222 against 208).
constexpr int kPend = 32;  // entries a lane may hold back
constexpr int kBlock = 8;  // candidates between two looks at the room left

struct ListPend {
    unsigned e[kPend][32];
};

// A lane's list on its way to memory.
struct ListWriter {
    static constexpr unsigned kRow = 32 * sizeof(unsigned);  // bytes between a lane's entries
    unsigned base, at;  // shared-memory addresses: of the lane's first entry, of the next
    int out = 0;        // entries sent to memory (whole groups)
    __device__ __forceinline__ explicit ListWriter(ListPend& p) {
        base = at = (unsigned)__cvta_generic_to_shared(&p.e[0][threadIdx.x & 31]);
    }
    static __device__ __forceinline__ void put(unsigned a, unsigned v) {
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
    }
    static __device__ __forceinline__ unsigned get(unsigned a) {
        unsigned v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
        return v;
    }
    __device__ __forceinline__ void append(bool hit, unsigned e) {
        if (hit) {
            put(at, e);
            at += kRow;
        }
    }
    __device__ __forceinline__ int count() const { return out + (int)((at - base) / kRow); }
    // send every lane's whole groups to memory (all lanes of the warp)
    __device__ __forceinline__ void flush(uint4* nbr4, int N, int i, int cap) {
        const int rows = (int)((at - base) / kRow), whole = rows & ~3;
        for (int k = 0; __any_sync(0xffffffffu, k < whole); k += 4)
            if (k < whole && out + k < cap) {
                const unsigned e = base + (unsigned)k * kRow;
                nbr4[(size_t)((out + k) >> 2) * N + i] = make_uint4(get(e), get(e + kRow), get(e + 2 * kRow), get(e + 3 * kRow));
            }
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (whole > 0 && whole + q < rows) put(base + q * kRow, get(base + (whole + q) * kRow));
        out += whole;
        at = base + (unsigned)(rows - whole) * kRow;
    }
    // flush if some lane has no room for another block
    __device__ __forceinline__ void make_room(uint4* nbr4, int N, int i, int cap) {
        if (__any_sync(0xffffffffu, at > base + (kPend - kBlock) * kRow)) flush(nbr4, N, i, cap);
    }
    // pad the last group with the ghost slot and send the rest; returns the list's
    // length before the cut at the capacity
    __device__ __forceinline__ int finish(bool own, uint4* nbr4, int* cnt, int N, int i, int cap) {
        int n = count();
        const int total = n;
        if (own) {
            cnt[i] = min(n, cap);
            for (; n & 3; ++n, at += kRow) put(at, make_entry((unsigned)N, kGhostCode));
        }
        flush(nbr4, N, i, cap);
        return total;
    }
};

// Shared memory of a warp that builds a cell's lists: 32 candidates and their entries.
struct __align__(16) CellSmem {
    float q[3][32];
    unsigned e[32];
    ListPend pend;
};

// One warp builds the lists of the atoms of list cell (ca, cb, cc), 32 at a time, one
// per lane.  `start` holds the slot ranges of the grid's cells (slots are global: N
// is the list stride and the ghost slot).  Atoms are stored cell by cell with z
// fastest, so the three stencil cells z - 1, z, z + 1 of each of the 9 stencil columns
// are one run of slots (two where the column wraps in z).  A run is staged 32
// candidates at a time, with their entries, and every lane tests them through
// broadcast reads, two per instruction with packed FP32 arithmetic.  Returns the
// largest list length of the warp's lanes (before the cut at the capacity).
// NC: start and the positions are not written by this launch.
template <bool NC>
__device__ __forceinline__ int build_cell_lists(int ca, int cb, int cc, const Grid& g, const int* start,
                                                const PosNeg& posn, float3 Lf, float cut2, int cap, uint4* nbr4,
                                                int* cnt, int N, CellSmem& sm, int lane) {
    auto first = [&](int c) { return NC ? __ldg(start + c) : start[c]; };
    auto load = [&](const float* p) { return NC ? __ldg(p) : *p; };
    const float* const px = posn.p;
    const float* const py = px + posn.np;
    const float* const pz = py + posn.np;
    const int nz = g.n[2], c = g.flat(ca, cb, cc);
    const int hs = first(c), he = first(c + 1);
    int wmax = 0;
    for (int h0 = hs; h0 < he; h0 += 32) {
        const int i = h0 + lane;
        const bool own = i < he;
        // a lane without an atom sits where nothing is near
        const float xi = own ? -load(px + i) : 3e18f, yi = own ? -load(py + i) : 3e18f, zi = own ? -load(pz + i) : 3e18f;
        ListWriter w(sm.pend);
#pragma unroll 1
        for (int col = 0; col < 9; ++col) {
            const int a = col / 3 - 1, b = col % 3 - 1;
            int na = ca + a, nb = cb + b;
            const int ia = na < 0 ? -1 : (na >= g.n[0] ? 1 : 0), ib = nb < 0 ? -1 : (nb >= g.n[1] ? 1 : 0);
            na -= ia * g.n[0];
            nb -= ib * g.n[1];
            const int c0 = g.flat(na, nb, 0);
            const float2 sx = make_float2(xi - ia * Lf.x, xi - ia * Lf.x), sy = make_float2(yi - ib * Lf.y, yi - ib * Lf.y);
            // the cell below the wrap, the cells in place, the cell above the wrap
#pragma unroll 1
            for (int part = cc == 0 ? -1 : 0; part <= (cc == nz - 1 ? 1 : 0); ++part) {
                const int z0 = part < 0 ? nz - 1 : (part > 0 ? 0 : max(cc - 1, 0));
                const int z1 = part < 0 ? nz - 1 : (part > 0 ? 0 : min(cc + 1, nz - 1));
                const int js = first(c0 + z0), je = first(c0 + z1 + 1);
                const unsigned code = offset_code(a, b, part != 0 ? part : z0 - cc);
                // slots from which the code is one and two z steps up
                const int up1 = z0 < z1 ? first(c0 + z0 + 1) : INT_MAX, up2 = z0 + 1 < z1 ? first(c0 + z0 + 2) : INT_MAX;
                const float2 sz = make_float2(zi - part * Lf.z, zi - part * Lf.z);
                auto test = [&](int t0, bool home, int self) {
#pragma unroll
                    for (int t = t0; t < t0 + kBlock; t += 4) {
                        const float4 qx = *reinterpret_cast<const float4*>(&sm.q[0][t]);
                        const float4 qy = *reinterpret_cast<const float4*>(&sm.q[1][t]);
                        const float4 qz = *reinterpret_cast<const float4*>(&sm.q[2][t]);
                        const uint4 qe = *reinterpret_cast<const uint4*>(&sm.e[t]);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float2 dx = __fadd2_rn(sx, h ? make_float2(qx.z, qx.w) : make_float2(qx.x, qx.y));
                            const float2 dy = __fadd2_rn(sy, h ? make_float2(qy.z, qy.w) : make_float2(qy.x, qy.y));
                            const float2 dz = __fadd2_rn(sz, h ? make_float2(qz.z, qz.w) : make_float2(qz.x, qz.y));
                            const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                            w.append(r2.x < cut2 && (!home || t + 2 * h != self), h ? qe.z : qe.x);
                            w.append(r2.y < cut2 && (!home || t + 2 * h + 1 != self), h ? qe.w : qe.y);
                        }
                    }
                    w.make_room(nbr4, N, i, cap);
                };
                for (int j0 = js; j0 < je; j0 += 32) {
                    const int n = min(32, je - j0), j = j0 + lane;
                    __syncwarp();
                    sm.q[0][lane] = lane < n ? load(px + j) : 1e18f;
                    sm.q[1][lane] = lane < n ? load(py + j) : 1e18f;
                    sm.q[2][lane] = lane < n ? load(pz + j) : 1e18f;
                    sm.e[lane] = make_entry((unsigned)j, code) + (j >= up1 ? 16u : 0u) + (j >= up2 ? 16u : 0u);
                    __syncwarp();
                    if (col == 4 && part == 0) {  // the run that holds the cell itself
                        for (int t0 = 0; t0 < n; t0 += kBlock) test(t0, true, i - j0);
                    } else {
#pragma unroll
                        for (int t0 = 0; t0 < 32; t0 += kBlock) {
                            if (t0 >= n) break;
                            test(t0, false, 0);
                        }
                    }
                }
            }
        }
        wmax = max(wmax, w.finish(own, nbr4, cnt, N, i, cap));
    }
    return wmax;
}

// The lists of a warp's atoms: slot i at position xd (own: there is an atom), one per
// lane; every lane of the warp calls this.  The 27 stencil cells of each lane are
// taken in turn, z fastest, in blocks of 8 candidates that start on a 16-byte
// boundary: four candidates per load and axis, tested two per instruction, the
// sign bits of r^2 - cut^2 collected and cut to the cell.  Every lane runs as many
// blocks as the longest cell of the warp has; past its own it tests its last
// block again and keeps nothing.  Returns the list's length before the cut at the
// capacity.
template <bool NC>
__device__ __forceinline__ int build_atom_lists(bool own, int i, const double4& xd, const Grid& g, const int* start,
                                                const PosNeg& posn, float3 Lf, float cut2, int cap, uint4* nbr4,
                                                int* cnt, int N, ListPend& pend) {
    auto first = [&](int c) { return NC ? __ldg(start + c) : start[c]; };
    const int ca = cell_coord(xd.x, g.ratio[0], g.n[0]), cb = cell_coord(xd.y, g.ratio[1], g.n[1]),
              cc = cell_coord(xd.z, g.ratio[2], g.n[2]);
    const float xi = (float)xd.x, yi = (float)xd.y, zi = (float)xd.z;
    const float2 mcut2 = make_float2(-cut2, -cut2);
    const float* const px = posn.p;
    const float* const py = px + posn.np;
    const float* const pz = py + posn.np;
    ListWriter w(pend);
#pragma unroll 1
    for (int col = 0; col < 9; ++col) {
        const int a = col / 3 - 1, b = col % 3 - 1;
        int na = ca + a, nb = cb + b;
        const int ia = na < 0 ? -1 : (na >= g.n[0] ? 1 : 0), ib = nb < 0 ? -1 : (nb >= g.n[1] ? 1 : 0);
        na -= ia * g.n[0];
        nb -= ib * g.n[1];
        const int c0 = g.flat(na, nb, 0);
        const float2 sx = make_float2(xi - ia * Lf.x, xi - ia * Lf.x), sy = make_float2(yi - ib * Lf.y, yi - ib * Lf.y);
#pragma unroll 1
        for (int c = -1; c <= 1; ++c) {
            int nc = cc + c;
            const int ic = nc < 0 ? -1 : (nc >= g.n[2] ? 1 : 0);
            nc -= ic * g.n[2];
            const int js = first(c0 + nc), je = own ? first(c0 + nc + 1) : js;
            const float2 sz = make_float2(zi - ic * Lf.z, zi - ic * Lf.z);
            const int self = col == 4 && c == 0 ? i : -2 * kBlock;
            int from = js & ~3, left = je - from;  // the block, and the candidates from it on
            const int mine = (left + kBlock - 1) / kBlock, last = from + kBlock * max(mine - 1, 0);
            const int blocks = (int)__reduce_max_sync(0xffffffffu, (unsigned)mine);
            unsigned valid = 0xffu >> (js & 3);  // candidates of the block, first highest
            for (int k = 0; k < blocks; ++k) {
                const int j = min(from, last);
                unsigned hit = 0;
#pragma unroll
                for (int t = 0; t < kBlock; t += 4) {
                    const float4 qx = ld_four<NC>(px + j + t), qy = ld_four<NC>(py + j + t), qz = ld_four<NC>(pz + j + t);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float2 dx = __fadd2_rn(sx, h ? make_float2(qx.z, qx.w) : make_float2(qx.x, qx.y));
                        const float2 dy = __fadd2_rn(sy, h ? make_float2(qy.z, qy.w) : make_float2(qy.x, qy.y));
                        const float2 dz = __fadd2_rn(sz, h ? make_float2(qz.z, qz.w) : make_float2(qz.x, qz.y));
                        const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                        const float2 sg = __fadd2_rn(r2, mcut2);
                        hit = __funnelshift_l(__float_as_uint(sg.x), hit, 1);
                        hit = __funnelshift_l(__float_as_uint(sg.y), hit, 1);
                    }
                }
                hit &= valid & ~(0xffu >> min(max(left, 0), kBlock));
                if ((unsigned)(self - from) < (unsigned)kBlock) hit &= ~(0x80u >> (self - from));
                const unsigned e = make_entry((unsigned)from, offset_code(a, b, c));
#pragma unroll
                for (int t = 0; t < kBlock; ++t) w.append((hit & (0x80u >> t)) != 0, e + ((unsigned)t << kCodeBits));
                valid = 0xffu;
                from += kBlock;
                left -= kBlock;
                w.make_room(nbr4, N, i, cap);
            }
        }
    }
    return w.finish(own, nbr4, cnt, N, i, cap);
}

// Atoms per list cell from which a warp per cell is the sooner done.
constexpr int kFullCell = 12;

__host__ __device__ __forceinline__ bool full_cells(int natoms, int ncell) { return natoms >= kFullCell * ncell; }

constexpr int kCellWarps = 4;

static __global__ void __launch_bounds__(32 * kCellWarps, 8)
build_cell_list_kernel(int N, PosNeg posn, Grid g, const int* __restrict__ start, float3 Lf, float cut2, int cap,
                       uint4* __restrict__ nbr4, int* __restrict__ cnt, Scalars* sc, Gate gate) {
    if (!gate.open()) return;
    __shared__ CellSmem sm[kCellWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * kCellWarps + warp;
    int n = 0;
    if (c < g.ncell())
        n = build_cell_lists<true>(c / (g.n[1] * g.n[2]), (c / g.n[2]) % g.n[1], c % g.n[2], g, start, posn, Lf, cut2, cap,
                                   nbr4, cnt, N, sm[warp], lane);
    n = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
    if (lane == 0) {
        atomicMax(&sc->max_count, n);
        if (n > cap) atomicExch(&sc->overflow, 1);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd((unsigned long long*)&sc->builds, 1ull);
}

static __global__ void __launch_bounds__(kThreads, 8)
build_atom_list_kernel(int N, const double4* __restrict__ pos, PosNeg posn, Grid g, const int* __restrict__ start, float3 Lf,
                  float cut2, int cap, uint4* __restrict__ nbr4, int* __restrict__ cnt, Scalars* sc, Gate gate) {
    if (!gate.open()) return;
    __shared__ ListPend pend[kThreads / 32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool own = i < N;
    int n = build_atom_lists<true>(own, i, pos[own ? i : 0], g, start, posn, Lf, cut2, cap, nbr4, cnt, N,
                                   pend[threadIdx.x >> 5]);
    n = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&sc->max_count, n);
        if (n > cap) atomicExch(&sc->overflow, 1);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd((unsigned long long*)&sc->builds, 1ull);
}

// ---------------------------------------------------------------------------
// FP64 pair force: full shell over the neighbour list (each atom sums its own
// row, so per-atom sums are deterministic and need no atomics), LJ spline of
// lennard_jones_force.cpp:107-119.  KICK fuses the second half kick
// (integrator.cpp:82) and the measurement partial sums into the epilogue.
//
// The loop runs over groups of 4 neighbours: the next group's indices are
// loaded (streaming, evict-first) while the current group's 4 positions are
// gathered and its 4 pairs evaluated without branches, the cutoff applied as a
// select.  That keeps several independent memory requests in flight per warp.
// ---------------------------------------------------------------------------
enum { KIND_LJ = 1, KIND_CONST = 2 };

// Fusion of the next step's first half kick and drift into the pair kernel's
// epilogue (kick_drift_kernel's arithmetic, in the same order): the new
// positions go to the other position buffer, which no pair kernel of this
// step reads.
struct Fuse {
    double4* pos_next;        // nullptr: no fusion
    float4* posl_next;        // mixed path: next step's cell-local coordinates
    const double4* pos;       // this step's positions (the mixed kernel reads FP32 copies)
    const double* bd;         // displacement at the last list build
    const double* bx;         // mixed path: cell-local position at the last list build
    Scalars* sc;
    int track, local, periodic;
};

// Second half kick (integrator.cpp:82) with the measurement partials and, when
// fused, the next step's first half kick, drift, displacement and periodic
// wrap (integrator.cpp:70-78).  Returns |d - d_build|^2 for the rebuild test.
__device__ __forceinline__ double step_epilogue(int N, int i, Soa s, const double4 x, const double (&f3)[3],
                                                const PairParams& pp, const Fuse& fz, double (&acc)[4]) {
    double xs[3] = {x.x, x.y, x.z};
    float l[3] = {0.f, 0.f, 0.f};
    double m = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = kick(s.at(VX + k, i), f3[k], pp.dt);
        acc[0] = fma(v, v, acc[0]);
        double d = s.at(DX + k, i);
        acc[3] = fma(d, d, acc[3]);
        if (fz.pos_next) {
            v = kick(v, f3[k], pp.dt);
            double inc = __dmul_rn(v, pp.dt);
            double xn = __dadd_rn(xs[k], inc);
            double dn = __dadd_rn(d, inc);
            if (fz.periodic) xn = wrap(xn, pp.L[k]);
            s.at(DX + k, i) = dn;
            xs[k] = xn;
            if (fz.track || fz.local) {
                double e = dn - fz.bd[(size_t)k * N + i];
                m = fma(e, e, m);
                if (fz.local) l[k] = (float)(fz.bx[(size_t)k * N + i] + e);
            }
        }
        s.at(VX + k, i) = v;
    }
    if (fz.pos_next) {
        fz.pos_next[i] = make_double4(xs[0], xs[1], xs[2], 0.0);
        if (fz.local) fz.posl_next[i] = make_float4(l[0], l[1], l[2], 0.f);
    }
    return fz.track ? m : 0.0;
}

// Warp max of the fused displacement into the next step's rebuild criterion.
__device__ __forceinline__ void fused_track(const Fuse& fz, double m) {
    if (fz.pos_next && fz.track) {
        m = warp_max(m);
        if ((threadIdx.x & 31) == 0 && m > 0.0)
            atomicMax(&fz.sc->max_disp2_next, (unsigned long long)__double_as_longlong(m));
    }
}

// One 32-byte position in a single 256-bit load (sm_100 ld.global.v4.f64;
// positions are double4 in cudaMalloc'd arrays, so always 32-byte aligned).
__device__ __forceinline__ double4 ld_pos(const double4* p) {
    double4 r;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
    return r;
}

// 1/x: the hardware's approximate FP64 reciprocal refined by one third-order
// (Householder) step y <- y (1 + e + e^2), e = 1 - x y: the seed's ~2^-20
// relative error cubes to ~2^-60, below the last bit of the result, in three
// dependent FMAs where two Newton-Raphson steps need four.
__device__ __forceinline__ double rcp_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

template <bool SMALL>
__device__ __forceinline__ void separation(const double4& xi, const double4& xj, unsigned e, bool near,
                                           const PairParams& pp, double& dx, double& dy, double& dz) {
    dx = __dsub_rn(xi.x, xj.x);
    dy = __dsub_rn(xi.y, xj.y);
    dz = __dsub_rn(xi.z, xj.z);
    if (SMALL) {
        int ia = entry_axis(e, 0), ib = entry_axis(e, 1), ic = entry_axis(e, 2);
        dx = __dsub_rn(dx, ia * pp.L[0]);
        dy = __dsub_rn(dy, ib * pp.L[1]);
        dz = __dsub_rn(dz, ic * pp.L[2]);
    } else if (near) {
        // minimum image; identical to the reference's stencil image for every
        // pair inside the cutoff (the list grid has >= 3 cells per axis)
        if ((__double2hiint(dx) & 0x7fffffff) > pp.halfL_hi[0]) dx = __dsub_rn(dx, copysign(pp.L[0], dx));
        if ((__double2hiint(dy) & 0x7fffffff) > pp.halfL_hi[1]) dy = __dsub_rn(dy, copysign(pp.L[1], dy));
        if ((__double2hiint(dz) & 0x7fffffff) > pp.halfL_hi[2]) dz = __dsub_rn(dz, copysign(pp.L[2], dz));
    }
}

template <int KIND>
__device__ __forceinline__ void pair_fp64(const PairParams& pp, double r2, double& f, double& V, double& W) {
    if (KIND == KIND_LJ) {
        bool hit = r2 < pp.rc2;
        double ir2 = rcp_nr(r2);
        double ir6 = ir2 * ir2 * ir2;
        double x = r2 * pp.inv_rc2;
        double v = fma(4.0 * ir6, ir6 - 1.0, fma(pp.beta, x - 1.0, pp.alpha));
        double w = fma(24.0 * ir6, fma(2.0, ir6, -1.0), -2.0 * pp.beta * x);
        f = hit ? w * ir2 : 0.0;
        V = hit ? v : 0.0;
        W = hit ? w : 0.0;
    } else {
        // tests/cpp/mock/constant_short_range_force.cpp:35-53
        double norm = sqrt(r2);
        bool hit = r2 < pp.rc2 && norm < pp.rc;
        V = hit ? pp.strength * (pp.rc - norm) : 0.0;
        W = hit ? pp.strength * norm : 0.0;
        f = hit ? W / (norm * norm) : 0.0;
    }
}

// LJ spline pairs of one atom (lennard_jones_force.cpp:107-119) accumulated as
// the force plus power sums: with u = r^-6 and x = r^2 / rc^2 the pair terms
// are V = 4u(u - 1) + beta x + (alpha - beta) and W = u(48u - 24) - 2 beta x,
// so the atom's energy and virial follow from sum u^2, sum u, sum r^2 and the
// pair count, formed once per atom, instead of V and W per pair; the force
// magnitude over r is W / r^2 = u(48u - 24) r^-2 - 2 beta / rc^2 (22 instead of
// 28 FP64 operations per pair).  Pairs at or beyond the cutoff add nothing.
struct LjSums {
    double fx = 0, fy = 0, fz = 0, su2 = 0, su = 0, sr2 = 0;
    int nh = 0;
};

__device__ __forceinline__ void lj_accumulate(const PairParams& pp, double dx, double dy, double dz, LjSums& a) {
    const double wq = -2.0 * pp.beta * pp.inv_rc2;
    double r2 = norm2(dx, dy, dz);
    bool hit = r2 < pp.rc2;
    double ir2 = rcp_nr(r2);
    double u = ir2 * ir2 * ir2;
    double f = hit ? fma(u * fma(48.0, u, -24.0), ir2, wq) : 0.0;  // W / r^2 = u(48u - 24) r^-2 + wq
    double uh = hit ? u : 0.0;
    a.su2 = fma(uh, uh, a.su2);
    a.su += uh;
    a.sr2 += hit ? r2 : 0.0;
    a.nh += hit ? 1 : 0;
    a.fx = fma(f, dx, a.fx);
    a.fy = fma(f, dy, a.fy);
    a.fz = fma(f, dz, a.fz);
}

// The atom's sum of pair energies and of pair virials (each pair counted in
// both of its atoms' rows, halved by the finalize).
__device__ __forceinline__ void lj_energy(const PairParams& pp, const LjSums& a, double& pe, double& w) {
    const double bq = pp.beta * pp.inv_rc2, abq = pp.alpha - pp.beta, wq = -2.0 * pp.beta * pp.inv_rc2;
    pe = fma(4.0, a.su2 - a.su, fma(bq, a.sr2, abq * (double)a.nh));
    w = fma(48.0, a.su2, fma(-24.0, a.su, wq * a.sr2));
}

// Loads of data that another block of the same launch may have written since
// the block started (the resident step kernel, lj_resident.cuh) must not take
// the non-coherent path; launches that only read them may.
template <bool NC>
__device__ __forceinline__ double4 ld_neighbour(const double4* p) {
    if (NC) return ld_pos(p);
    double4 r;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
    return r;
}

template <bool NC>
__device__ __forceinline__ uint4 ld_group(const uint4* p) {
    if (NC) return __ldcs(p);
    uint4 r;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

// The list groups (4 neighbours) of one atom: indices stream from HBM, two
// groups in flight ahead of the two being evaluated.
template <class Group>
__device__ __forceinline__ void for_groups(const uint4* lp, int N, int ng, Group group) {
    const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
    uint4 A = ng > 0 ? ld_group<true>(lp) : z4;
    uint4 B = ng > 1 ? ld_group<true>(lp + (size_t)N) : z4;
    for (int g = 0; g < ng; g += 2) {
        uint4 C = g + 2 < ng ? ld_group<true>(lp + (size_t)(g + 2) * N) : z4;
        uint4 D = g + 3 < ng ? ld_group<true>(lp + (size_t)(g + 3) * N) : z4;
        group(A);
        if (g + 1 < ng) group(B);
        A = C;
        B = D;
    }
}

// One group of a row: 4 neighbours gathered, then 4 pairs evaluated without branches.
template <bool SMALL, bool NC>
__device__ __forceinline__ void lj_group(const double4* pos, const uint4 grp, const double4& xi, bool near,
                                         const PairParams& pp, LjSums& a) {
    const unsigned e[4] = {grp.x, grp.y, grp.z, grp.w};
    double4 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) q[u] = ld_neighbour<NC>(pos + entry_slot(e[u]));
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        double dx, dy, dz;
        separation<SMALL>(xi, q[u], e[u], near, pp, dx, dy, dz);
        lj_accumulate(pp, dx, dy, dz, a);
    }
}

// ---- rows that several lanes may share -------------------------------------
//
// The systems that step in the resident kernel (lj_resident.cuh) sum a row in
// chunks of 2 groups = 8 neighbours: each chunk from zero, the chunk sums then
// added in list order.  LANES lanes (a power of two up to 16) may share the row,
// lane l taking the chunks l, l + LANES, ...; after each round the lanes leave
// their chunk sums in shared memory and every lane adds the round's sums of its
// own components, in list order.  The sums do not depend on LANES.
//
// The six components are fx, fy, fz, sum u^2, sum u, sum r^2; lane l ends with
// components l, l + LANES, ... in tot[0], tot[1], ... (all six with LANES = 1),
// so the force along axis k is in lane k mod LANES.
constexpr int kRowPad = 7;  // doubles between two lanes' chunk sums: no bank conflicts
constexpr int kRowWords = 32 * kRowPad;

template <int LANES>
struct RowSums {
    static constexpr int kOwn = (6 + LANES - 1) / LANES;
    double tot[kOwn];
    int nh = 0;  // pairs inside the cutoff (of this lane's chunks until finish())
    __device__ __forceinline__ RowSums() {
#pragma unroll
        for (int q = 0; q < kOwn; ++q) tot[q] = 0.0;
    }
    // add one round's chunk sums (T: the arithmetic of the chunk)
    template <class T>
    __device__ __forceinline__ void add(const T (&c)[6], double* xch, int lane) {
        if (LANES == 1) {
#pragma unroll
            for (int q = 0; q < 6; ++q) tot[q] += (double)c[q];
            return;
        }
        T* const w = reinterpret_cast<T*>(xch);
#pragma unroll
        for (int q = 0; q < 6; ++q) w[lane * kRowPad + q] = c[q];
        __syncwarp();
        const int l = lane % LANES, base = lane - l;
#pragma unroll
        for (int q = 0; q < kOwn; ++q) {
            const int k = l + q * LANES;
            if (k < 6)
#pragma unroll
                for (int u = 0; u < LANES; ++u) tot[q] += (double)w[(base + u) * kRowPad + k];
        }
        __syncwarp();
    }
    // component k, in every lane of the atom
    __device__ __forceinline__ double get(int k) const {
        return LANES == 1 ? tot[k] : __shfl_sync(0xffffffffu, tot[k / LANES], k % LANES, LANES);
    }
    // the force's axes that this lane owns
    __device__ __forceinline__ double own(int k) const { return tot[k / LANES]; }
    // energy and virial sums, in every lane
    __device__ __forceinline__ void energy(const PairParams& pp, double& pe, double& w) {
#pragma unroll
        for (int off = 1; off < LANES; off <<= 1) nh += __shfl_xor_sync(0xffffffffu, nh, off);
        LjSums a;
        a.su2 = get(3);
        a.su = get(4);
        a.sr2 = get(5);
        a.nh = nh;
        lj_energy(pp, a, pe, w);
    }
};

// A lane's first two groups.  Where many lanes share a row, its length `count` (an
// atom's list entries; null: no atom) is not waited for: the groups are there up to the list's
// capacity, whatever they hold beyond it.  Sets ng, the row's groups.
template <int LANES, bool NC>
__device__ __forceinline__ void first_groups(const uint4* lp, int N, int capg, const int* count, int g0, int& ng, uint4& A,
                                             uint4& B) {
    const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
    if (LANES >= 4) {
        A = count && g0 < capg ? ld_group<NC>(lp + (size_t)g0 * N) : z4;
        B = count && g0 + 1 < capg ? ld_group<NC>(lp + (size_t)(g0 + 1) * N) : z4;
        ng = count ? (*count + 3) >> 2 : 0;
    } else {
        ng = count ? (*count + 3) >> 2 : 0;
        A = g0 < ng ? ld_group<NC>(lp + (size_t)g0 * N) : z4;
        B = g0 + 1 < ng ? ld_group<NC>(lp + (size_t)(g0 + 1) * N) : z4;
    }
}

// Every lane of the warp calls this when LANES > 1 (count null where there is no atom).
template <int LANES, bool SMALL, bool NC>
__device__ __forceinline__ void row_lj(const double4* pos, const uint4* lp, int N, int capg, const int* count, int lane,
                                       const double4& xi, bool near, const PairParams& pp, double* xch,
                                       RowSums<LANES>& r) {
    const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
    const int g0 = LANES == 1 ? 0 : 2 * (lane % LANES);
    int ng;
    uint4 A, B;
    first_groups<LANES, NC>(lp, N, capg, count, g0, ng, A, B);
    const int end = LANES == 1 ? ng : (int)__reduce_max_sync(0xffffffffu, (unsigned)ng);
    for (int s = 0; s < end; s += 2 * LANES) {
        const int g = s + g0;
        uint4 C = g + 2 * LANES < ng ? ld_group<NC>(lp + (size_t)(g + 2 * LANES) * N) : z4;
        uint4 D = g + 2 * LANES + 1 < ng ? ld_group<NC>(lp + (size_t)(g + 2 * LANES + 1) * N) : z4;
        LjSums a;
        if (LANES == 1 || g < ng) lj_group<SMALL, NC>(pos, A, xi, near, pp, a);
        if (g + 1 < ng) lj_group<SMALL, NC>(pos, B, xi, near, pp, a);
        r.nh += a.nh;
        const double c[6] = {a.fx, a.fy, a.fz, a.su2, a.su, a.sr2};
        r.add(c, xch, lane);
        A = C;
        B = D;
    }
}

// Partial sums of these systems: units of 8 atoms, added over the bits of the
// atom's index from the lowest up, whatever the lanes per atom.  Unit u of a
// system goes to partials[u].  a: the atom's index in its system; acc: its terms
// (zero where there is no atom), valid in the atom's lane 0.  With 8 or 16 lanes a
// unit spans warps: every thread of the block (a multiple of 128 threads) calls this.
constexpr int kUnit = 8;

template <int LANES>
__device__ __forceinline__ void unit_partials(double (&acc)[4], int a, int natoms, double* partials) {
#pragma unroll
    for (int off = LANES; off < 8 * LANES && off < 32; off <<= 1)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], off);
    if (LANES <= 4) {
        if (threadIdx.x % (8 * LANES) == 0 && a < natoms)
#pragma unroll
            for (int q = 0; q < 4; ++q) partials[4 * (size_t)(a / kUnit) + q] = acc[q];
        return;
    }
    __shared__ double sm[32][4];
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x % 32 == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q) sm[warp][q] = acc[q];
    __syncthreads();
    const int per = LANES == 8 ? 2 : 4;  // warps per unit
    if (threadIdx.x % (32 * per) < 4 && a - (int)(threadIdx.x % 32) / LANES < natoms) {
        const int q = threadIdx.x % 32;
        double v = sm[warp][q] + sm[warp + 1][q];
        if (per == 4) v += sm[warp + 2][q] + sm[warp + 3][q];
        partials[4 * (size_t)(a / kUnit) + q] = v;
    }
    __syncthreads();
}

// Whether an atom is so near a face of the box that a neighbour may be an image.
__device__ __forceinline__ bool near_face(const double4& x, const PairParams& pp) {
    return !(x.x >= pp.near_lo && x.x < pp.near_hi[0] && x.y >= pp.near_lo && x.y < pp.near_hi[1] &&
             x.z >= pp.near_lo && x.z < pp.near_hi[2]);
}

// Occupancy bound: 768 resident threads' worth of blocks per SM caps the kernel
// at 80 registers (no spills); it is latency-bound on the neighbour gathers,
// and 24 resident warps per SM measured ~12 % faster than 16 at 114 registers.
// UNITS: the row and partial sums of the systems that step in the resident
// kernel (chunks of 8 neighbours, units of 8 atoms).
template <int KIND, bool SMALL, bool KICK, int BS = kThreads, bool UNITS = false>
static __global__ void __launch_bounds__(BS, (UNITS ? 640 : 768) / BS)
force_fp64_kernel(int N, const double4* __restrict__ pos, Soa s, const uint4* __restrict__ nbr4,
                  const int* __restrict__ cnt, PairParams pp, double* __restrict__ partials, Fuse fu) {
    static_assert(!UNITS || KIND == KIND_LJ, "the resident kernel has the LJ force only");
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[4] = {0, 0, 0, 0};  // sum v^2, sum pe_i, sum w_i, sum d^2
    double m = 0.0;
    if (i < N) {
        const double4 xi = pos[i];
        const bool near = near_face(xi, pp);
        LjSums a;        // the LJ sums, or the mock's force
        double pe = 0, w = 0;
        const int ng = (cnt[i] + 3) >> 2;
        const uint4* lp = nbr4 + i;
        if (UNITS) {
            RowSums<1> r;
            row_lj<1, SMALL, true>(pos, lp, N, 0, cnt + i, 0, xi, near, pp, nullptr, r);
            a.fx = r.tot[0];
            a.fy = r.tot[1];
            a.fz = r.tot[2];
            r.energy(pp, pe, w);
        } else if (KIND == KIND_LJ) {
            for_groups(lp, N, ng, [&](const uint4 grp) { lj_group<SMALL, true>(pos, grp, xi, near, pp, a); });
            lj_energy(pp, a, pe, w);
        } else {
            for_groups(lp, N, ng, [&](const uint4 grp) {
                const unsigned e[4] = {grp.x, grp.y, grp.z, grp.w};
                double4 q[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) q[u] = ld_pos(pos + entry_slot(e[u]));
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    double dx, dy, dz, f, V, W;
                    separation<SMALL>(xi, q[u], e[u], near, pp, dx, dy, dz);
                    pair_fp64<KIND>(pp, norm2(dx, dy, dz), f, V, W);
                    a.fx = fma(f, dx, a.fx);
                    a.fy = fma(f, dy, a.fy);
                    a.fz = fma(f, dz, a.fz);
                    pe += V;
                    w += W;
                }
            });
        }
        if (!KICK || !fu.pos_next) {  // a fused step's forces end with its two kicks
            s.at(FX, i) = a.fx;
            s.at(FY, i) = a.fy;
            s.at(FZ, i) = a.fz;
        }
        acc[1] = pe;
        acc[2] = w;
        if (KICK) {
            const double f3[3] = {a.fx, a.fy, a.fz};
            m = step_epilogue(N, i, s, xi, f3, pp, fu, acc);
        }
    }
    if (KICK) fused_track(fu, m);
    if (UNITS) {
        unit_partials<1>(acc, i, N, partials);
        return;
    }
    block_sum<4, BS>(acc);
    if (threadIdx.x == 0)
        for (int q = 0; q < 4; ++q) partials[(size_t)blockIdx.x * 4 + q] = acc[q];
}

// ---------------------------------------------------------------------------
// Step finalisation: sum the per-block partials in a fixed order and publish
// ThermodynamicMeasurement::Result (measurements.hpp:59-70).
// mode 0: after a step (t += dt); 1: after a force evaluation (PE, W only);
// 2: measurement of the current state; 3: as 0, what the next step's rebuild depends
// on left to advance_kernel.
// ---------------------------------------------------------------------------
// Step graphs: between a fused pair kernel and the next step's rebuild node, the next
// step's displacement becomes this step's and the conditional is set.  One thread:
// the step's sums and record (finalize_kernel) are off this path, beside the next
// step's rebuild and pair kernel (a step of 1 048 576 atoms has 7 to 8 us of it).
static __global__ void advance_kernel(Gate gate, cudaGraphConditionalHandle h, Scalars* sc) {
    const unsigned long long md2 = sc->max_disp2_next;
    sc->max_disp2 = md2;
    sc->max_disp2_next = 0ull;
    sc->need_rebuild = 0;
    const bool open = gate.always || __longlong_as_double((long long)md2) > gate.thresh2;
    if (open) sc->graph_rebuilds += 1;
    cudaGraphSetConditional(h, open ? 1u : 0u);
}

static __global__ void __launch_bounds__(1024)
finalize_kernel(const double* __restrict__ partials, int nblocks, int N, double dt, int mode,
                int forces_valid, Scalars* sc, double* __restrict__ ring, int ring_cap) {
    // thread 0 loads the scalars it updates before the reduction, so that those
    // loads overlap the partials' instead of following one another at the end
    // (only this kernel changes them while it runs)
    double t0 = 0, pe0 = 0, vir0 = 0;
    long long steps0 = 0;
    const bool step = mode == 0 || mode == 3;
    if (threadIdx.x == 0) {
        t0 = sc->t;
        pe0 = sc->pe;
        vir0 = sc->vir;
        steps0 = sc->steps;
    }
    // each thread sums blocks tid, tid + 1024, ... in that order; eight blocks'
    // partials (32-byte loads) are in flight at a time
    double acc[4] = {0, 0, 0, 0};
    const double4* p4 = reinterpret_cast<const double4*>(partials);
    for (int b0 = threadIdx.x; b0 < nblocks; b0 += 8 * 1024) {
        double4 t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int b = b0 + u * 1024;
            t[u] = b < nblocks ? p4[b] : make_double4(0.0, 0.0, 0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (b0 + u * 1024 < nblocks) {
                acc[0] += t[u].x;
                acc[1] += t[u].y;
                acc[2] += t[u].z;
                acc[3] += t[u].w;
            }
        }
    }
    block_sum<4, 1024>(acc);
    if (threadIdx.x == 0) {
        double pe = pe0, vir = vir0, t = t0;
        if (forces_valid) {
            pe = 0.5 * acc[1];
            vir = 0.5 * acc[2];
            sc->pe = pe;
            sc->vir = vir;
        }
        // a step's record goes to ring slot (step index mod ring_cap); the extra
        // slot ring_cap holds single measurements
        double* out = ring + 7 * (size_t)(step ? (int)(steps0 % ring_cap) : ring_cap);
        if (step) {
            t = t0 + dt;  // integrator.cpp:85
            sc->t = t;
            sc->steps = steps0 + 1;
        }
        if (mode != 1) {
            double ke = 0.5 * acc[0];
            double rec[7];
            rec[0] = t;
            rec[1] = ke;
            rec[2] = pe;
            rec[3] = pe + ke;
            rec[4] = vir;
            rec[5] = (2. / 3.) * ke / (double)N;
            rec[6] = acc[3] / (double)N;
            for (int q = 0; q < 7; ++q) out[q] = rec[q];
            if (!isfinite(ke) || !isfinite(pe) || !isfinite(vir)) sc->nonfinite = 1;
        } else if (!isfinite(pe) || !isfinite(vir)) {
            sc->nonfinite = 1;
        }
        if (mode <= 1) {  // (a measurement changes nothing that a rebuild depends on)
            sc->max_disp2 = 0ull;
            sc->need_rebuild = 0;
        }
    }
}

// ThermodynamicAnalyzer::result (analyzers.cpp:44-159) over the last W step
// records of a record ring, one block per system: record k of the window
// (k = 0 oldest) of system s sits at ring + 7 * (slot(k) * nsys + s) with
// slot(k) = (last - (W - 1) + k) mod ring_cap.  Two passes as
// tools::MovingSample::statistics (moving_sample.hpp:107-188): the means, then
// the Bessel-corrected variance of T and the covariance of (t, MSD); each sum
// is a fixed-order block reduction.
constexpr int kStatsThreads = 256;

static __global__ void __launch_bounds__(kStatsThreads)
window_stats_kernel(const double* __restrict__ ring, int ring_cap, int nsys, long long last, int W,
                    const int* __restrict__ natoms, const double* __restrict__ density, double* __restrict__ out) {
    int s = blockIdx.x;
    auto rec = [&](int k) {
        long long step = last - (W - 1) + k;
        int slot = (int)(((step % ring_cap) + ring_cap) % ring_cap);
        return ring + 7 * ((size_t)slot * nsys + s);
    };
    // pass 1: sums of T, TE, W, t, MSD
    double a[5] = {0, 0, 0, 0, 0};
    for (int k = threadIdx.x; k < W; k += kStatsThreads) {
        const double* r = rec(k);
        a[0] += r[5];
        a[1] += r[3];
        a[2] += r[4];
        a[3] += r[0];
        a[4] += r[6];
    }
    block_sum<5, kStatsThreads>(a);
    __shared__ double mean[5];
    if (threadIdx.x == 0)
        for (int q = 0; q < 5; ++q) mean[q] = a[q] / (double)W;
    __syncthreads();
    // pass 2: sum (T - <T>)^2, (t - <t>)(MSD - <MSD>), (t - <t>)^2
    double c[3] = {0, 0, 0};
    for (int k = threadIdx.x; k < W; k += kStatsThreads) {
        const double* r = rec(k);
        double dT = r[5] - mean[0], dt = r[0] - mean[3], dm = r[6] - mean[4];
        c[0] += dT * dT;
        c[1] += dt * dm;
        c[2] += dt * dt;
    }
    block_sum<3, kStatsThreads>(c);
    if (threadIdx.x == 0) {
        double N = (double)natoms[s], rho = density[s];
        double T = mean[0];
        double varT = c[0] / (double)(W - 1);
        double* o = out + 6 * (size_t)s;
        o[0] = T;
        o[1] = rho;
        o[2] = mean[1];
        o[3] = rho * (T + mean[2] / (3.0 * N));
        o[4] = (3. / 2.) / (1 - (3. / 2.) * N * (varT / (T * T)));
        o[5] = (1. / 6.) * ((c[1] / (double)(W - 1)) / (c[2] / (double)(W - 1)));
    }
}

// Graph step: decide on the device whether the rebuild subgraph runs this step.
static __global__ void decide_rebuild_kernel(Gate gate, cudaGraphConditionalHandle h, Scalars* sc) {
    bool open = gate.open();
    if (open) sc->graph_rebuilds += 1;
    cudaGraphSetConditional(h, open ? 1u : 0u);
}

static __global__ void __launch_bounds__(kThreads)
scale_kernel(int N, Soa s, double factor) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
#pragma unroll
    for (int k = 0; k < 3; ++k) s.at(VX + k, i) = __dmul_rn(s.at(VX + k, i), factor);
}

// set_temperature (transformations.cpp:94-116): the factor is computed on the
// device from the KE of the record written by the preceding measurement.
static __global__ void set_temperature_factor_kernel(const double* rec, double target, double* factor) {
    *factor = sqrt(target / rec[5]);
}

static __global__ void __launch_bounds__(kThreads)
scale_from_device_kernel(int N, Soa s, const double* __restrict__ factor) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    double f = *factor;
#pragma unroll
    for (int k = 0; k < 3; ++k) s.at(VX + k, i) = __dmul_rn(s.at(VX + k, i), f);
}

// ---------------------------------------------------------------------------
// Host <-> device layout conversion (atom-id order <-> sorted slots)
// ---------------------------------------------------------------------------
// The arrays of a transfer -- positions, velocities, displacements, forces, `stride`
// doubles per atom in id order -- in device or in mapped host memory; null: not
// asked for (out), zeros (in).
struct StateArrays {
    double* a[4];
    int stride;
};

__device__ __forceinline__ int state_field(int q) { return q == 1 ? VX : (q == 2 ? DX : FX); }

// What a resident launch that ended early leaves half done, as a launch expects it:
// the barrier's word, and the counts of the list cells.
struct Restart {
    unsigned long long* word;  // null: nothing to restart
    int* count;
    int ncell;
};

// State of n atoms into slots first, first + 1, ..., in id order; sc (may be null)
// takes `init`, apart from the counters of builds and steps.
static __global__ void unpack_state_kernel(int first, int n, StateArrays in, double4* __restrict__ pos, Soa s,
                                           int* __restrict__ ids, Scalars* sc, Scalars init, Restart re) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (re.word) {
        if (i == 0) *re.word = 0ull;
        for (int c = i; c < re.ncell; c += gridDim.x * blockDim.x) re.count[c] = 0;
    }
    if (sc && i == 0) {
        init.builds = sc->builds;
        init.steps = sc->steps;
        *sc = init;
    }
    if (i >= n) return;
    const double* x = in.a[0] + (size_t)i * in.stride;
    pos[first + i] = make_double4(x[0], x[1], x[2], 0.0);
    ids[first + i] = i;
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        const double* p = in.a[q] ? in.a[q] + (size_t)i * in.stride : nullptr;
#pragma unroll
        for (int k = 0; k < 3; ++k) s.at(state_field(q) + k, first + i) = p ? p[k] : 0.0;
    }
}

// State of slots first, first + 1, ... out in id order.
static __global__ void pack_state_kernel(int first, int n, StateArrays out, const double4* __restrict__ pos, Soa s,
                                         const int* __restrict__ ids) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int slot = first + k;
    const size_t at = (size_t)ids[slot] * out.stride;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        double* p = out.a[q];
        if (!p) continue;
        double v[3];
        if (q == 0) {
            const double4 x = pos[slot];
            v[0] = x.x; v[1] = x.y; v[2] = x.z;
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c] = s.at(state_field(q) + c, slot);
        }
        p += at;
        if (out.stride == 4 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
            reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
            reinterpret_cast<double2*>(p)[1] = make_double2(v[2], 0.0);
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) p[c] = v[c];
            if (out.stride == 4) p[3] = 0.0;
        }
    }
}

// Where the GPU can reach `bytes` bytes from p on, if all of them are pinned (mapped) host
// memory and doubles there are aligned; otherwise null, and the array is copied.  One
// query of the driver: the runtime's knows of the first byte only, and behind the end of
// a registered range a kernel faults where a copy returns an error.
inline double* mapped_host(const double* p, size_t bytes) {
    using Query = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
    static const Query query = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Query>(f);
    }();
    if (!query || reinterpret_cast<uintptr_t>(p) % alignof(double)) return nullptr;
    unsigned type = 0, managed = 0;
    CUdeviceptr at = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                  CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                  CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* values[] = {&type, &managed, &at, &start, &size};
    const CUdeviceptr first = reinterpret_cast<CUdeviceptr>(p);
    if (query(5, what, values, first) != CUDA_SUCCESS || type != CU_MEMORYTYPE_HOST || managed) return nullptr;
    return first >= start && bytes <= size && first - start <= size - bytes ? reinterpret_cast<double*>(at) : nullptr;
}

// Arrays of up to this many atoms in mapped memory are read and written in place: a
// copy's launch costs more than the slower single accesses (a download of 2000 atoms
// 24 us in place; of 4000 41 in place, 33 copied; of 16 000 112 and 53).
constexpr int kMappedAtoms = 3072;

// Reference binning for the debug API: cell of each atom id, and members as ids.
static __global__ void debug_members_kernel(int N, const int* __restrict__ cell_of_slot,
                                     const int* __restrict__ rank, const int* __restrict__ start,
                                     const int* __restrict__ ids, int* __restrict__ members,
                                     int* __restrict__ cell_of_id) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    members[start[cell_of_slot[k]] + rank[k]] = ids[k];
    cell_of_id[ids[k]] = cell_of_slot[k];
}

static __global__ void sort_members_kernel(int ncell, const int* __restrict__ start, int* __restrict__ m) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncell) return;
    for (int k = start[c] + 1; k < start[c + 1]; ++k) {
        int v = m[k], q = k - 1;
        while (q >= start[c] && m[q] > v) {
            m[q + 1] = m[q];
            --q;
        }
        m[q + 1] = v;
    }
}

// The in-cutoff pair set as seen by the force kernel (i < j by id).
template <bool SMALL>
static __global__ void debug_pairs_kernel(int N, const double4* __restrict__ pos,
                                   const uint4* __restrict__ nbr4, const int* __restrict__ cnt,
                                   const int* __restrict__ ids, PairParams pp, long long cap,
                                   int* oi, int* oj, int* oimg, double* or2,
                                   unsigned long long* counter) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    double4 xi = pos[i];
    const unsigned* nbr = reinterpret_cast<const unsigned*>(nbr4);
    for (int k = 0; k < cnt[i]; ++k) {
        unsigned e = nbr[((size_t)(k >> 2) * N + i) * 4 + (k & 3)];
        int j = (int)entry_slot(e);
        if (ids[i] >= ids[j]) continue;
        double4 xj = pos[j];
        double d[3] = {__dsub_rn(xi.x, xj.x), __dsub_rn(xi.y, xj.y), __dsub_rn(xi.z, xj.z)};
        int img[3] = {0, 0, 0};
        if (SMALL) {
            for (int q = 0; q < 3; ++q) img[q] = entry_axis(e, q);
        } else {
            for (int q = 0; q < 3; ++q)
                if ((__double2hiint(d[q]) & 0x7fffffff) > pp.halfL_hi[q]) img[q] = d[q] > 0 ? 1 : -1;
        }
        for (int q = 0; q < 3; ++q) d[q] = __dsub_rn(d[q], img[q] * pp.L[q]);
        double r2 = norm2(d[0], d[1], d[2]);
        if (r2 < pp.rc2) {
            unsigned long long slot = atomicAdd(counter, 1ull);
            if ((long long)slot < cap) {
                oi[slot] = ids[i];
                oj[slot] = ids[j];
                oimg[slot] = image_code(img[0], img[1], img[2]);
                or2[slot] = r2;
            }
        }
    }
}

}  // namespace ljb
