// lj_resident.cuh -- many velocity-Verlet steps of one or several systems in one
// cooperative launch, for systems too small to fill the GPU for long.
//
// A step of a few thousand atoms is a few microseconds of work; run as separate
// kernels (graph or not) it is bound by launches, by the conditional node and by
// the nine kernels of a list rebuild.  Here a system is owned by a group of
// blocks that stay on the GPU for the whole call and meet in a barrier of their
// own in global memory: one barrier a step, one to six more on a step that
// rebuilds the list.  Groups do not know of each other, so the systems of a batch step
// independently, each at its own pace, and rebuild when they need to.
//
//   drift of the first step
//   per step: barrier
//     rebuild if some block found |d - d_build| > skin / 2 (a vote in the barrier):
//       bin | scan + scatter | sort + move | lists       (a barrier after each, and two in
//       the scan of more cells than each block scans for itself; up to 4096 atoms every
//       block sorts all of them for itself, and there is only the last)
//     pair rows, second kick, partial sums, next step's kick and drift
//     (meanwhile one block adds up the previous step's record)
//
// The positions alternate between two buffers (a step reads one and writes the
// next step's into the other) and a rebuild permutes the rest of the state from
// one buffer into the other; the last step writes everything to the first
// buffers, so that between launches the state is where every other entry point
// expects it.  Arithmetic and summation orders are those of the kernels that run
// one phase per launch (lj_kernels.cuh, lj_mixed.cuh): results agree bit for bit.
//
// What bounds it: latency -- the barrier (1.4 us over one block per SM; with blocks of
// 128 threads it grew from 1.4 us over 33 to 2.7 us over 500 of them) and the chain
// list length -> list group -> positions -> FP64 pairs -> kick (3 to 4 us).  Measured
// per step, as graphs of one kernel per phase and in this form: N = 256 in a box of
// 2 cells 127 -> 17.9 us, N = 500 30 -> 6.3 us, N = 4000 34 -> 10.0 us, N = 31 987 mixed
// 32 -> 18.2 us, N = 90 000 49.5 -> 39.2 us (mixed 41.5 ->
// 28.8 us); 64 systems of 576 536 atoms together 384 -> 213 us.  Which sizes take this
// form: steps_resident().
//
// What another block wrote in this launch is read with plain loads after the
// barrier (an acquire at GPU scope), never through the non-coherent path.  The
// launch is cooperative, so all blocks of a group are resident; every wait is
// bounded all the same, and a wait that runs out sets an error word and ends the
// block: it arrives at no later barrier, so the others end at the next one, and
// none gets further than that.  The barrier's word, the cell counts and the state are
// then a part of a step, on which no later launch may run until an upload restores all
// three: a launch that follows another whose end the host has not seen gets that error
// word as its `active` flag and returns at once.
#pragma once

#include "lj_mixed.cuh"

namespace ljb {

constexpr int kResidentThreads = 128;      // of a block where systems share the GPU (a batch)
// Of those per SM: 96 registers.  The FP64 instances spill a little there (96 bytes stored
// and 80 loaded a thread, a small box 76 and 72, a batch 192 and 332; mixed none).
constexpr int kResidentBlocks = 5;
constexpr int kResidentMost = kResidentThreads * kResidentBlocks;  // threads of a block that has its SM to itself
constexpr int kResidentPolls = 1 << 22;    // bound of one barrier wait (about a second)
constexpr int kResidentMaxAtoms = 94720;   // an atom per thread of 148 SMs
constexpr int kGraphWaveAtoms = 113664;    // atoms of one wave of the graphs' pair kernel: 768 per SM
constexpr int kMaxLanes = 16;              // lanes that may share an atom's row
// Cells that every block scans for itself, in shared memory: of a system that shares
// its SMs with others, and of one that has them to itself.
constexpr int kScanCells = 1024, kScanCellsAlone = 4096;
// Atoms that every block of a single system sorts for itself: three barriers of a rebuild
// against every block reading all positions.  Measured per step, sorted by all blocks
// together and by each: N = 1500 9.37 -> 8.86 us, 2048 8.58 -> 8.42, 4000 9.89 -> 9.77
// (rho 0.8; at 0.4 8.72 -> 8.13, 9.05 -> 8.70, 10.50 -> 10.31); the arrays take 78 KB of
// shared memory.
constexpr int kTinyAtoms = 4096;

// Buffers of all systems of a launch (slots and cells are global indices).
struct ResArrays {
    double4* pos[2];
    float4* posl[2];
    double* soa[2];
    int* ids[2];
    double* bd;
    double* bx;
    PosNeg posn;
    int* cell_of;
    int* rank;
    int* order;
    int* count;
    int* start;
    int* tiles;        // one per block of the launch
    uint4* nbr;
    int* cnt;
    double* partials;  // two halves of part_stride records of 4
    int part_stride;
    int N;             // atoms of all systems: stride of the arrays, and the ghost slot
    int cap;
};

// A group's barrier word (Group).
struct ResSync {
    unsigned long long word;
};

// One system.
struct ResSys {
    int atom_off, natoms;
    int cell_off, ncell;
    int lanes;           // per atom
    int part_off;        // this system's first partial-sum record
    int cta_first, ncta;
    int rec_off;         // doubles from a ring slot's start to this system's record
    int always;          // zero skin: rebuild every step
    float cut2;          // FP32 list radius^2
    float3 Lf;
    double thresh2;
    Grid grid;
    PairParams pp;
    MixedParams mp;
    // state
    double *t, *pe, *vir;
    int *need_rebuild, *active, *overflow, *nonfinite, *max_count;
    long long *builds, *steps;
    ResSync* sync;
};

// While one is alive, launches that take the whole GPU are under way on its device
// (lj_gpu.cu).
struct WholeGpu {
    int device;
    explicit WholeGpu(int d);
    ~WholeGpu();
    WholeGpu(const WholeGpu&) = delete;
    WholeGpu& operator=(const WholeGpu&) = delete;
};

// What a launch leaves in pinned host memory when it is done.
struct ResDone {
    double t, pe, vir;
    int overflow, nonfinite;
    long long ticket;  // of the launch; written last
};

struct ResRun {
    int nsteps;
    int kick;        // 0: one force evaluation, nothing moves
    double* ring;
    int ring_cap;    // slots
    int ring_slot;   // doubles per slot
    long long first; // index of the first step (its record goes to slot first mod ring_cap)
    int* intact;     // 0 once a wait ran out
    double* host;    // mapped: the steps' records in a row (may be null)
    ResDone* done;   // mapped (may be null)
    long long ticket;
};

// The launch shape of a system that has the GPU to itself: blocks of as few threads as
// leave one per SM (fewer arrivals at the barrier, all SMs in use), in whole units of
// partial sums, which 8 lanes per atom spread over 2 warps and 16 over 4.
inline int alone_threads(long long threads, int lanes, int sms) {
    const long long unit = lanes == 16 ? 128 : (lanes == 8 ? 64 : 32);
    const long long t = unit * ((threads + sms * unit - 1) / (sms * unit));
    return (int)(t < kResidentMost ? t : kResidentMost);
}

// Which systems step in this form; the others step in graphs (lj_gpu.cu), where a step
// is long enough to hide its launches.  Up to 94 720 atoms every thread has at most one.
// With more, threads take a second atom behind the first, and that is the faster form
// only where the graphs' pair kernel is in its second wave as well.  Measured per step,
// graphs and this form, FP64 (mixed): N = 107 001 56.4 and 67.6 us (45.9, 47.8);
// 120 000 71.8 and 67.3 (54.1, 47.3); 150 000 80.0 and 72.4 (59.8, 52.4); 188 000 90.7
// and 76.5 (67.1, 57.9); with a third atom nothing is gained: 280 000 122.0 and 120.6
// (90.4, 91.5), 370 000 153.0 and 155.5 (114.6, 118.3).
inline bool steps_resident(int N) {
    return N <= kResidentMaxAtoms || (N > kGraphWaveAtoms && N <= 2 * kResidentMaxAtoms);
}

// Shared memory of a block (dynamic): per warp a row's chunk sums or the list build's
// staging; the cells' first slots where every block scans them for itself; and for
// tiny systems the whole system, sorted.
struct ResPiece {
    int js, je;          // candidate slots
    float sx, sy, sz;    // periodic shift
    unsigned entry;      // code of the first cell of the piece
    int home, above;     // slots from which the code's z offset is one and two steps up
};

// A list on its way to memory, and the stencil's pieces it is made from.
struct ResList {
    static constexpr int kStaged = 928;
    unsigned e[kStaged];
    ResPiece piece[27];
};

union ResWarp {
    double xch[kRowWords];
    ListPend pend;
    CellSmem cell;
    ResList list;
};

struct ResTiny {
    float q[3][kTinyAtoms];               // negated positions, sorted
    unsigned short order[kTinyAtoms];     // atoms cell by cell
    unsigned short cell[kTinyAtoms];      // by atom, then (below) by sorted slot
    unsigned short sorted_cell[kTinyAtoms];
    int count[kScanCells];
};

struct ResSmem {
    ResWarp* warp;   // one per warp
    int* start;      // cells + 1
    int cells;       // room
    ResTiny* tiny;   // null: no room
};

__host__ __device__ __forceinline__ size_t res_smem_bytes(int threads, int cells, bool tiny) {
    return sizeof(ResWarp) * (threads / 32) + sizeof(int) * (cells + 4) + (tiny ? sizeof(ResTiny) : 0);
}

__device__ __forceinline__ int res_warps() { return (int)blockDim.x >> 5; }

// The blocks of a launch that share a barrier, whose word counts arrivals in its top
// 12 bits -- the first block adds what makes a full round flip the top bit and leave
// the rest zero, so the word needs no reset -- and, below them, votes: those of even
// and of odd barriers apart (26 bits each), since a block may vote in the next
// barrier before another has read this one's.  The votes are cleared at the end of
// a launch, and in a launch of unbounded length by renew() when either field has seen
// kManyVotes: a barrier adds at most 2047, so that no field ever carries.
constexpr unsigned kManyVotes = 1u << 12;
constexpr int kResidentSteps = 4096;  // steps of a launch (lj_gpu.cu): no field fills up
static_assert(kResidentSteps * 2047ll < 1ll << 26, "votes of a launch must fit their field");

struct Group {
    ResSync* sync;
    int rank, n;
    int* intact;  // 0 once a wait ran out
    unsigned turn = 0, even = 0, odd = 0;  // barriers passed, votes seen in them

    __device__ __forceinline__ Group(ResSync* s, int r, int blocks, int* i) : sync(s), rank(r), n(blocks), intact(i) {}

    __device__ __forceinline__ unsigned long long arrive(bool vote) const {
        unsigned long long old, inc = (unsigned long long)(rank == 0 ? 2048 - (n - 1) : 1) << 52;
        if (vote) inc += 1ull << (turn & 1 ? 26 : 0);
        // (a release at GPU scope: it also covers what the block's other threads wrote
        // before the __syncthreads ahead of it)
        asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;"
                     : "=l"(old)
                     : "l"(&sync->word), "l"(inc)
                     : "memory");
        return old;
    }
    // The word once the last block has arrived; its lowest bit pattern is never all
    // ones, which stands for a wait that ran out.
    __device__ __forceinline__ unsigned long long wait(unsigned long long old) const {
        for (int it = 0; it < kResidentPolls; ++it) {
            unsigned long long now;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(&sync->word) : "memory");
            if ((now ^ old) >> 63) return now;
        }
        atomicExch(intact, 0);
        return ~0ull;
    }
    // All threads of the group's blocks; *any: whether some thread voted.  False when
    // the wait ran out.
    __device__ __forceinline__ bool barrier(bool vote = false, bool* any = nullptr) {
        __shared__ unsigned long long word;
        const bool mine = __syncthreads_or(vote) != 0;
        if (n == 1) {
            if (any) *any = mine;
            return true;
        }
        if (threadIdx.x == 0) word = wait(arrive(mine));
        __syncthreads();
        const unsigned long long w = word;
        if (w == ~0ull) return false;
        const bool second = (turn & 1) != 0;
        const unsigned votes = (unsigned)(w >> (second ? 26 : 0)) & 0x3ffffffu;
        if (any) *any = votes != (second ? odd : even);
        if (second) odd = votes; else even = votes;
        ++turn;
        return true;
    }
    // Whether the votes are due for renew(); the same in every block of the group.
    __device__ __forceinline__ bool many() const { return max(even, odd) >= kManyVotes; }
    // Clear the votes (all threads of the group's blocks; false when a wait ran out).
    // Once the first barrier is passed every block has read the votes of those before it;
    // none is cast until the second is.
    __device__ __forceinline__ bool renew() {
        if (!barrier()) return false;
        if (rank == 0 && threadIdx.x == 0) clear_votes();
        if (!barrier()) return false;
        even = odd = 0;
        return true;
    }
    // the launch's end: one block, after the last barrier
    __device__ __forceinline__ void clear_votes() const { atomicAnd(&sync->word, ~0ull << 52); }
};

__device__ __forceinline__ double& comp(double4* p, int i, int k) { return reinterpret_cast<double*>(p + i)[k]; }
__device__ __forceinline__ float& comp(float4* p, int i, int k) { return reinterpret_cast<float*>(p + i)[k]; }

// |e|^2 of an atom whose axes k are held by lanes k mod LANES, in axis order.
template <int LANES>
__device__ __forceinline__ double lanes_norm2(const double (&e)[3]) {
    double m = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = LANES == 1 ? e[k] : __shfl_sync(0xffffffffu, e[k], k % LANES, LANES);
        m = fma(v, v, m);
    }
    return m;
}

// First half kick and drift of the launch's first step (kick_drift_kernel); whether
// one of this thread's atoms is out of the list's skin.
template <bool MIXED>
__device__ __forceinline__ bool res_drift(const ResSys& S, const ResArrays& A, int rank) {
    bool far = false;
    for (int a = rank * blockDim.x + threadIdx.x; a < S.natoms; a += S.ncta * blockDim.x) {
        const int i = S.atom_off + a;
        Soa s{A.soa[0], A.N};
        double m = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double v = kick(s.at(VX + k, i), s.at(FX + k, i), S.pp.dt);
            double inc = __dmul_rn(v, S.pp.dt);
            double xn = wrap(__dadd_rn(comp(A.pos[0], i, k), inc), S.pp.L[k]);
            double dn = __dadd_rn(s.at(DX + k, i), inc);
            s.at(VX + k, i) = v;
            s.at(DX + k, i) = dn;
            comp(A.pos[1], i, k) = xn;
            double e = dn - A.bd[(size_t)k * A.N + i];
            m = fma(e, e, m);
            if (MIXED) comp(A.posl[1], i, k) = (float)(A.bx[(size_t)k * A.N + i] + e);
        }
        far |= m > S.thresh2;
    }
    return far;
}

// The rows of one warp's 32 / LANES atoms (from atom a0 of the system) at the
// positions in buffer `cur`, the second half kick and the partial sums; then the
// next step's kick and drift into the other buffer, or on the last step the whole
// state into the first buffers.  Whether this thread's atom is out of the skin.
template <int LANES, bool SMALL, bool MIXED>
__device__ __forceinline__ bool res_force(const ResSys& S, const ResArrays& A, int a0, int cur, int sb, bool do_kick,
                                          bool last, double* partials, double* xch) {
    const int lane = threadIdx.x & 31, l = lane % LANES, a = a0 + lane / LANES, i = S.atom_off + a;
    const bool own = a < S.natoms;
    const Soa s{A.soa[sb], A.N}, out{A.soa[0], A.N};
    const int* const count = own ? A.cnt + i : nullptr;
    // with an axis per lane, what the epilogue needs is loaded ahead of the row
    constexpr bool kAhead = LANES >= 4;
    double v_l = 0, d_l = 0, bd_l = 0, bx_l = 0;
    if (kAhead && own && l < 3) {
        v_l = s.at(VX + l, i);
        d_l = s.at(DX + l, i);
        if (!last) bd_l = A.bd[(size_t)l * A.N + i];
        if (MIXED && !last) bx_l = A.bx[(size_t)l * A.N + i];
    }
    RowSums<LANES> r;
    double x3[3] = {0, 0, 0};
    if (MIXED) {
        const float4 xl = own ? A.posl[cur][i] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (kAhead && own && l < 3) x3[0] = comp(A.pos[cur], i, l);
        row_mixed<LANES, false, false>(A.posl[cur], A.nbr + i, A.N, A.cap >> 2, count, lane, xl, S.mp, xch, r);
    } else {
        const double4 xi = own ? ld_neighbour<false>(A.pos[cur] + i) : make_double4(0.0, 0.0, 0.0, 0.0);
        row_lj<LANES, SMALL, false>(A.pos[cur], A.nbr + i, A.N, A.cap >> 2, count, lane, xi, near_face(xi, S.pp), S.pp, xch,
                                   r);
        x3[0] = xi.x; x3[1] = xi.y; x3[2] = xi.z;
    }
    double acc[4];  // sum v^2, pe, w, sum d^2 of the atom
    r.energy(S.pp, acc[1], acc[2]);
    double vk[3] = {0, 0, 0}, dk[3] = {0, 0, 0}, e[3] = {0, 0, 0};
    if (own) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (LANES > 1 && k % LANES != l) continue;
            const double f = r.own(k);
            double v = kAhead ? v_l : s.at(VX + k, i), d = kAhead ? d_l : s.at(DX + k, i);
            double x = MIXED ? (kAhead ? x3[0] : comp(A.pos[cur], i, k)) : x3[k];
            if (do_kick) v = kick(v, f, S.pp.dt);
            vk[k] = v;
            dk[k] = d;
            if (last) {
                out.at(VX + k, i) = v;
                out.at(FX + k, i) = f;
                if (sb) out.at(DX + k, i) = d;
                if (cur) comp(A.pos[0], i, k) = x;
            } else {
                v = kick(v, f, S.pp.dt);
                double inc = __dmul_rn(v, S.pp.dt);
                double xn = wrap(__dadd_rn(x, inc), S.pp.L[k]);
                double dn = __dadd_rn(d, inc);
                s.at(VX + k, i) = v;
                s.at(DX + k, i) = dn;
                comp(A.pos[cur ^ 1], i, k) = xn;
                e[k] = dn - (kAhead ? bd_l : A.bd[(size_t)k * A.N + i]);
                if (MIXED) comp(A.posl[cur ^ 1], i, k) = (float)((kAhead ? bx_l : A.bx[(size_t)k * A.N + i]) + e[k]);
            }
        }
        if (last && sb && l == 0) A.ids[0][i] = A.ids[1][i];
    }
    const bool far = !last && lanes_norm2<LANES>(e) > S.thresh2;
    acc[0] = lanes_norm2<LANES>(vk);
    acc[3] = lanes_norm2<LANES>(dk);
    if (!own) acc[1] = acc[2] = 0.0;
    unit_partials<LANES>(acc, a, S.natoms, partials + 4 * (size_t)S.part_off);
    return far;
}

// finalize_kernel's sums over the system's partials and its record, by one block:
// the 1024 strided sums and the tree over 32 warps in the same order, the block's warps
// taking the 32 in turn.
__device__ __forceinline__ void res_finalize(const ResSys& S, const ResRun& R, const double* partials, int step) {
    __shared__ double sm[32][4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nparts = (S.natoms + kUnit - 1) / kUnit;
    const double4* const p = reinterpret_cast<const double4*>(partials) + S.part_off;
    for (int vw = warp; vw < 32; vw += res_warps()) {
        double acc[4] = {0, 0, 0, 0};
        if (32 * vw < nparts) {  // uniform across the warp
            for (int b = 32 * vw + lane; b < nparts; b += 1024) {
                const double4 t = ld_neighbour<false>(p + b);
                acc[0] += t.x;
                acc[1] += t.y;
                acc[2] += t.z;
                acc[3] += t.w;
            }
            warp_sum<4>(acc);
        }
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < 4; ++q) sm[vw][q] = acc[q];
    }
    __syncthreads();
    if (warp == 0) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = sm[lane][q];
        warp_sum<4>(v);
        if (lane == 0) {
            double pe = 0.5 * v[1], vir = 0.5 * v[2], ke = 0.5 * v[0];
            *S.pe = pe;
            *S.vir = vir;
            if (R.kick) {
                double t = *S.t + S.pp.dt;  // integrator.cpp:85
                *S.t = t;
                *S.steps += 1;
                double* out = R.ring + (size_t)((R.first + step) % R.ring_cap) * R.ring_slot + S.rec_off;
                out[0] = t;
                out[1] = ke;
                out[2] = pe;
                out[3] = pe + ke;
                out[4] = vir;
                out[5] = (2. / 3.) * ke / (double)S.natoms;
                out[6] = v[3] / (double)S.natoms;
                if (R.host) {
                    double* h = R.host + 7 * (size_t)step;
#pragma unroll
                    for (int q = 0; q < 7; ++q) h[q] = out[q];
                }
                if (!isfinite(ke)) *S.nonfinite = 1;
            }
            if (!isfinite(pe) || !isfinite(vir)) *S.nonfinite = 1;
        }
    }
    __syncthreads();
}

// Move the state of slot `from` in the buffers (cur, sb) to slot `to` in the others.
template <bool MIXED>
__device__ __forceinline__ void res_move_to(const ResSys& S, const ResArrays& A, int from, int to, int cur, int sb) {
    const Soa s{A.soa[sb], A.N}, out{A.soa[sb ^ 1], A.N};
    const double4 x = A.pos[cur][from];
    A.pos[cur ^ 1][to] = x;
    A.posn.set(to, x);
    A.ids[sb ^ 1][to] = A.ids[sb][from];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        out.at(VX + q, to) = s.at(VX + q, from);  // the force is not needed across a rebuild
        double d = s.at(DX + q, from);
        out.at(DX + q, to) = d;
        A.bd[(size_t)q * A.N + to] = d;
    }
    if (MIXED) {  // as copy_back_kernel
        const double xs[3] = {x.x, x.y, x.z};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            int cc = cell_coord(xs[q], S.grid.ratio[q], S.grid.n[q]);
            double o = (double)cc * (1.0 / S.grid.ratio[q]);
            double loc = xs[q] - o;
            A.bx[(size_t)q * A.N + to] = loc;
            comp(A.posl[cur ^ 1], to, q) = (float)loc;
        }
    }
}

// One warp: the list of slot i.  The lanes set up the pieces of the stencil (runs of
// consecutive slots with one periodic shift: the cells of a box under 3 cells per
// axis, otherwise the columns, split where they wrap), then test 32 candidates at
// a time, three pieces' loads in flight, and append the hits in candidate order:
// entries and order are those of build_small_list_kernel and of build_atom_lists.
// Returns the list's length before the cut at the capacity.
// (ca, cb, cc): the atom's cell; at(j): the negated position of slot j.
template <bool SMALL, class At>
__device__ __forceinline__ int res_atom_list(const ResSys& S, const ResArrays& A, const int* start, int ca, int cb, int cc,
                                             int i, At at, ResList& sm, int lane) {
    const Grid& g = S.grid;
    unsigned* const list = reinterpret_cast<unsigned*>(A.nbr);
    ResPiece* const pieces = sm.piece;
    float3 xi = at(i);
    xi.x = -xi.x; xi.y = -xi.y; xi.z = -xi.z;
    const int nz = g.n[2];
    const int npc = SMALL ? 3 : (cc == 0 || cc == nz - 1 ? 2 : 1), np = 9 * npc;
    __syncwarp();
    if (lane < np) {
        const int col = lane / npc, pc = lane % npc, a = col / 3 - 1, b = col % 3 - 1;
        int na = ca + a, nb = cb + b;
        const int ia = na < 0 ? -1 : (na >= g.n[0] ? 1 : 0), ib = nb < 0 ? -1 : (nb >= g.n[1] ? 1 : 0);
        na -= ia * g.n[0];
        nb -= ib * g.n[1];
        const int c0 = g.flat(na, nb, 0);
        ResPiece p;
        int ic = 0;
        if (SMALL) {
            int nc = cc + pc - 1;
            ic = nc < 0 ? -1 : (nc >= nz ? 1 : 0);
            nc -= ic * nz;
            p.js = start[c0 + nc];
            p.je = start[c0 + nc + 1];
            p.entry = offset_code(ia, ib, ic);
            p.home = p.above = INT_MAX;
            p.sx = ia * S.Lf.x;
            p.sy = ib * S.Lf.y;
            p.sz = ic * S.Lf.z;
        } else {
            int d0 = -1, d1 = 1;  // z offsets of the piece's cells
            if (cc == 0) {
                ic = pc == 0 ? -1 : 0;
                d0 = pc == 0 ? -1 : 0;
                d1 = pc == 0 ? -1 : 1;
            } else if (cc == nz - 1) {
                ic = pc == 0 ? 0 : 1;
                d0 = pc == 0 ? -1 : 1;
                d1 = pc == 0 ? 0 : 1;
            }
            p.js = start[c0 + cc + d0 - ic * nz];
            p.je = start[c0 + cc + d1 - ic * nz + 1];
            p.entry = offset_code(a, b, d0);
            p.home = d0 < 0 && d1 >= 0 ? start[c0 + cc] : INT_MAX;
            p.above = d0 < 1 && d1 >= 1 ? start[c0 + cc + 1] : INT_MAX;
            p.sx = xi.x - ia * S.Lf.x;
            p.sy = xi.y - ib * S.Lf.y;
            p.sz = xi.z - ic * S.Lf.z;
        }
        pieces[lane] = p;
    }
    __syncwarp();
    int n = 0;
    auto test = [&](const ResPiece& p, int j, const float3& xj) {
        bool hit = false;
        if (j < p.je) {
            float dx, dy, dz;
            if (SMALL) {
                dx = (xi.x + xj.x) - p.sx;  // the candidates are negated
                dy = (xi.y + xj.y) - p.sy;
                dz = (xi.z + xj.z) - p.sz;
            } else {
                dx = p.sx + xj.x;
                dy = p.sy + xj.y;
                dz = p.sz + xj.z;
            }
            hit = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < S.cut2 && j != i;
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        const int k = n + __popc(m & ((1u << lane) - 1u));
        if (hit) {
            unsigned e = make_entry((unsigned)j, p.entry);
            if (!SMALL) e += (j >= p.home ? 16u : 0u) + (j >= p.above ? 16u : 0u);
            if (k < ResList::kStaged)
                sm.e[k] = e;
            else if (k < A.cap)
                list[((size_t)(k >> 2) * A.N + i) * 4 + (k & 3)] = e;
        }
        n += __popc(m);
    };
    const float3 none = make_float3(0.f, 0.f, 0.f);
    for (int p0 = 0; p0 < np; p0 += 3) {
        float3 x[3][2];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            const int j = pieces[p0 + u].js + lane, je = pieces[p0 + u].je;
            x[u][0] = j < je ? at(j) : none;
            x[u][1] = j + 32 < je ? at(j + 32) : none;
        }
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            const ResPiece p = pieces[p0 + u];
            if (p.js < p.je) test(p, p.js + lane, x[u][0]);
            if (p.js + 32 < p.je) test(p, p.js + 32 + lane, x[u][1]);
            for (int j0 = p.js + 64; j0 < p.je; j0 += 32) test(p, j0 + lane, j0 + lane < p.je ? at(j0 + lane) : none);
        }
    }
    // pad the last group with the ghost slot; whole staged groups to memory
    const int m = min(n, A.cap), pad = m + lane, end = (m + 3) & ~3;
    if (lane == 0) A.cnt[i] = m;
    if (pad < end) {
        if (pad < ResList::kStaged)
            sm.e[pad] = make_entry((unsigned)A.N, kGhostCode);
        else
            list[((size_t)(pad >> 2) * A.N + i) * 4 + (pad & 3)] = make_entry((unsigned)A.N, kGhostCode);
    }
    __syncwarp();
    for (int q = lane; 4 * q < min(end, (int)ResList::kStaged); q += 32)
        A.nbr[(size_t)q * A.N + i] = *reinterpret_cast<const uint4*>(&sm.e[4 * q]);
    return n;
}

// Exclusive scan of one int per thread over the block.
__device__ __forceinline__ int res_block_scan(int x, int* total) {
    __shared__ int warp_tot[33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int w = lane < res_warps() ? warp_tot[lane] : 0;
        int wi = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, wi, off);
            if (lane >= off) wi += y;
        }
        warp_tot[lane] = wi - w;
        if (lane == 31) warp_tot[32] = wi;
    }
    __syncthreads();
    const int res = incl - x + warp_tot[warp];
    *total = warp_tot[32];
    __syncthreads();
    return res;
}

// Exclusive scan of the counts of cells [c0, c1) of the system by one block, from
// `base` on; the first slots go to `start` (indexed like the counts).
__device__ __forceinline__ void res_scan(const int* count, int* start, int c0, int c1, int base) {
    for (int t0 = c0; t0 < c1; t0 += 8 * blockDim.x) {
        const int idx = t0 + 8 * threadIdx.x;
        int c[8], sum = 0, tot;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            c[q] = idx + q < c1 ? count[idx + q] : 0;
            sum += c[q];
        }
        int ex = res_block_scan(sum, &tot) + base;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (idx + q < c1) start[idx + q] = ex;
            ex += c[q];
        }
        base += tot;
    }
}

// The first slots of a group's cells (from `base` on) by all of its blocks, after a
// barrier: small grids every block for itself in shared memory, larger ones in
// global memory, a range per block, with two barriers.  Null when a wait ran out.
__device__ __forceinline__ const int* group_scan(Group& grp, const int* count, int ncell, int base, int natoms,
                                                 int* start_global, int* start_shared, int cells,
                                                 int* tiles) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (ncell <= cells) {
        res_scan(count, start_shared, 0, ncell, base);
        if (tid == 0) start_shared[ncell] = base + natoms;
        __syncthreads();
        return start_shared;
    }
    const int per = (ncell + grp.n - 1) / grp.n;
    const int c0 = min(grp.rank * per, ncell), c1 = min(c0 + per, ncell);
    __shared__ int red[32];
    auto block_total = [&](int v) {
        v = __reduce_add_sync(0xffffffffu, v);
        __syncthreads();
        if (lane == 0) red[warp] = v;
        __syncthreads();
        int t = 0;
        for (int q = 0; q < res_warps(); ++q) t += red[q];
        return t;
    };
    int v = 0;
    for (int c = c0 + tid; c < c1; c += blockDim.x) v += count[c];
    v = block_total(v);
    if (tid == 0) tiles[grp.rank] = v;
    if (!grp.barrier()) return nullptr;
    v = 0;
    for (int q = tid; q < grp.rank; q += blockDim.x) v += tiles[q];
    v = block_total(v);
    res_scan(count, start_global, c0, c1, base + v);
    if (grp.rank == 0 && tid == 0) start_global[ncell] = base + natoms;
    if (!grp.barrier()) return nullptr;
    return start_global;
}

// What a list takes, about, in microseconds: an atom by a warp; up to 32 atoms of a cell
// by a warp; an atom by a thread, apart from what that takes per atom of a cell.  Weights
// that order the three forms; measured in us per step (FP64, T 1.5), by atom, by cell, by
// thread and as they choose:
//           rho 0.05                 0.2                     0.45                    0.8442
//   4097    9.8 10.7 10.7  9.8    10.6 10.9 12.9 10.7    10.0 11.1 12.8 10.0    11.1 13.5 15.6 11.1
//  12 000  13.5 18.2 11.1 11.1    15.2 12.8 12.8 12.8    16.4 13.3 15.1 16.5    19.0 16.5 18.8 19.2
//  31 987  20.3 25.0 13.3 13.3    25.8 21.7 18.0 18.0    28.4 22.1 21.3 21.2    33.4 23.9 26.6 23.8
//  90 000  36.3 47.2 16.6 16.5    43.6 33.6 23.4 23.2    52.1 35.4 30.9 30.7    61.8 42.0 40.3 40.1
// 189 440  72.2 91.6 33.2 33.0    84.5 67.4 45.2 45.0   102.2 69.3 60.8 60.7   123.6 87.7 83.7 83.1
// (from 6000 to 20 000 atoms by cell would be up to a fifth faster than what they choose).
constexpr int kAtomCost = 2, kCellCost = 25, kThreadCost = 5, kThreadCellCost = 2;

// The rebuild of a tiny system: every block bins and sorts all of its atoms for itself
// in shared memory, so that nothing is waited for before the lists are done; the
// moves and the lists are shared out.
template <bool SMALL, bool MIXED>
__device__ __forceinline__ void res_rebuild_tiny(const ResSys& S, const ResArrays& A, int rank, int cur, int sb,
                                                 ResSmem& sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Grid& g = S.grid;
    ResTiny& t = *sm.tiny;
    for (int c = tid; c < S.ncell; c += blockDim.x) t.count[c] = 0;
    __syncthreads();
    for (int i = tid; i < S.natoms; i += blockDim.x) {
        const double4 x = ld_neighbour<false>(A.pos[cur] + i);
        const int c = g.flat(cell_coord(x.x, g.ratio[0], g.n[0]), cell_coord(x.y, g.ratio[1], g.n[1]),
                             cell_coord(x.z, g.ratio[2], g.n[2]));
        t.cell[i] = (unsigned short)c;
        atomicAdd(&t.count[c], 1);
    }
    __syncthreads();
    res_scan(t.count, sm.start, 0, S.ncell, 0);
    if (tid == 0) sm.start[S.ncell] = S.natoms;
    __syncthreads();
    for (int c = tid; c < S.ncell; c += blockDim.x) t.count[c] = 0;
    __syncthreads();
    for (int i = tid; i < S.natoms; i += blockDim.x) {
        const int c = t.cell[i];
        t.order[sm.start[c] + atomicAdd(&t.count[c], 1)] = (unsigned short)i;
    }
    __syncthreads();
    for (int i = tid; i < S.natoms; i += blockDim.x) {
        const int c = t.cell[i], b = sm.start[c], e = sm.start[c + 1];
        int to = b;
        for (int k = b; k < e; ++k) to += t.order[k] < i ? 1 : 0;
        const double4 x = ld_neighbour<false>(A.pos[cur] + i);
        t.q[0][to] = -(float)x.x;
        t.q[1][to] = -(float)x.y;
        t.q[2][to] = -(float)x.z;
        t.sorted_cell[to] = (unsigned short)c;
        if ((i / 32) % S.ncta == rank) res_move_to<MIXED>(S, A, i, to, cur, sb);
    }
    __syncthreads();
    int wmax = 0;
    for (int a = rank * res_warps() + warp; a < S.natoms; a += S.ncta * res_warps()) {
        const int c = t.sorted_cell[a];
        wmax = max(wmax, res_atom_list<SMALL>(
                             S, A, sm.start, c / (g.n[1] * g.n[2]), (c / g.n[2]) % g.n[1], c % g.n[2], a,
                             [&](int j) { return make_float3(t.q[0][j], t.q[1][j], t.q[2][j]); }, sm.warp[warp].list, lane));
    }
    if (lane == 0 && wmax > 0) {
        if (S.max_count) atomicMax(S.max_count, wmax);
        if (wmax > A.cap) atomicExch(S.overflow, 1);
    }
}

// The list rebuild at the positions in buffer `cur` (state in buffer `sb`),
// leaving both in the other buffers.  False when a wait ran out.
template <bool SMALL, bool MIXED>
__device__ __forceinline__ bool res_rebuild(const ResSys& S, const ResArrays& A, Group& grp, int cur, int sb,
                                            ResSmem& sm) {
    const int rank = grp.rank, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int first = rank * blockDim.x + tid, stride = S.ncta * blockDim.x, warps = S.ncta * res_warps();
    const Grid& g = S.grid;
    if (sm.tiny && S.natoms <= kTinyAtoms && S.ncell <= kScanCells) {
        res_rebuild_tiny<SMALL, MIXED>(S, A, rank, cur, sb, sm);
        return grp.barrier();
    }
    int* const count = A.count + S.cell_off;
    for (int a = first; a < S.natoms; a += stride) {
        const int i = S.atom_off + a;
        const double4 x = A.pos[cur][i];
        const int c = g.flat(cell_coord(x.x, g.ratio[0], g.n[0]), cell_coord(x.y, g.ratio[1], g.n[1]),
                             cell_coord(x.z, g.ratio[2], g.n[2]));
        A.cell_of[i] = c;
        A.rank[i] = atomicAdd(&count[c], 1);
    }
    if (!grp.barrier()) return false;
    const int* const start = group_scan(grp, count, S.ncell, S.atom_off, S.natoms, A.start + S.cell_off, sm.start,
                                        sm.cells, A.tiles + S.cta_first);
    if (!start) return false;
    for (int a = first; a < S.natoms; a += stride) {
        const int i = S.atom_off + a;
        A.order[start[A.cell_of[i]] + A.rank[i]] = i;
    }
    if (!grp.barrier()) return false;
    for (int c = first; c < S.ncell; c += stride) count[c] = 0;  // ready for the next binning
    for (int a = first; a < S.natoms; a += stride) {
        // an atom's place among its cell's, which are ordered by slot, is the number of
        // them in lower slots
        const int i = S.atom_off + a, c = A.cell_of[i], b = start[c], e = start[c + 1];
        int to = b;
        for (int k = b; k < e; ++k) to += A.order[k] < i ? 1 : 0;
        res_move_to<MIXED>(S, A, i, to, cur, sb);
    }
    if (!grp.barrier()) return false;
    // lists: the form whose slowest worker is the sooner done
    int wmax = 0;
    const double4* const pos = A.pos[cur ^ 1];
    const int by_atom = kAtomCost * ((S.natoms + warps - 1) / warps),
              by_cell = kCellCost * ((S.ncell + warps - 1) / warps) * (1 + S.natoms / (32 * S.ncell)),
              by_thread = (kThreadCost + kThreadCellCost * S.natoms / S.ncell) * ((S.natoms + stride - 1) / stride);
    if (SMALL || (by_atom <= by_cell && by_atom <= by_thread)) {
        for (int a = rank * res_warps() + warp; a < S.natoms; a += warps) {
            const int i = S.atom_off + a;
            const double4 x = ld_neighbour<false>(pos + i);
            wmax = max(wmax, res_atom_list<SMALL>(S, A, start, cell_coord(x.x, g.ratio[0], g.n[0]),
                                                  cell_coord(x.y, g.ratio[1], g.n[1]), cell_coord(x.z, g.ratio[2], g.n[2]),
                                                  i, [&](int j) { return A.posn.at(j); }, sm.warp[warp].list, lane));
        }
    } else if (by_cell <= by_thread) {
        for (int c = rank * res_warps() + warp; c < S.ncell; c += warps)
            wmax = max(wmax, build_cell_lists<false>(c / (g.n[1] * g.n[2]), (c / g.n[2]) % g.n[1], c % g.n[2], g, start,
                                                     A.posn, S.Lf, S.cut2, A.cap, A.nbr, A.cnt, A.N, sm.warp[warp].cell,
                                                     lane));
    } else {
        for (int a0 = rank * blockDim.x; a0 < S.natoms; a0 += stride) {
            const bool own = a0 + tid < S.natoms;
            const int i = S.atom_off + min(a0 + tid, S.natoms - 1);
            wmax = max(wmax, build_atom_lists<false>(own, i, pos[i], g, start, A.posn, S.Lf, S.cut2, A.cap, A.nbr, A.cnt,
                                                     A.N, sm.warp[warp].pend));
        }
    }
    wmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)wmax);
    if (lane == 0 && wmax > 0) {
        if (S.max_count) atomicMax(S.max_count, wmax);
        if (wmax > A.cap) atomicExch(S.overflow, 1);
    }
    return grp.barrier();
}

template <int LANES, bool SMALL, bool MIXED>
__device__ __forceinline__ bool res_forces(const ResSys& S, const ResArrays& A, int cur, int sb, bool kick, bool last,
                                           double* partials, ResSmem& sm) {
    constexpr int kPerWarp = 32 / LANES;
    const int rank = (int)blockIdx.x - S.cta_first, warp = threadIdx.x >> 5;
    const int per_block = res_warps() * kPerWarp;
    bool far = false;
    if (LANES <= 4) {  // a warp's units are its own
        for (int a = rank * per_block + warp * kPerWarp; a < S.natoms; a += S.ncta * per_block)
            far |= res_force<LANES, SMALL, MIXED>(S, A, a, cur, sb, kick, last, partials, sm.warp[warp].xch);
    } else {
        for (int a = rank * per_block; a < S.natoms; a += S.ncta * per_block)
            far |= res_force<LANES, SMALL, MIXED>(S, A, a + warp * kPerWarp, cur, sb, kick, last, partials,
                                                  sm.warp[warp].xch);
    }
    return far;
}

// BATCH: the block's system comes from a table; otherwise it is `one`, whose
// constants then are operands from the constant bank, and its blocks are as large as
// leaves one per SM (fewer arrivals at the barrier).
template <bool BATCH, bool SMALL, bool MIXED>
static __global__ void __launch_bounds__(BATCH ? kResidentThreads : kResidentMost, BATCH ? kResidentBlocks : 1)
resident_steps_kernel(const __grid_constant__ ResArrays A, const __grid_constant__ ResRun R,
                      const __grid_constant__ ResSys one, const ResSys* __restrict__ systems,
                      const int* __restrict__ cta_sys) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ ResSys table;
    ResSmem sm;
    sm.warp = reinterpret_cast<ResWarp*>(dyn);
    sm.start = reinterpret_cast<int*>(dyn + sizeof(ResWarp) * res_warps());
    sm.cells = BATCH ? kScanCells : kScanCellsAlone;
    sm.tiny = BATCH || one.natoms > kTinyAtoms ? nullptr : reinterpret_cast<ResTiny*>(sm.start + sm.cells + 4);
    if (BATCH) {
        const int* src = reinterpret_cast<const int*>(systems + cta_sys[blockIdx.x]);
        for (int q = threadIdx.x; q < (int)(sizeof(ResSys) / sizeof(int)); q += blockDim.x)
            reinterpret_cast<int*>(&table)[q] = src[q];
        __syncthreads();
    }
    const ResSys& S = BATCH ? table : one;
    if (S.active && !*S.active) return;
    Group grp(S.sync, (int)blockIdx.x - S.cta_first, S.ncta, R.intact);
    const bool fin = grp.rank == S.ncta - 1;  // the block that adds up the records (it has the least to do)
    const bool kick = R.kick != 0;
    int cur = 0, sb = 0;
    long long builds = 0;
    const bool need = *S.need_rebuild != 0;
    bool far = false;
    if (kick) {
        far = res_drift<MIXED>(S, A, grp.rank);
        cur = 1;
    }
    for (int step = 0; step < R.nsteps; ++step) {
        bool open;
        if (!grp.barrier(far && !S.always, &open)) return;
        double* const half = A.partials + (step & 1 ? 4 * (size_t)A.part_stride : 0);
        if (fin && step > 0) res_finalize(S, R, A.partials + (step & 1 ? 0 : 4 * (size_t)A.part_stride), step - 1);
        if (open || S.always || (step == 0 && (need || !kick))) {
            if (!res_rebuild<SMALL, MIXED>(S, A, grp, cur, sb, sm)) return;
            cur ^= 1;
            sb ^= 1;
            ++builds;
        }
        const bool last = step == R.nsteps - 1;
        switch (S.lanes) {
            case 16: far = res_forces<16, SMALL, MIXED>(S, A, cur, sb, kick, last, half, sm); break;
            case 8: far = res_forces<8, SMALL, MIXED>(S, A, cur, sb, kick, last, half, sm); break;
            case 4: far = res_forces<4, SMALL, MIXED>(S, A, cur, sb, kick, last, half, sm); break;
            case 2: far = res_forces<2, SMALL, MIXED>(S, A, cur, sb, kick, last, half, sm); break;
            default: far = res_forces<1, SMALL, MIXED>(S, A, cur, sb, kick, last, half, sm); break;
        }
        cur ^= 1;
    }
    // the last record: every block arrives, the finalizing one waits
    __syncthreads();
    if (S.ncta > 1 && !fin) {
        if (threadIdx.x == 0) grp.arrive(false);
        return;
    }
    if (!grp.barrier()) return;
    res_finalize(S, R, A.partials + (R.nsteps & 1 ? 0 : 4 * (size_t)A.part_stride), R.nsteps - 1);
    if (threadIdx.x == 0) {
        grp.clear_votes();
        *S.need_rebuild = 0;
        *S.builds += builds;
        if (R.done) {
            R.done->t = *S.t;
            R.done->pe = *S.pe;
            R.done->vir = *S.vir;
            R.done->overflow = *S.overflow;
            R.done->nonfinite = *S.nonfinite;
            __threadfence_system();
            R.done->ticket = R.ticket;
        }
    }
}

}  // namespace ljb
