// The persistent chain kernel (run_mc + movemc on the device) and its launch helpers.
// Included by the engine (types and declarations) and by one instantiation file per LJ type
// count (yamc_chain_inst.cu, compiled once per count), so the kernel variants compile in parallel.
#pragma once

#include <cooperative_groups.h>
#include <cuda_pipeline.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <type_traits>

#include "yamc_device.cuh"
#include "yamc_internal.h"

#define CUDA_TRY(expr)                                                                        \
    do {                                                                                      \
        cudaError_t _e = (expr);                                                              \
        if (_e != cudaSuccess) {                                                              \
            (void)cudaGetLastError(); /* the next call must not meet it */                    \
            yamc::set_error(std::string(#expr) + ": " + cudaGetErrorString(_e));              \
            return YAMC_ECUDA;                                                                \
        }                                                                                     \
    } while (0)

#ifndef YAMC_WIDE_THREADS
#define YAMC_WIDE_THREADS 384  // threads of the wide streamed variant (up to 170 registers each)
#endif

namespace yamc {

namespace cg = cooperative_groups;

// Lets blocks of `kernel` have `bytes` of dynamic shared memory.  The limit belongs to the kernel
// on the device, for the whole process: it is only ever raised, and to all that a block can have, so
// no handle or thread takes back what another has planned with.  Kernels start with 48 KB, their
// static part included, of which none here takes more than 36 (k_rdf_tiles: 33): small requests need
// no query, which takes 0.6 us (a host-driven move makes two).
template <class Kernel>
int grant_smem(Kernel *kernel, size_t bytes) {
    if (bytes <= 12 * 1024) return YAMC_OK;
    cudaFuncAttributes a;
    CUDA_TRY(cudaFuncGetAttributes(&a, kernel));
    if ((long long)bytes <= (long long)a.maxDynamicSharedSizeBytes - (long long)a.sharedSizeBytes) return YAMC_OK;
    int device, optin;
    CUDA_TRY(cudaGetDevice(&device));
    CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  std::max((int)bytes, optin - (int)a.sharedSizeBytes)));
    return YAMC_OK;
}

struct LaunchCfg {
    int G = 0, B = 0, EPT = 0;  // EPT: entries per worker in registers; 0 streamed; -1 streamed, wide CTAs
    int nown_max = 0;
    size_t smem = 0;
};

// ------------------------------------------------------------------------------------------
// the chain kernel
// ------------------------------------------------------------------------------------------
// One thread-block cluster runs one Markov chain.  Warp 0 of every CTA is the control warp:
// its lane 0 draws the random numbers, proposes moves and takes the Metropolis decision
// (redundantly in every CTA, on identical data, so the CTAs agree without talking).  The
// other warps are workers: they run the fused real-space + k-space pass of the current move
// over the CTA's atoms and k-vector entries.  For unbiased moves the control warp prepares
// the next move while the workers run the current pass: after the acceptance draw, and as the next
// molecule's old positions depend on the decision when it is the one being moved, lanes 1 and 2
// prepare two candidates and the decision picks one.  After a hard-core overlap (no acceptance draw)
// the next move starts one number earlier: it is rare, and not prepared.

// per-replica run control, in device memory
struct RunSlot {
    const float *rng;       // stream positions [rng_off, n_rng)
    long long rng_off;
    long long n_rng;
    long long cursor;       // in: start cursor; out: cursor after the last completed move
    long long n_moves;      // moves requested
    long long moves_done;   // out
    yamc_move_record *log;  // optional, n_moves records
    double *rows;           // optional energy rows (9 doubles)
    int max_rows, n_rows;
    int status, accepted;
    double sc[SC_COUNT];    // out: the engine scalars and counters, so the host has them with the slot
    long long cnt[CN_COUNT];
};

struct ChainArgs {
    const DevSys *sys;  // [R]
    RunSlot *run;       // [R]
    int G;              // CTAs per chain (cluster size)
    int nown_max;       // atoms staged per CTA (interleaved ownership: atom j lives in CTA j % G, in slot D.slot[j])
    double2 *scratch;      // [2][(1+nt) S]: molecule old sums, rho deltas (scratch_buf: FP32 pairs in the mixed form)
    long long *prof;       // optional per-phase cycle counters (PH_* layout), CTA 0
};

// phases timed when ChainArgs::prof is set (control lane 0 or worker thread 32 of CTA 0)
enum Phase { PH_CHOOSE = 0, PH_SPECULATE, PH_PROPOSE, PH_TABLES, PH_KSPACE, PH_FILTER, PH_PAIRS, PH_REDUCE,
             PH_OLD_PASS, PH_DECIDE, PH_COMMIT, PH_KSPACE_NEXT, PH_COUNT };

// reduction vector of one pass: the moved molecule's energies, k-space energy change, overlap
// flag and per-atom forces
constexpr int RV_EW = 0, RV_LJ6 = 1, RV_LJ12 = 2, RV_DUC = 3, RV_DUL = 4, RV_OVL = 5, RV_F = 6;
constexpr int kNV = 6 + 3 * kMaxA;

enum PassKind { PASS_OLD = 0, PASS_NEW = 1, PASS_BOTH = 2 };

struct Slot { double x, y, z, q, iq, dhs; int type, pad; };
constexpr int kMaxSpecies = 8;
constexpr int kBlk = 32;  // atoms per bounding box of the pair filter: one warp's lanes
constexpr int kNear = 256;  // near atoms a warp gathers before it tests them against the molecule's slots
constexpr int kPairs = 32 * 2 * kMaxA + 64;  // pairs a warp's queue holds: those of 32 atoms and a rest below 64
constexpr int kBlkList = 96;  // near blocks of one warp: those of kMaxOwn atoms over three warps and more
constexpr int kWarpBuf = (kNear + kPairs + kBlkList) / 2;  // a warp's buffers, ints
constexpr int kWin = 256; // random-stream window held in shared memory
constexpr int kMaxOwn = 8192;  // atoms staged per CTA: a pair names its atom in 13 bits

// ints of the warps' near-atom and pair buffers of a B-thread CTA; at least room for the phase
// tables of two atoms (the mixed form's refresh works in it)
__host__ __device__ inline int wbuf_ints(int B, int kmax) {
    const int warps = (B / 32) * kWarpBuf, tables = 4 + 2 * (3 * 4 * (kmax + 1) + 3);
    return ((warps > tables ? warps : tables) + 1) & ~1;
}
constexpr int kCtl = 32;  // threads of the control warp
constexpr int kChainMaxThreads = 256;  // one CTA per SM, up to 255 registers per thread
constexpr int kChainMaxThreadsWide = YAMC_WIDE_THREADS;  // streamed k entries, more warps, fewer registers

// ------------------------------------------------------------------ spatial staging
// Each CTA stages its atoms in spatial order (k_stage_order), so kBlk consecutive slots hold
// atoms of a compact region; per block a bounding box (centre and half extent per axis, box
// units, float) lets the pair filter skip blocks that lie outside the query sphere.  The box
// holds every staged position p of the block as p = centre + t + n (n integer, |t| <= half);
// kBoxPad widens the half extents beyond the rounding of centre and extent to float.
constexpr double kBoxPad = 1e-6;

__device__ __forceinline__ double wrap_half(double d) { return d - rint(d); }  // into [-1/2, 1/2]

// the block's box from its staged positions, relative to its first atom
__device__ inline void block_box(const double4 *atom_s, int b, int nown, float4 *box_s) {
    const int s0 = b * kBlk, s1 = min(s0 + kBlk, nown);
    const double4 r = atom_s[s0];
    double lx = 0, ly = 0, lz = 0, hx = 0, hy = 0, hz = 0;
    for (int s = s0 + 1; s < s1; ++s) {
        const double4 p = atom_s[s];
        const double tx = wrap_half(p.x - r.x), ty = wrap_half(p.y - r.y), tz = wrap_half(p.z - r.z);
        lx = fmin(lx, tx); ly = fmin(ly, ty); lz = fmin(lz, tz);
        hx = fmax(hx, tx); hy = fmax(hy, ty); hz = fmax(hz, tz);
    }
    box_s[2 * b] = make_float4((float)(r.x + 0.5 * (lx + hx)), (float)(r.y + 0.5 * (ly + hy)),
                               (float)(r.z + 0.5 * (lz + hz)), 0.f);
    box_s[2 * b + 1] = make_float4(__double2float_ru(0.5 * (hx - lx) + kBoxPad), __double2float_ru(0.5 * (hy - ly) + kBoxPad),
                                   __double2float_ru(0.5 * (hz - lz) + kBoxPad), 0.f);
}

// the block's box grown to hold position (x, y, z) as well (an accepted move's new position)
__device__ inline void box_expand(float4 *box_s, int b, double x, double y, double z) {
    float4 c = box_s[2 * b], h = box_s[2 * b + 1];
    const double p[3] = {x, y, z};
    float *cc[3] = {&c.x, &c.y, &c.z}, *hh[3] = {&h.x, &h.y, &h.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double t = wrap_half(p[d] - (double)*cc[d]), e = (double)*hh[d];
        if (t > e || t < -e) {
            const double lo = fmin(-e, t), hi = fmax(e, t);
            *cc[d] = (float)((double)*cc[d] + 0.5 * (lo + hi));
            *hh[d] = __double2float_ru(0.5 * (hi - lo) + kBoxPad);
        }
    }
    box_s[2 * b] = c;
    box_s[2 * b + 1] = h;
}

// false only if no position the box holds is within sqrt(r2) of (qx, qy, qz) under any periodic
// image: per axis the nearest image of the box is |wrap(q - centre)| - half away (or 0)
__device__ __forceinline__ bool box_near(const float4 *box_s, int b, double qx, double qy, double qz, double r2) {
    const float4 c = box_s[2 * b], h = box_s[2 * b + 1];
    const double ex = fmax(fabs(wrap_half(qx - (double)c.x)) - (double)h.x, 0.0);
    const double ey = fmax(fabs(wrap_half(qy - (double)c.y)) - (double)h.y, 0.0);
    const double ez = fmax(fabs(wrap_half(qz - (double)c.z)) - (double)h.z, 0.0);
    return ex * ex + ey * ey + ez * ez < r2;
}

// Order of the staged atoms (one block per chain and CTA, before each chain launch): CTA r of a
// chain of G CTAs owns atoms j = r + G i; they are ordered by the Morton index of their cell on
// an nc^3 grid (nc a power of two <= 16, about four owned atoms per cell), stably (by i) within a
// cell.  Writes D.slot[j] (the slot of atom j in its CTA) and D.atom_of[s G + r] (the atom in
// slot s of CTA r), and the FP32 copy of rho that the mixed form's streamed sweeps read (the
// chain's blocks split its entries).  Shared memory: kStageMaxCells + atoms-per-CTA ints.
constexpr int kStageThreads = 256;
constexpr int kStageMaxCells = 4096;

__device__ __forceinline__ unsigned spread3(unsigned v) {  // bits b of v (b < 4) to bits 3 b
    return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6);
}

__device__ __forceinline__ int cell_axis(double u, int nc) {
    const double w = u - floor(u);
    return min((int)(w * nc), nc - 1);
}

static __global__ void __launch_bounds__(kStageThreads) k_stage_order(const DevSys *sys, int G) {
    extern __shared__ int st_smem[];
    const int rank = blockIdx.x % G;
    const DevSys &D = sys[blockIdx.x / G];
    const int tid = threadIdx.x, lane = tid & 31;
    const int nown = (D.N - rank + G - 1) / G;
    for (int i = rank * kStageThreads + tid, n = (1 + D.nt) * D.S; i < n; i += G * kStageThreads) {
        const double2 r = D.rho[i];
        D.rho_f[i] = make_float2((float)r.x, (float)r.y);
    }
    int nc = 1;
    while (nc < 16 && 4 * (2 * nc) * (2 * nc) * (2 * nc) <= nown) nc *= 2;
    const int ncell = nc * nc * nc;
    int *hist = st_smem, *key = st_smem + kStageMaxCells;
    for (int c = tid; c < ncell; c += kStageThreads) hist[c] = 0;
    __syncthreads();
    for (int i = tid; i < nown; i += kStageThreads) {
        const double4 p = D.atom[rank + G * i];
        const int k = (int)(spread3(cell_axis(p.x, nc)) | (spread3(cell_axis(p.y, nc)) << 1) |
                            (spread3(cell_axis(p.z, nc)) << 2));
        key[i] = k;
        atomicAdd(&hist[k], 1);
    }
    __syncthreads();
    if (tid < 32) {
        // exclusive prefix of the cell counts: each lane a contiguous run of cells
        const int per = (ncell + 31) / 32;
        const int lo = min(lane * per, ncell), hi = min(lo + per, ncell);
        int sum = 0;
        for (int c = lo; c < hi; ++c) sum += hist[c];
        int x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        int run = x - sum;
        for (int c = lo; c < hi; ++c) { const int h = hist[c]; hist[c] = run; run += h; }
        __syncwarp();
        // stable placement, 32 atoms at a time: atoms of one cell take consecutive slots in i order
        for (int i0 = 0; i0 < nown; i0 += 32) {
            const int i = i0 + lane;
            const int k = i < nown ? key[i] : -1;
            const unsigned peers = __match_any_sync(0xffffffffu, k);
            const int before = __popc(peers & ((1u << lane) - 1u));
            const int pos = i < nown ? hist[k] + before : 0;
            __syncwarp();
            if (i < nown && before == __popc(peers) - 1) hist[k] = pos + 1;
            if (i < nown) key[i] = pos;
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = tid; i < nown; i += kStageThreads) {
        const int j = rank + G * i, s = key[i];
        D.slot[j] = s;
        D.atom_of[YAMC_IX(s * G + rank, D.N + 16)] = j;
    }
}

// a prepared move: the molecule, its atoms at the old and proposed positions, the proposal
struct Cand {
    int valid, imol, first, na;
    long long cur_start;  // stream position at the start of the move
    long long cur_prop;   // stream position after the proposal
    double mu_old[3];     // dipole of the molecule at the old positions
    Slot slot[2 * kMaxA]; // [0, na): proposed positions, [na, 2na): old positions
    double mass[kMaxA];
    MoveState mv;
};

// the CTA's staged atoms and buffers (shared memory), as the real-space part reads them
struct StageView {
    const double4 *atom;   // x, y, z, q by staging slot
    const int2 *meta;      // molecule, LJ type
    const float4 *box;     // bounding boxes of the blocks
    const double *dhs_ts, *lj;  // hard cores by LJ type; LJ tables
    double *red;           // [worker warp][kNV]
    int *wbuf;             // the warps' near atoms and pairs
    int nown, grank, gsize;
};

struct ChainShared {
    StageView view;
    Cand cand[4];         // the move being evaluated (cand[icur]) and up to three prepared next moves
    int icur;             // buffer of the move being evaluated
    int spec[3];          // buffers of the candidates: after an overlap (never valid) / after a draw / accepted same molecule
    int abort, accepted, overlap, last_mol, spec_ok;
    int prop_out;         // the stream ran out in the proposal (a word of its own: see there)
    long long cursor;     // stream position after the last completed move
    long long icycle, mic;
    double eold[3];
    // the biased proposal on two warps: the rotation thread's result and stream positions
    MoveState mrot;
    long long disp_end, rot_start, rot_end;
    int disp_out, rot_out;
    double sc[SC_COUNT];
    double lx[kMaxA], ly[kMaxA], lz[kMaxA];  // last accepted move (staged copies may lag in other CTAs)
    // the move just decided, for the workers' commit (its candidate buffer may be taken meanwhile)
    int mv_first, mv_na, mv_tmask, mv_simple, mv_slot[kMaxA];
    double tot[kNV];
    double du[4];
    int flags;
    // molecule species (runs of identical consecutive molecules): first molecule, count, atoms, first atom
    int nspec;
    int sp_m0[kMaxSpecies], sp_cnt[kMaxSpecies], sp_na[kMaxSpecies], sp_a0[kMaxSpecies];
    Slot sp_atom[kMaxSpecies][kMaxA];
    double sp_mass[kMaxSpecies][kMaxA];
    // two windows of the random stream
    long long wbase[2];
    int wn[2];
    int wnext;
};

// why a chain stops before its last move (ChainShared::abort)
constexpr int kAbortStream = 1;     // the random stream ran out (YAMC_ERNG_EXHAUSTED, resumable)
constexpr int kAbortNonFinite = 2;  // a non-finite energy change or bias force (YAMC_ENAN)

__device__ __forceinline__ void worker_sync(int nwork) {
    asm volatile("bar.sync 1, %0;" ::"r"(nwork) : "memory");
}

template <int I>
struct IntC { static constexpr int value = I; };

// calls f(IntC<I>) for I in [B, E): loop indices known at compile time
template <int B, int E, class F>
__device__ __forceinline__ void static_for(F &&f) {
    if constexpr (B < E) {
        f(IntC<B>{});
        static_for<B + 1, E>(f);
    }
}

template <int NT>
struct NPair { static constexpr int value = NT * (NT + 1) / 2; };

// row of the packed upper triangle t1 <= t2 (the host's pair_index enumeration)
template <int NT>
__host__ __device__ constexpr int pair_idx(int a, int b) {
    return a <= b ? a * NT - a * (a - 1) / 2 + (b - a) : b * NT - b * (b - 1) / 2 + (a - b);
}

// Arithmetic of a pass: MX = false is the plain FP64 method; MX = true the mixed form (pair
// terms, erfc_Luc, phases and per-thread sums in FP32; rho(k), the cross-warp and cross-CTA
// sums, the energy bookkeeping and the Metropolis test in FP64).
template <bool MX> struct Prec { using R = double; using R2 = double2; };
template <> struct Prec<true> { using R = float; using R2 = float2; };

__device__ __forceinline__ double2 mk2(double x, double y) { return make_double2(x, y); }
__device__ __forceinline__ float2 mk2(float x, float y) { return make_float2(x, y); }
template <class R2> __device__ __forceinline__ R2 cvt2(double2 v);
template <> __device__ __forceinline__ double2 cvt2<double2>(double2 v) { return v; }
template <> __device__ __forceinline__ float2 cvt2<float2>(double2 v) { return make_float2((float)v.x, (float)v.y); }
template <class R2> __device__ __forceinline__ R2 cvt2(float2 v);  // (FP32 rho copies: the mixed form only)
template <> __device__ __forceinline__ float2 cvt2<float2>(float2 v) { return v; }
// a product rounded on its own (never fused into a following sum)
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
// a or b as values (a conditional over array elements selects their addresses, which would keep
// the array in local memory)
template <class T> __device__ __forceinline__ T pick(bool c, T a, T b) { return c ? a : b; }
__device__ __forceinline__ double2 to_d2(double2 v) { return v; }
__device__ __forceinline__ double2 to_d2(float2 v) { return make_double2((double)v.x, (double)v.y); }

// Buffer i of a chain's scratch (0: the moved molecule's old phase sums, 1: the rho deltas of the
// pass), in the pass's arithmetic type: FP64 pairs in the plain form, FP32 pairs in the mixed
// form (half the bytes, and loads that need no conversion).
template <bool MX>
__host__ __device__ __forceinline__ typename Prec<MX>::R2 *scratch_buf(double2 *base, int i, int nstruct, int S) {
    return reinterpret_cast<typename Prec<MX>::R2 *>(base) + (size_t)i * nstruct * S;
}

// Per-thread partial sums of a pass: FP64; in the mixed form FP64 for the pair terms (which
// reach tens of kT) and FP32 with two-sum compensation (the running sum and its rounding
// error, added in FP64 when the warp reduces) for the FP32 k-space terms.
template <bool MX, int N = kNV>
struct Acc {
    double v[N];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = 0.0;
    }
    __device__ __forceinline__ void add(int i, double x) { v[i] += x; }
    __device__ __forceinline__ void add_plain(int i, double x) { v[i] += x; }
    __device__ __forceinline__ void flag(int i) { v[i] = 1.0; }
    __device__ __forceinline__ double get(int i) const { return v[i]; }
    __device__ __forceinline__ double kpart(int i) const { return v[i]; }
};
template <int N>
struct Acc<true, N> {
    double d[N];
    float s[N], c[N];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < N; ++i) { d[i] = 0.0; s[i] = 0.f; c[i] = 0.f; }
    }
    __device__ __forceinline__ void add(int i, double x) { d[i] += x; }
    __device__ __forceinline__ void add(int i, float x) {  // TwoSum (Knuth)
        const float t = s[i] + x;
        const float bp = t - s[i];
        c[i] += (s[i] - (t - bp)) + (x - bp);
        s[i] = t;
    }
    // plain FP32 sum, for the k-space forces: they only bias the proposal (their error is
    // reported beside the dE error), and a few entries per thread keep it near FP32 rounding
    __device__ __forceinline__ void add_plain(int i, float x) { s[i] += x; }
    __device__ __forceinline__ void flag(int i) { d[i] = 1.0; }
    __device__ __forceinline__ double get(int i) const { return d[i] + ((double)s[i] + (double)c[i]); }
    // the FP32 part alone (the k-space sums are reduced before the real space)
    __device__ __forceinline__ double kpart(int i) const { return (double)s[i] + (double)c[i]; }
};

template <int NT, int EPT, bool MX = false>
struct EntryRegs {
    using R = typename Prec<MX>::R;
    using R2 = typename Prec<MX>::R2;
    int e[EPT];
    int kx[EPT], ky[EPT], kz[EPT];
    R beta[EPT];
    R bl[EPT][NPair<NT>::value];  // beta_LJ of every type pair for this entry
    double2 rho[EPT][1 + NT];     // FP64 in both forms
    R2 mold[EPT][1 + NT];
    R2 dl[EPT][1 + NT];
};

// EPT <= 0: the streamed layout (EPT == -1: the same with wide CTAs) -- no entry lives in
// registers; each worker loops over its entries and reads k, beta, beta_LJ and rho from memory
// (L2-resident) every pass.  The register block of one (never touched) entry only keeps the
// code uniform.
template <int NT, int EPT, bool MX = false>
using RegsOf = EntryRegs<NT, (EPT > 0 ? EPT : 1), MX>;

// The per-move phase tables of the molecule's slots, T[axis][m][slot] = (cos, sin)(2 pi m u): an
// entry's thread forms one address per axis and reaches every slot at a fixed offset from it.  A
// row holds kTabRow slots, one more than the molecule's at most 2 kMaxA, so the rows of consecutive
// m fall into different banks (9 x 8 B or 9 x 16 B apart) for the lanes of a warp, which take
// consecutive kz.
constexpr int kTabRow = 2 * kMaxA + 1;
template <bool MX>
struct PhaseTabs {
    const typename Prec<MX>::R2 *T;
    int KM;
};

// Phase tables of slots [s0, s1) of move m, by the workers.  The FP32 form reduces 2 k u
// modulo 2 in FP64 before the FP32 sincospi.
template <bool MX>
__device__ __forceinline__ void build_tables(typename Prec<MX>::R2 *tab, const Slot *slots, int s0, int s1, int KM,
                                             int wtid, int nwork) {
    using R = typename Prec<MX>::R;
    const int n = (s1 - s0) * 3 * KM;
    for (int idx = wtid; idx < n; idx += nwork) {
        const int sl = s0 + idx / (3 * KM), r = idx % (3 * KM), d = r / KM, k = r % KM;
        const double u = d == 0 ? slots[sl].x : (d == 1 ? slots[sl].y : slots[sl].z);
        R s, c;
        if constexpr (MX) {
            double t = 2.0 * (double)k * u;
            t = t - 2.0 * rint(0.5 * t);
            sincospif((float)t, &s, &c);
        } else {
            sincospi(2.0 * (double)k * u, &s, &c);
        }
        if (k == 0) { s = R(0); c = R(1); }
        tab[(d * KM + k) * kTabRow + sl] = mk2(c, s);
    }
}

// What the k-space sweep reads of the moving molecule, in registers: read from the slots once per
// pass.  (Read per entry they cost a shared load, an FP64 compare and an FP64-to-FP32 conversion
// per atom and entry: the sweep's stores keep the compiler from hoisting them.)
// `simple`: three charged atoms with LJ on the first only (rigid 3-site water): the sweep then
// holds one LJ row per entry instead of one per LJ type, and runs without branches on the atoms.
template <bool MX>
struct MolK {
    using R = typename Prec<MX>::R;
    R q[kMaxA], iq[kMaxA];
    int type[kMaxA];  // LJ type (0 = none)
    int na, cmask;    // atoms; bit a: atom a is charged
    int tmask;        // bit t: the molecule carries LJ type t + 1
    bool simple;
    __device__ __forceinline__ explicit MolK(const Slot *slots, int n) : na(n), cmask(0), tmask(0) {
#pragma unroll
        for (int a = 0; a < kMaxA; ++a) {
            q[a] = R(0); iq[a] = R(0); type[a] = 0;
            if (a < n) {
                q[a] = (R)slots[a].q; iq[a] = (R)slots[a].iq; type[a] = slots[a].type;
                if (slots[a].q != 0.0) cmask |= 1 << a;
                if (type[a] > 0) tmask |= 1 << (type[a] - 1);
            }
        }
        simple = n == 3 && cmask == 7 && type[0] > 0 && type[1] == 0 && type[2] == 0;
    }
};

// q (cos, sin)(2 pi (x kx + y ky + z kz)) of one slot (entry_phase's arithmetic) from the slot's
// elements X, Y, Z of the entry's three table rows
template <class R, class R2>
__device__ __forceinline__ void slot_phase(R2 X, R2 Y, R2 Z, bool yneg, bool zneg, R q, R &c, R &s) {
    const R cx = X.x, sx = X.y, cy = Y.x, sy = yneg ? -Y.y : Y.y, cz = Z.x, sz = zneg ? -Z.y : Z.y;
    const R qcc = q * cx * cy, qss = q * sx * sy, qsc = q * sx * cy, qcs = q * cx * sy;
    const R qc = qcc - qss, qs = qsc + qcs;
    const R c1 = qc * cz, s1 = qs * sz, s2 = qs * cz, c2 = qc * sz;
    c = c1 - s1;
    s = s2 + c2;
}

// one entry's three table rows and signs
template <bool MX>
struct EntryRows {
    const typename Prec<MX>::R2 *tx, *ty, *tz;
    bool yneg, zneg;
    __device__ __forceinline__ EntryRows(const PhaseTabs<MX> &pt, int kx, int ky, int kz)
        : tx(pt.T + kx * kTabRow), ty(pt.T + (pt.KM + (ky < 0 ? -ky : ky)) * kTabRow),
          tz(pt.T + (2 * pt.KM + (kz < 0 ? -kz : kz)) * kTabRow), yneg(ky < 0), zneg(kz < 0) {}
};

// Molecule phase sums of one entry over slots [s0, s0+na) -- RhoSquared_addAtom per atom:
// Coulomb phase q (cos, sin), LJ phase = Coulomb phase * (1/q) (the unit phase when q == 0),
// accumulated per LJ type in atom order.  ph/phl keep the per-atom phases for the forces.
template <int NT, bool MX>
__device__ __forceinline__ void mol_phase_sum(const EntryRows<MX> &er, const MolK<MX> &mk, int s0,
                                              typename Prec<MX>::R2 (&out)[1 + NT],
                                              typename Prec<MX>::R2 (&ph)[kMaxA], typename Prec<MX>::R2 (&phl)[kMaxA]) {
    using R = typename Prec<MX>::R;
    using R2 = typename Prec<MX>::R2;
#pragma unroll
    for (int t = 0; t <= NT; ++t) out[t] = mk2(R(0), R(0));
#pragma unroll
    for (int a = 0; a < kMaxA; ++a) {
        ph[a] = mk2(R(0), R(0));
        phl[a] = mk2(R(0), R(0));
        if (a < mk.na) {
            const R2 X = er.tx[s0 + a], Y = er.ty[s0 + a], Z = er.tz[s0 + a];
            const bool charged = (mk.cmask >> a) & 1;
            R c = 0, s = 0;
            if (charged) {
                slot_phase<R, R2>(X, Y, Z, er.yneg, er.zneg, mk.q[a], c, s);
                out[0].x = out[0].x + c; out[0].y = out[0].y + s;
            }
            ph[a] = mk2(c, s);
            if (mk.type[a] > 0) {
                R cl, sl;
                if (charged) { cl = c * mk.iq[a]; sl = s * mk.iq[a]; }
                else slot_phase<R, R2>(X, Y, Z, er.yneg, er.zneg, R(1), cl, sl);
#pragma unroll
                for (int t = 0; t < NT; ++t) {  // (selects of values: an indexed or conditional store would put out in local memory)
                    const bool hit = t == mk.type[a] - 1;
                    out[1 + t].x = pick<R>(hit, out[1 + t].x + cl, out[1 + t].x);
                    out[1 + t].y = pick<R>(hit, out[1 + t].y + sl, out[1 + t].y);
                }
                phl[a] = mk2(cl, sl);
            }
        }
    }
}

// element (t0, t) of an entry's beta_LJ row set, t0 known at run time (selects of values)
template <int NT, class R>
__device__ __forceinline__ R beta_lj_of(const R (&bl)[NPair<NT>::value], int t0, int t) {
    R b = bl[pair_idx<NT>(0, t)];
#pragma unroll
    for (int u = 1; u < NT; ++u) {
        b = pick<R>(t0 == u, bl[pair_idx<NT>(u, t)], b);
    }
    return b;
}

// k-space force on one atom from one entry: 4 pi beta (C sin - S cos) k, Coulomb with the
// q-weighted phase (ForceKSpace.f90:59-302); w also holds the dispersion terms where there are any
template <class R, class AccT>
__device__ __forceinline__ void add_force(int a, R w, int kx, int ky, int kz, AccT &acc) {
    acc.add_plain(RV_F + 3 * a, w * (R)kx);
    acc.add_plain(RV_F + 3 * a + 1, w * (R)ky);
    acc.add_plain(RV_F + 3 * a + 2, w * (R)kz);
}

// k-space force on the molecule's atoms from one entry, plus the dispersion terms of the atom's
// LJ type against every type's structure factor.
template <int NT, bool MX, class AccT>
__device__ __forceinline__ void entry_forces(const MolK<MX> &mk, int kx, int ky, int kz,
                                             typename Prec<MX>::R beta,
                                             const typename Prec<MX>::R (&bl)[NPair<NT>::value],
                                             const typename Prec<MX>::R2 (&C)[1 + NT],
                                             const typename Prec<MX>::R2 (&ph)[kMaxA],
                                             const typename Prec<MX>::R2 (&phl)[kMaxA], AccT &acc) {
    using R = typename Prec<MX>::R;
    const R fourpi = (R)kFourPi;
#pragma unroll
    for (int a = 0; a < kMaxA; ++a) {
        if (a < mk.na) {
            R w = mul_rn(fourpi, (C[0].x * ph[a].y - C[0].y * ph[a].x) * beta);
            if (mk.type[a] > 0) {
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const R b = beta_lj_of<NT, R>(bl, mk.type[a] - 1, t);
                    w += fourpi * ((C[1 + t].x * phl[a].y - C[1 + t].y * phl[a].x) * b);
                }
            }
            add_force(a, w, kx, ky, kz, acc);
        }
    }
}

// One signed entry of a pass: the molecule's phase sums at the old positions (into mold) and/or
// the new ones, the delta (into dl), dU_k Coulomb + LJ against rho, and the k-space forces.
template <int NT, int KIND, bool FORCES, bool MX, class AccT, class RhoT>
__device__ __forceinline__ void kspace_entry(const PhaseTabs<MX> &pt, const MolK<MX> &mk, int kx,
                                             int ky, int kz, typename Prec<MX>::R beta,
                                             const typename Prec<MX>::R (&bl)[NPair<NT>::value],
                                             const RhoT (&rho)[1 + NT], typename Prec<MX>::R2 (&mold)[1 + NT],
                                             typename Prec<MX>::R2 (&dl)[1 + NT], AccT &acc) {
    using R = typename Prec<MX>::R;
    using R2 = typename Prec<MX>::R2;
    const EntryRows<MX> er(pt, kx, ky, kz);
    R2 ph[kMaxA], phl[kMaxA];
    R2 C[1 + NT];
#pragma unroll
    for (int t = 0; t <= NT; ++t) C[t] = cvt2<R2>(rho[t]);
    if constexpr (KIND != PASS_NEW) mol_phase_sum<NT, MX>(er, mk, mk.na, mold, ph, phl);
    if constexpr (KIND == PASS_OLD) {
        if constexpr (FORCES) entry_forces<NT, MX>(mk, kx, ky, kz, beta, bl, C, ph, phl, acc);
    } else {
        R2 mnew[1 + NT];
        mol_phase_sum<NT, MX>(er, mk, 0, mnew, ph, phl);
#pragma unroll
        for (int t = 0; t <= NT; ++t) dl[t] = mk2(mnew[t].x - mold[t].x, mnew[t].y - mold[t].y);
        {   // EwaldSumKSpace_calc_dU_coulomb (EwaldSumKSpace.f90:528-620)
            const R2 Cc = C[0], d = dl[0];
            acc.add(RV_DUC, (((Cc.x + Cc.x) + d.x) * d.x + ((Cc.y + Cc.y) + d.y) * d.y) * beta);
        }
        // EwaldSumKSpace_calc_dU_LJ (EwaldSumKSpace.f90:623-753): t1 over all types, t2 over the
        // molecule's types (a type absent from the molecule has a zero delta and adds nothing)
        // (the entry's terms summed in order first, then added to the compensated running sum)
        R dul = R(0);
#pragma unroll
        for (int t1 = 0; t1 < NT; ++t1) {
            const R2 C1 = C[1 + t1], D1 = dl[1 + t1];
            const R tc = (C1.x + C1.x) + D1.x, ts = (C1.y + C1.y) + D1.y;
#pragma unroll
            for (int t2 = 0; t2 < NT; ++t2) {
                const R2 D2 = dl[1 + t2];
                const R u = dul + (tc * D2.x + ts * D2.y) * bl[pair_idx<NT>(t1, t2)];
                dul = pick<R>((mk.tmask >> t2) & 1, u, dul);
            }
        }
        acc.add(RV_DUL, dul);
        if constexpr (KIND == PASS_NEW && FORCES) {  // against total_new = rho + delta (MC.f90:1136-1163)
            R2 Cn[1 + NT];
#pragma unroll
            for (int t = 0; t <= NT; ++t) Cn[t] = mk2(C[t].x + dl[t].x, C[t].y + dl[t].y);
            entry_forces<NT, MX>(mk, kx, ky, kz, beta, bl, Cn, ph, phl, acc);
        }
    }
}

// The same entry for a `simple` molecule (MolK): the same terms in the same order, with the one LJ
// row (type t0 + 1) that its delta has; mold / dl: row 0 Coulomb, row 1 that LJ row; b[t]: beta_LJ
// of the pair (t0, t).
template <int NT, int KIND, bool FORCES, bool MX, class AccT, class RhoT>
__device__ __forceinline__ void kspace_entry_simple(const PhaseTabs<MX> &pt, const MolK<MX> &mk, int kx, int ky, int kz,
                                                    typename Prec<MX>::R beta, const typename Prec<MX>::R (&b)[NT],
                                                    const RhoT (&rho)[1 + NT], typename Prec<MX>::R2 &mold0,
                                                    typename Prec<MX>::R2 &mold1, typename Prec<MX>::R2 &dl0,
                                                    typename Prec<MX>::R2 &dl1, AccT &acc) {
    using R = typename Prec<MX>::R;
    using R2 = typename Prec<MX>::R2;
    constexpr int NA = 3;
    const EntryRows<MX> er(pt, kx, ky, kz);
    const int t0 = mk.type[0] - 1;
    const R fourpi = (R)kFourPi;
    R2 C[1 + NT];
#pragma unroll
    for (int t = 0; t <= NT; ++t) C[t] = cvt2<R2>(rho[t]);
    R2 ph[NA], phl;
    auto phases = [&](int s0, R2 &sum0, R2 &sum1) {
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            R c, s;
            slot_phase<R, R2>(er.tx[s0 + a], er.ty[s0 + a], er.tz[s0 + a], er.yneg, er.zneg, mk.q[a], c, s);
            sum0 = a == 0 ? mk2(c, s) : mk2(sum0.x + c, sum0.y + s);
            ph[a] = mk2(c, s);
        }
        phl = mk2(mul_rn(ph[0].x, mk.iq[0]), mul_rn(ph[0].y, mk.iq[0]));
        sum1 = phl;
    };
    auto forces = [&](const R2 (&F)[1 + NT]) {
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            R w = mul_rn(fourpi, (F[0].x * ph[a].y - F[0].y * ph[a].x) * beta);
            if (a == 0) {
#pragma unroll
                for (int t = 0; t < NT; ++t) w += fourpi * ((F[1 + t].x * phl.y - F[1 + t].y * phl.x) * b[t]);
            }
            add_force(a, w, kx, ky, kz, acc);
        }
    };
    if constexpr (KIND != PASS_NEW) phases(NA, mold0, mold1);
    if constexpr (KIND == PASS_OLD) {
        if constexpr (FORCES) forces(C);
    } else {
        R2 n0, n1;
        phases(0, n0, n1);
        dl0 = mk2(n0.x - mold0.x, n0.y - mold0.y);
        dl1 = mk2(n1.x - mold1.x, n1.y - mold1.y);
        acc.add(RV_DUC, (((C[0].x + C[0].x) + dl0.x) * dl0.x + ((C[0].y + C[0].y) + dl0.y) * dl0.y) * beta);
        R dul = R(0);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const R dx = t == t0 ? dl1.x : R(0), dy = t == t0 ? dl1.y : R(0);
            const R tc = (C[1 + t].x + C[1 + t].x) + dx, ts = (C[1 + t].y + C[1 + t].y) + dy;
            dul += (tc * dl1.x + ts * dl1.y) * b[t];
        }
        acc.add(RV_DUL, dul);
        if constexpr (KIND == PASS_NEW && FORCES) {
            R2 Cn[1 + NT];
            Cn[0] = mk2(C[0].x + dl0.x, C[0].y + dl0.y);
#pragma unroll
            for (int t = 0; t < NT; ++t)
                Cn[1 + t] = mk2(C[1 + t].x + (t == t0 ? dl1.x : R(0)), C[1 + t].y + (t == t0 ? dl1.y : R(0)));
            forces(Cn);
        }
    }
}

// The k-space sweep of one pass over the worker's entries.  Registers layout: k, beta, beta_LJ and
// rho stay in registers (R), the old phase sums are R.mold and the delta R.dl; all EPT entries run
// without a branch between them, so their dependency chains interleave (an entry past the last has
// k = 0 and zero beta, beta_LJ and rho: it adds exact zeros).  Streamed layout: every entry is read
// from memory (L2-resident), the next entry's loads in flight while the current one computes; the
// old sums go to the chain's scratch in PASS_OLD and come from there in PASS_NEW, the delta goes to
// the scratch.  SIMPLE: only rows 0 and 1 + t0 of mold and dl exist (in registers: rows 0 and 1).
template <int NT, int EPT, int KIND, bool FORCES, bool MX, bool SIMPLE, class AccT>
__device__ __forceinline__ void kspace_sweep(const DevSys &D, RegsOf<NT, EPT, MX> &R, const PhaseTabs<MX> &pt,
                                             const MolK<MX> &mk, int e0, int estep, typename Prec<MX>::R2 *mold_g,
                                             AccT &acc) {
    using Rt = typename Prec<MX>::R;
    using R2 = typename Prec<MX>::R2;
    const int S = D.S;
    const int t0 = SIMPLE ? mk.type[0] - 1 : 0;
    if constexpr (EPT > 0) {
        static_for<0, EPT>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            if constexpr (SIMPLE) {
                Rt b[NT];
#pragma unroll
                for (int t = 0; t < NT; ++t) b[t] = beta_lj_of<NT, Rt>(R.bl[k], t0, t);
                kspace_entry_simple<NT, KIND, FORCES, MX>(pt, mk, R.kx[k], R.ky[k], R.kz[k], R.beta[k], b, R.rho[k],
                                                          R.mold[k][0], R.mold[k][1], R.dl[k][0], R.dl[k][1], acc);
            } else {
                kspace_entry<NT, KIND, FORCES, MX>(pt, mk, R.kx[k], R.ky[k], R.kz[k], R.beta[k], R.bl[k],
                                                   R.rho[k], R.mold[k], R.dl[k], acc);
            }
        });
    } else {
        constexpr bool IN_MOLD = KIND == PASS_NEW;   // read the old sums
        constexpr int NB = SIMPLE ? NT : NPair<NT>::value;  // beta_LJ rows read per entry
        constexpr int NR = SIMPLE ? 2 : 1 + NT;             // rows of mold and dl
        R2 *dl_g = scratch_buf<MX>(D.scratch, 1, 1 + NT, S);
        // the mixed form reads FP32 rho (D.rho_f, equal to rho rounded to FP32, which is what its
        // arithmetic takes), FP32 beta tables and FP32 scratch; k comes packed in one word
        using RhoT = std::conditional_t<MX, float2, double2>;
        auto row = [&](int r) { return (SIMPLE && r == 1) ? 1 + t0 : r; };
        auto brow = [&](int p) { return SIMPLE ? pair_idx<NT>(t0, p) : p; };
        int kv_n;
        Rt beta_n, bl_n[NB];
        RhoT rho_n[1 + NT];
        R2 mold_n[NR];
        // the loads of the next entry stay in flight until the entry is taken up: no value is
        // converted here
        auto fetch = [&](int e) {
            kv_n = D.kpack[YAMC_IX(e, S)];
            if constexpr (MX) {
                beta_n = D.ebeta_f[e];
#pragma unroll
                for (int p = 0; p < NB; ++p) bl_n[p] = D.ebetalj_f[(size_t)brow(p) * S + e];
            } else {
                beta_n = D.ebeta[e];
#pragma unroll
                for (int p = 0; p < NB; ++p) bl_n[p] = D.ebetalj[(size_t)brow(p) * S + e];
            }
#pragma unroll
            for (int t = 0; t <= NT; ++t) {
                if constexpr (MX) rho_n[t] = D.rho_f[(size_t)t * S + e];
                else rho_n[t] = D.rho[(size_t)t * S + e];
            }
            if constexpr (IN_MOLD) {
#pragma unroll
                for (int r = 0; r < NR; ++r) mold_n[r] = mold_g[(size_t)row(r) * S + e];
            }
        };
        if (e0 < S) fetch(e0);
        for (int e = e0; e < S; e += estep) {
            const int kx = kv_n & 255, ky = ((kv_n >> 8) & 255) - 128, kz = (kv_n >> 16) - 128;
            const Rt beta = beta_n;
            Rt bl[NB];
            RhoT rho[1 + NT];
            R2 mold[NR], dl[NR];
#pragma unroll
            for (int p = 0; p < NB; ++p) bl[p] = bl_n[p];
#pragma unroll
            for (int t = 0; t <= NT; ++t) rho[t] = rho_n[t];
#pragma unroll
            for (int r = 0; r < NR; ++r) mold[r] = IN_MOLD ? mold_n[r] : mk2(Rt(0), Rt(0));
            if (e + estep < S) fetch(e + estep);
            if constexpr (SIMPLE)
                kspace_entry_simple<NT, KIND, FORCES, MX>(pt, mk, kx, ky, kz, beta, bl, rho, mold[0], mold[1], dl[0],
                                                          dl[1], acc);
            else
                kspace_entry<NT, KIND, FORCES, MX>(pt, mk, kx, ky, kz, beta, bl, rho, mold, dl, acc);
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                if (KIND == PASS_OLD) mold_g[(size_t)row(r) * S + e] = mold[r];
                else dl_g[(size_t)row(r) * S + e] = dl[r];
            }
        }
    }
}

// Sums N <= 16 values over the warp: a tree that halves the values each lane holds at every step
// (15 exchanges for 16 values and one more, against 80 for a butterfly per value; the same pairs
// are added in the same order, so the sums are the butterfly's bit for bit).  Value i ends in lane
// 2 i (and 2 i + 1); returns the lane's value.
template <int N>
__device__ __forceinline__ double warp_sums(const double (&v)[N]) {
    static_assert(N <= 16, "at most 16 values");
    const int lane = threadIdx.x & 31;
    double a[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) a[i] = i < N ? v[i < N ? i : 0] : 0.0;
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        const bool up = lane & (2 * h);
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double keep = pick<double>(up, a[i + h], a[i]), give = pick<double>(up, a[i], a[i + h]);
            a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
        }
    }
    return a[0] + __shfl_xor_sync(0xffffffffu, a[0], 1);
}

// The k-space part of a pass: the sweep over the worker's entries, then its sums (dU_k and, with
// FORCES, the k-space forces) over the warp into the warp's row of red -- all values of the row
// that the pass uses, so the real-space part adds to it.
constexpr int kKV = 2 + 3 * kMaxA;  // k-space values: dU_k Coulomb, dU_k LJ, forces
template <int NT, int EPT, int KIND, bool FORCES, bool MX, bool SIMPLE>
__device__ __forceinline__ void kspace_part(const DevSys &D, RegsOf<NT, EPT, MX> &R, const PhaseTabs<MX> &pt,
                                            const MolK<MX> &mk, int e0, int estep, typename Prec<MX>::R2 *mold_g,
                                            double *row) {
    Acc<MX> acc;
    acc.zero();
    kspace_sweep<NT, EPT, KIND, FORCES, MX, SIMPLE>(D, R, pt, mk, e0, estep, mold_g, acc);
    double v[FORCES ? kKV : 2];
#pragma unroll
    for (int i = 0; i < (FORCES ? kKV : 2); ++i) v[i] = acc.kpart(i < 2 ? RV_DUC + i : RV_F + i - 2);
    const double x = warp_sums(v);
    const int lane = threadIdx.x & 31, i = lane >> 1;
    if (!(lane & 1) && i < (FORCES ? kKV : 2)) row[i < 2 ? RV_DUC + i : RV_F + i - 2] = x;
}
template <int NT, int EPT, int KIND, bool FORCES, bool MX, bool SIMPLE>
__device__ __noinline__ void kspace_part_call(const DevSys &D, RegsOf<NT, EPT, MX> &R, const PhaseTabs<MX> &pt,
                                              const Slot *slots, int na, int e0, int estep,
                                              typename Prec<MX>::R2 *mold_g, double *row) {
    kspace_part<NT, EPT, KIND, FORCES, MX, SIMPLE>(D, R, pt, MolK<MX>(slots, na), e0, estep, mold_g, row);
}

// Real space of one pass, by the worker warps: the moving molecule's pairs with the CTA's staged atoms,
// and the reduction into red[worker warp][value].  FORCES: the old positions (is_new false) or the new
// ones with their forces; otherwise both positions at once, signed.
#define YAMC_WPH(ph) do { if (pf) { const long long t_now = clock64(); prof[ph] += t_now - t_mark; t_mark = t_now; } } while (0)
template <bool FORCES, bool MX>
__device__ __forceinline__ void real_part(const DevSys &D, ChainShared &sh, bool is_new, long long *prof) {
    const Cand &m = sh.cand[sh.icur];
    const StageView &V = sh.view;
    const double4 *atom_s = V.atom;
    const int2 *meta_s = V.meta;
    const float4 *box_s = V.box;
    const double *lj_s = V.lj;
    const int na = m.na, nt = D.nt, nown = V.nown, imol0 = m.imol - 1;
    const int wtid = threadIdx.x - kCtl, lane = threadIdx.x & 31;
    const int wwarp = wtid >> 5, nww = (blockDim.x - kCtl) >> 5;
    const int s_lo = FORCES && !is_new ? na : 0, s_hi = FORCES && is_new ? na : 2 * na;  // active slots [s_lo, s_hi)
    const bool hard = !FORCES || is_new;  // hard cores are tested at the new positions
    const int nv = FORCES ? (RV_F + 3 * na) : RV_F;
    double *red = V.red;
    int *wbuf = V.wbuf;
    const bool pf = prof && wtid == 0;
    long long t_mark = pf ? clock64() : 0;
    Acc<MX> acc;
    acc.zero();

    // Real space, warp by warp: the staged blocks are dealt to the warps in turn (neighbours in space
    // go to different warps); a warp gathers the atoms of its near blocks inside the query sphere, four
    // blocks at a time, tests them 32 at a time against the molecule's slots (cutoff, hard core), and
    // evaluates the pairs that pass 64 at a time from its own queue: no barrier between the warps,
    // full warps in every step, and in each step independent work (with two warps per scheduler it is
    // latency that bounds it), in an order that the positions alone decide.
    {
        unsigned short *nb = reinterpret_cast<unsigned short *>(wbuf + wwarp * kWarpBuf);  // near atoms
        unsigned short *queue = nb + kNear, *blocks = queue + kPairs;                      // pairs (slot << 13 | atom); near blocks
        const unsigned lt = (1u << lane) - 1u;
        // the query sphere: an atom farther than the pair filter's reach plus the molecule's radius from
        // its centre (slot 0 new, slot na old) is outside the cutoff and every hard core of all slots
        // (triangle inequality on the periodic box).  A pass over both positions takes one sphere
        // around the midpoint of the two centres that holds both (the centre may have been wrapped: the
        // shift is taken by minimum image).  Radii in FP32, rounded up.
        double qx, qy, qz, qr2;
        {
            double rad2 = 0.0;
            for (int a = 1; a < na; ++a) {
                const double dx = m.slot[a].x - m.slot[0].x, dy = m.slot[a].y - m.slot[0].y, dz = m.slot[a].z - m.slot[0].z;
                const double ex = m.slot[na + a].x - m.slot[na].x, ey = m.slot[na + a].y - m.slot[na].y,
                             ez = m.slot[na + a].z - m.slot[na].z;
                rad2 = fmax(rad2, fmax(dx * dx + dy * dy + dz * dz, ex * ex + ey * ey + ez * ez));
            }
            double r = D.rpre + (double)__fsqrt_ru(__double2float_ru(rad2));
            const Slot &c = m.slot[is_new ? 0 : na];
            qx = c.x; qy = c.y; qz = c.z;
            if constexpr (!FORCES) {
                const double hx = 0.5 * min_image(m.slot[0].x - qx), hy = 0.5 * min_image(m.slot[0].y - qy),
                             hz = 0.5 * min_image(m.slot[0].z - qz);
                qx += hx; qy += hy; qz += hz;
                r += (double)__fsqrt_ru(__double2float_ru(hx * hx + hy * hy + hz * hz));
            }
            r *= 1.0 + 1e-9;
            qr2 = r * r;
        }
        // this warp's blocks whose bounding box comes within the query sphere.  A block outside it
        // holds no atom that the per-atom test below keeps.
        const int nblk = (nown + kBlk - 1) / kBlk;
        int nnear = 0, npair = 0, nmine = 0;
        bool ovl = false;
        for (int b0 = wwarp; b0 < nblk; b0 += 32 * nww) {
            const int b = b0 + nww * lane;
            const bool near = b < nblk && box_near(box_s, b, qx, qy, qz, qr2);
            const unsigned bal = __ballot_sync(0xffffffffu, near);
            if (near) blocks[YAMC_IX(nmine + __popc(bal & lt), kBlkList)] = (unsigned short)b;
            nmine += __popc(bal);
        }
        __syncwarp();
        // (one loop with one copy of each step: the code of a move runs once per move, so its size is
        // instruction fetches, not only cache)
        for (int i0 = 0;;) {
            if (i0 < nmine) {
                // near atoms of four blocks
                int jl[4];
                bool near[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    jl[u] = i0 + u < nmine ? blocks[YAMC_IX(i0 + u, kBlkList)] * kBlk + lane : nown;
                    const int j = jl[u] < nown ? jl[u] : 0;
                    const double4 pj = atom_s[YAMC_IX(j, nown)];
                    const double dx = min_image(qx - pj.x), dy = min_image(qy - pj.y), dz = min_image(qz - pj.z);
                    near[u] = jl[u] < nown && meta_s[YAMC_IX(j, nown)].x != imol0 && dx * dx + dy * dy + dz * dz < qr2;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const unsigned bal = __ballot_sync(0xffffffffu, near[u]);
                    if (near[u]) nb[YAMC_IX(nnear + __popc(bal & lt), kNear)] = (unsigned short)jl[u];
                    nnear += __popc(bal);
                }
                i0 += 4;
            }
            const bool last = i0 >= nmine;
            if (!last && nnear <= kNear - 4 * kBlk) continue;
            __syncwarp();
            if (last) YAMC_WPH(PH_FILTER);
            int k0 = 0;
            do {
                // slot tests of 32 gathered atoms
                const bool valid = k0 + lane < nnear;
                const int jl = valid ? nb[YAMC_IX(k0 + lane, kNear)] : 0;
                const double4 pj = atom_s[YAMC_IX(jl, nown)];
                const int tj = meta_s[YAMC_IX(jl, nown)].y;
                // hard-core diameter: by LJ type when every atom of a type has the same one (a
                // shared-memory table), else the atom's own (global memory, by the atom in slot jl)
                const double dj = !hard        ? 0.0
                                  : D.dhs_typed ? V.dhs_ts[tj]
                                                : D.dhs[D.atom_of[YAMC_IX(jl * V.gsize + V.grank, D.N + 16)]];
                unsigned in = 0;  // slots inside the cutoff
#pragma unroll 3
                for (int s = s_lo; s < s_hi; ++s) {
                    const Slot &sl = m.slot[s];
                    const double dx = min_image(sl.x - pj.x), dy = min_image(sl.y - pj.y), dz = min_image(sl.z - pj.z);
                    const double r2 = dx * dx + dy * dy + dz * dz;
                    if (hard && s < na && sl.type > 0 && tj > 0) {  // hard core (EwaldSumRealSpace.f90:409)
                        const double d12 = (sl.dhs + dj) / 2;
                        if (valid && r2 < d12 * d12) ovl = true;
                    }
                    if (valid && r2 < D.rmax2) in |= 1u << s;
                }
                // the pairs slot by slot, an atom each lane
                for (int s = s_lo; s < s_hi; ++s) {
                    const unsigned bal = __ballot_sync(0xffffffffu, in >> s & 1);
                    if (in >> s & 1) queue[YAMC_IX(npair + __popc(bal & lt), kPairs)] = (unsigned short)(s << 13 | jl);
                    npair += __popc(bal);
                }
                __syncwarp();
                k0 += 32;
                // whole groups of 64 pairs (at the end all) are evaluated, two per lane side by side; the
                // rest moves to the queue's front
                const int n = last && k0 >= nnear ? npair : npair & ~63;
                for (int q0 = lane; q0 < n; q0 += 64) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int q = q0 + 32 * u;
                        const int item = queue[YAMC_IX(q < n ? q : q0, kPairs)];
                        const int ji = item & 8191, s = item >> 13;
                        const Slot &sl = m.slot[s];
                        const double4 pi = atom_s[YAMC_IX(ji, nown)];
                        const int ti = meta_s[YAMC_IX(ji, nown)].y;
                        const double dx = min_image(sl.x - pi.x), dy = min_image(sl.y - pi.y), dz = min_image(sl.z - pi.z);
                        const double r2 = dx * dx + dy * dy + dz * dz;
                        const bool lj = sl.type > 0 && ti > 0;
                        const int off = lj ? (sl.type - 1) * nt + (ti - 1) : 0;
                        const double qq = D.xclb * sl.q * pi.w;
                        const double s6 = lj ? lj_s[off] : 0.0, fe = lj ? lj_s[nt * nt + off] : 0.0;
                        const bool isnew = s < na;
                        const double sign = (!FORCES && !isnew) ? -1.0 : 1.0;
                        const PairTerm<double> t = MX ? pair_term_mx<FORCES>(r2, qq, lj, s6, fe, D.alpha, D.taosp, false)
                                                      : pair_term<double, FORCES>(r2, qq, lj, s6, fe, D.alpha, D.taosp, false);
                        if (q < n) {
                            acc.add(RV_EW, sign * t.ew); acc.add(RV_LJ6, sign * t.lj6); acc.add(RV_LJ12, sign * t.lj12);
                            if constexpr (FORCES) {
                                const int a = isnew ? s : s - na;
#pragma unroll
                                for (int aa = 0; aa < kMaxA; ++aa)
                                    if (aa == a) {
                                        acc.add(RV_F + 3 * aa, dx * t.FR);
                                        acc.add(RV_F + 3 * aa + 1, dy * t.FR);
                                        acc.add(RV_F + 3 * aa + 2, dz * t.FR);
                                    }
                            }
                        }
                    }
                }
                if (n > 0) {
                    __syncwarp();
                    const unsigned short r0 = n + lane < npair ? queue[YAMC_IX(n + lane, kPairs)] : 0,
                                         r1 = n + 32 + lane < npair ? queue[YAMC_IX(n + 32 + lane, kPairs)] : 0;
                    __syncwarp();
                    queue[lane] = r0; queue[32 + lane] = r1;
                    npair -= n;
                    __syncwarp();
                }
            } while (k0 < nnear);
            nnear = 0;
            if (last) break;
        }
        if (ovl) acc.flag(RV_OVL);
        YAMC_WPH(PH_PAIRS);
    }

    // the real-space sums over the warp, added to the k-space sums in the warp's row
    {
        constexpr int NR = FORCES ? 3 + 3 * kMaxA : 3;
        double v[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) v[i] = acc.get(i < 3 ? RV_EW + i : RV_F + i - 3);
        const double x = warp_sums(v);
        const bool ovl = __any_sync(0xffffffffu, acc.get(RV_OVL) > 0.0);
        const int i = lane >> 1, at = i < 3 ? RV_EW + i : RV_F + i - 3;
        double *row = red + wwarp * kNV;
        if (!(lane & 1) && i < NR && at < nv) row[at] = i < 3 ? x : row[at] + x;
        if (lane == 31) {
            row[RV_OVL] = ovl ? 1.0 : 0.0;
            if (!hard) row[RV_DUC] = row[RV_DUL] = 0.0;
        }
    }
}

// One copy for the two passes of a biased move, out of line: the second finds its instructions where
// the first fetched them.  (WIDE: the copy of the wide CTAs, which have fewer registers a thread.)
template <bool MX, bool WIDE>
__device__ __noinline__ void real_part_forces(const DevSys &D, ChainShared &sh, bool is_new, long long *prof) {
    real_part<true, MX>(D, sh, is_new, prof);
}

// The workers' part of one pass over the molecule's slots: the phase tables, k space over the worker's
// entries, real space over the CTA's atoms (PASS_OLD and PASS_NEW with forces, PASS_BOTH without).
// One worker barrier (bar 1), after the tables.
template <int NT, int EPT, int KIND, bool MX>
__device__ __forceinline__ void worker_pass(const DevSys &D, ChainShared &sh, RegsOf<NT, EPT, MX> &R, double2 *tab_raw, int e0,
                                            int estep, long long *prof, typename Prec<MX>::R2 *mold_buf) {
    constexpr bool FORCES = KIND != PASS_BOTH;
    const Cand &m = sh.cand[sh.icur];
    const int na = m.na;
    const int KM = D.kmax + 1;
    const int nwork = blockDim.x - kCtl;
    const int wtid = threadIdx.x - kCtl;
    const int s_lo = (KIND == PASS_OLD) ? na : 0;  // active slots [s_lo, s_hi)
    const int s_hi = (KIND == PASS_NEW) ? na : 2 * na;
    using R2 = typename Prec<MX>::R2;
    R2 *tab = reinterpret_cast<R2 *>(tab_raw);
    const bool pf = prof && wtid == 0;
    long long t_mark = pf ? clock64() : 0;

    build_tables<MX>(tab, m.slot, s_lo, s_hi, KM, wtid, nwork);
    worker_sync(nwork);
    YAMC_WPH(PH_TABLES);
    const PhaseTabs<MX> pt{tab, KM};

    // k space, out of line when the entries are streamed: each sweep then has the register budget to
    // itself (entries in registers must stay there across the passes)
    {
        const MolK<MX> mk(m.slot, na);
        double *row = sh.view.red + (wtid >> 5) * kNV;
        if constexpr (EPT > 0) {
            if (mk.simple) kspace_part<NT, EPT, KIND, FORCES, MX, true>(D, R, pt, mk, e0, estep, mold_buf, row);
            else kspace_part<NT, EPT, KIND, FORCES, MX, false>(D, R, pt, mk, e0, estep, mold_buf, row);
        } else {
            if (mk.simple) kspace_part_call<NT, EPT, KIND, FORCES, MX, true>(D, R, pt, m.slot, na, e0, estep, mold_buf, row);
            else kspace_part_call<NT, EPT, KIND, FORCES, MX, false>(D, R, pt, m.slot, na, e0, estep, mold_buf, row);
        }
    }
    YAMC_WPH(PH_KSPACE);
    if constexpr (FORCES) real_part_forces<MX, (EPT < 0)>(D, sh, KIND == PASS_NEW, prof);
    else real_part<false, MX>(D, sh, false, prof);
}
#undef YAMC_WPH

// Control warp, after the workers' per-warp partials: trees over the worker warps, then over the
// cluster's CTAs in a fixed order, so every CTA holds bit-identical totals in sh.tot.  Called by
// all threads (the cluster barrier needs everyone).  Lane v of the control warp owns value v (a lane
// writes its value to every CTA's exchange row, so there is no index arithmetic per value and CTA).
static_assert(kNV <= 32, "a lane per value");
__device__ __forceinline__ void reduce_pass(ChainShared &sh, const double *red, double *xch, int nv, int G, int rank,
                                            int xpar, cg::cluster_group &cluster) {
    // the worker warps' partials in warp order, then (cluster) every CTA's sum in rank order --
    // the same order in every CTA
    const int v = threadIdx.x;
    const int nww = (blockDim.x - kCtl) >> 5;
    const bool own = v < nv, flag = v == RV_OVL;
    if (own) {
        double x = 0.0;
#pragma unroll 4
        for (int w = 0; w < nww; ++w) {
            const double y = red[w * kNV + v];
            x = flag ? fmax(x, y) : x + y;
        }
        if (G > 1) {
            const int at = (xpar * G + rank) * kNV + v;
#pragma unroll 4
            for (int r = 0; r < G; ++r) cluster.map_shared_rank(xch, r)[at] = x;
        } else {
            sh.tot[v] = x;
        }
    }
    if (G > 1) {
        cluster.sync();
        if (own) {
            double x = 0.0;
#pragma unroll 4
            for (int r = 0; r < G; ++r) {
                const double y = xch[(xpar * G + r) * kNV + v];
                x = flag ? fmax(x, y) : x + y;
            }
            sh.tot[v] = x;
        }
    }
}

// Control lane work: molecule choice (run_mc draws) and the static atom data of the chosen
// molecule at its current positions.  `moving` is the molecule of the move in flight (0-based,
// -1 if none) whose positions come from `moving_pos` (its old or its proposed positions).
struct ChooseCtx {
    const DevSys *D;
    const RunSlot *run;
    const float *w0, *w1;
    const double4 *atom_s;
    int G;
};

__device__ inline RngReader make_reader(const ChooseCtx &X, const ChainShared &sh, long long cur) {
    // the window that holds cur (the newer one where both do): the draws of a move fit in it, and
    // one that passes its end reads the stream itself
    const int b = sh.wnext ^ 1;
    const unsigned long long k = (unsigned long long)(cur - sh.wbase[b]), k2 = (unsigned long long)(cur - sh.wbase[b ^ 1]);
    const bool in = sh.wbase[b] >= 0 && k < (unsigned long long)sh.wn[b];
    const bool in2 = !in && sh.wbase[b ^ 1] >= 0 && k2 < (unsigned long long)sh.wn[b ^ 1];
    const int s = in ? b : b ^ 1;
    const bool any = in || in2;
    return RngReader{X.run->rng, X.run->rng_off, X.run->n_rng, s ? X.w1 : X.w0, any ? sh.wbase[s] : cur, any ? sh.wn[s] : 0,
                     any ? (int)(in ? k : k2) : 0, 0};
}

__device__ inline void stage_molecule(const ChooseCtx &X, ChainShared &sh, Cand &C, int imol, int moving,
                                      const Slot *moving_pos, cg::cluster_group &cluster) {
    const DevSys &D = *X.D;
    int sp = -1;
    for (int q = 0; q < sh.nspec; ++q)
        if (imol - 1 >= sh.sp_m0[q] && imol - 1 < sh.sp_m0[q] + sh.sp_cnt[q]) { sp = q; break; }
    int first, nam;
    if (sp >= 0) { nam = sh.sp_na[sp]; first = sh.sp_a0[sp] + (imol - 1 - sh.sp_m0[sp]) * nam; }
    else { const int2 mr = D.mol[YAMC_IX(imol - 1, D.M)]; first = mr.x; nam = mr.y; }
    C.imol = imol; C.first = first; C.na = nam;
    double mx = 0, my = 0, mz = 0;
    int slots[kMaxA];  // staging slots of the molecule's atoms (loaded together), then their positions
    double4 pos[kMaxA];
#pragma unroll
    for (int a = 0; a < kMaxA; ++a) slots[a] = a < nam ? ld_table(D.slot + YAMC_IX(first + a, D.N)) : 0;
    const bool staged = imol - 1 != moving && imol - 1 != sh.last_mol;
#pragma unroll
    for (int a = 0; a < kMaxA; ++a)
        if (staged && a < nam) {
            const double4 *src = (X.G > 1) ? cluster.map_shared_rank(X.atom_s, (first + a) % X.G) : X.atom_s;
            pos[a] = src[slots[a]];
        }
#pragma unroll
    for (int a = 0; a < kMaxA; ++a) {
        if (a >= nam) break;
        const int j = first + a;
        Slot s;
        if (sp >= 0) { s = sh.sp_atom[sp][a]; C.mass[a] = sh.sp_mass[sp][a]; }
        else {
            const int jc = (int)YAMC_IX(j, D.N);
            const double q = D.atom[jc].w;
            s.q = q; s.iq = q != 0.0 ? 1.0 / q : 0.0; s.dhs = D.dhs[jc]; s.type = D.meta[jc].y;
            C.mass[a] = D.mass[jc];
        }
        s.pad = slots[a];  // the commit updates the staged copy in this slot of CTA j % G
        if (imol - 1 == moving) { s.x = moving_pos[a].x; s.y = moving_pos[a].y; s.z = moving_pos[a].z; }
        else if (imol - 1 == sh.last_mol) { s.x = sh.lx[a]; s.y = sh.ly[a]; s.z = sh.lz[a]; }
        else { s.x = pos[a].x; s.y = pos[a].y; s.z = pos[a].z; }
        C.slot[nam + a] = s;  // old positions
        C.slot[a] = s;        // proposed positions, replaced by propose()
        // dipole of the molecule at the old positions (EwaldSumExternal_calc_mu)
        mx = mx + s.q * s.x; my = my + s.q * s.y; mz = mz + s.q * s.z;
    }
    C.mu_old[0] = mx; C.mu_old[1] = my; C.mu_old[2] = mz;
}

// run_mc's draws before movemc: the per-cycle pressure draw, the exchange draw, the molecule
// draw (runmc.f90:206, 232, 258).  Returns the 1-based molecule, or 0 when the stream ran out or
// the draws make this step an exchange step or the cycle a volume cycle (the chain then stops
// before it, like at the end of the stream, and the host runs it).
__device__ inline int draw_molecule(const DevSys &D, RngReader &rng, bool cycle_start) {
    const double pd = cycle_start ? rng.next() : 0.0;
    const double xd = rng.next();
    const double r = rng.next();
    if (rng.out || xd < D.xprob) return 0;
    if (cycle_start && D.psm > 0 && pd * (D.psm + 1) > D.psm) return 0;  // a volume cycle: the host runs it
    return choose_molecule_guess(r, D.freq_beg, D.freq_end, D.M, D.freq_monotone);
}

// movemc Step 5 (MC.f90:1031-1067) of an unbiased move for a staged molecule
__device__ inline void propose(const DevSys &D, Cand &C, RngReader &rng) {
    const int na = C.na;
    MoveState &m = C.mv;
    mcm_choose_unbiased(m, rng, D.dr, D.d_angle);
    if (rng.out) return;
    // old positions from slots [na, 2 na), new ones into [0, na): no overlap
    const Slot *os = C.slot + na;
    Slot *ns = C.slot;
    place_molecule_f(m, na, [&](int i, int d) { return d == 0 ? os[i].x : (d == 1 ? os[i].y : os[i].z); }, C.mass,
                     [&](int i, double x, double y, double z) { ns[i].x = x; ns[i].y = y; ns[i].z = z; });
}

// The mixed form's FP64 recomputation of rho(k) (RhoSquared_addAtoms, RhoSquared.f90:188-243)
// inside the chain, by all threads of every CTA of the cluster: the worker threads recompute the
// entries they own from every atom's FP64 position (D.atom, kept current by rank 0), with the
// atoms' per-axis phase tables built in chunks in the scratch region; then the k-space energies
// (EwaldSumKSpace_calc_coulomb_energy / _calc_LJ_energy, EwaldSumKSpace.f90:389-526) are
// reduced over the cluster into the engine scalars.
// (the entries of the register layout come back through D.rho: taking the address of the
// register-held rows would keep them in local memory for the whole launch)
template <int NT, int EPT>
__device__ __noinline__ void refresh_in_chain(const DevSys &D, double2 *scr, int scr_atoms, int e0, int estep,
                                              int G, int rank, ChainShared &sh, double *red, double *xch, int xpar,
                                              cg::cluster_group &cluster) {
    const int tid = threadIdx.x, B = blockDim.x;
    const bool ctl = tid < kCtl;
    const int lane = tid & 31, wwarp = (tid - kCtl) >> 5;
    const int KM = D.kmax + 1, S = D.S, N = D.N;
    const int CH = scr_atoms < 64 ? scr_atoms : 64;
    double2 *tabs = scr;                                                  // [CH][3][KM]
    double *sq = reinterpret_cast<double *>(tabs + (size_t)CH * 3 * KM);  // [CH]
    int *st = reinterpret_cast<int *>(sq + CH);                           // [CH]
    // the positions rank 0 wrote for accepted moves are visible to every CTA after this barrier
    __threadfence();
    if (G > 1) cluster.sync(); else __syncthreads();
    constexpr int EB = EPT > 0 ? EPT : 4;  // entries per batch
    const int nbatch = EPT > 0 ? 1 : (S + estep * EB - 1) / (estep * EB);
    double ekc = 0.0, ekl = 0.0;
    for (int b = 0; b < nbatch; ++b) {
        int ent[EB];
        int4 kv[EB];
        double2 acc[EB][1 + NT];
#pragma unroll
        for (int j = 0; j < EB; ++j) {
            const int e = e0 + (b * EB + j) * estep;
            ent[j] = (!ctl && e >= 0 && e < S) ? e : -1;
            kv[j] = ent[j] >= 0 ? D.kvec[ent[j]] : make_int4(0, 0, 0, 0);
#pragma unroll
            for (int t = 0; t <= NT; ++t) acc[j][t] = make_double2(0.0, 0.0);
        }
        // the entries of the batch that the warp has: its first lane's (a lane's one past its last has
        // k = 0, and its sums go nowhere)
        int nent = 0;
#pragma unroll
        for (int j = 0; j < EB; ++j) nent += ent[j] >= 0;
        nent = __shfl_sync(0xffffffffu, nent, 0);
        for (int a0 = 0; a0 < N; a0 += CH) {
            const int na = min(CH, N - a0);
            for (int idx = tid; idx < na * 3 * KM; idx += B) {
                const int a = idx / (3 * KM), r = idx % (3 * KM), d = r / KM, m = r % KM;
                const double4 p = D.atom[a0 + a];
                const double u = d == 0 ? p.x : (d == 1 ? p.y : p.z);
                double sn, cs;
                sincospi(2.0 * (double)m * u, &sn, &cs);
                if (m == 0) { sn = 0.0; cs = 1.0; }
                tabs[(a * 3 + d) * KM + m] = make_double2(cs, sn);
            }
            for (int a = tid; a < na; a += B) { sq[a] = D.atom[a0 + a].w; st[a] = D.meta[a0 + a].y; }
            __syncthreads();
            if (!ctl) {
                // Two entries side by side, with no branch between them or before their phases: latency binds
                // (7 or 11 worker warps a CTA).  A branch per entry and atom took 10.3 ms a refresh of 12,440
                // atoms on 16 CTAs and 137 ms of 49,752, this 7.8 and 100; four side by side 5.6 and 77, but
                // their registers cost every move of the streamed mixed form up to 8 %.
                auto sum = [&](auto jc, auto nc) {
                    constexpr int j0 = decltype(jc)::value, n = decltype(nc)::value;
#pragma unroll 1
                    for (int a = 0; a < na; ++a) {
                        const double2 *T = tabs + (size_t)a * 3 * KM;
                        const double q = sq[a], w = q != 0.0 ? q : 1.0;
                        const int ty = st[a];
                        double c[n], s[n];
#pragma unroll
                        for (int j = 0; j < n; ++j)
                            entry_phase<double, double2>(T, T + KM, T + 2 * KM, kv[j0 + j].x, kv[j0 + j].y, kv[j0 + j].z, w,
                                                         c[j], s[j]);
                        if (q != 0.0) {
#pragma unroll
                            for (int j = 0; j < n; ++j) {
                                double2 &A = acc[j0 + j][0];
                                A.x = A.x + c[j]; A.y = A.y + s[j];
                            }
                        }
                        if (ty > 0) {
                            const double iw = 1.0 / w;
#pragma unroll
                            for (int t = 0; t < NT; ++t)
                                if (t == ty - 1) {
#pragma unroll
                                    for (int j = 0; j < n; ++j) {
                                        double2 &A = acc[j0 + j][1 + t];
                                        A.x = A.x + c[j] * iw; A.y = A.y + s[j] * iw;
                                    }
                                }
                        }
                    }
                };
                static_for<0, (EB + 1) / 2>([&](auto hc) {
                    constexpr int j0 = 2 * decltype(hc)::value;
                    if (nent == j0 + 1) sum(IntC<j0>{}, IntC<1>{});
                    if constexpr (j0 + 1 < EB)
                        if (nent > j0 + 1) sum(IntC<j0>{}, IntC<2>{});
                });
            }
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < EB; ++j) {
            const int e = ent[j];
            if (e < 0) continue;
#pragma unroll
            for (int t = 0; t <= NT; ++t) {
                D.rho[(size_t)t * S + e] = acc[j][t];
                if constexpr (EPT <= 0) {
                    D.rho_f[(size_t)t * S + e] = make_float2((float)acc[j][t].x, (float)acc[j][t].y);
                }
            }
            ekc += D.ebeta[e] * (acc[j][0].x * acc[j][0].x + acc[j][0].y * acc[j][0].y);
#pragma unroll
            for (int t1 = 0; t1 < NT; ++t1)
#pragma unroll
                for (int t2 = t1; t2 < NT; ++t2) {
                    double l = D.ebetalj[(size_t)pair_idx<NT>(t1, t2) * S + e] *
                               (acc[j][1 + t1].x * acc[j][1 + t2].x + acc[j][1 + t1].y * acc[j][1 + t2].y);
                    if (t1 != t2) l = l + l;
                    ekl += l;
                }
        }
    }
    // k-space energies over the cluster (the pass reduction with two values)
    if (!ctl) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ekc += __shfl_xor_sync(0xffffffffu, ekc, o);
            ekl += __shfl_xor_sync(0xffffffffu, ekl, o);
        }
        if (lane == 0)
            for (int v = 0; v <= RV_DUL; ++v) red[wwarp * kNV + v] = v == RV_DUC ? ekc : (v == RV_DUL ? ekl : 0.0);
    }
    __syncthreads();
    reduce_pass(sh, red, xch, RV_DUL + 1, G, rank, xpar, cluster);
    __syncthreads();
    if (tid == 0) { sh.sc[SC_EK_C] = sh.tot[RV_DUC]; sh.sc[SC_EK_LJ] = sh.tot[RV_DUL]; }
    __syncthreads();
}

// The static shared memory of k_chain: its __shared__ variables, each on its own 16 bytes.  (As members of
// one object, whose size would say it without this list, they cost the FP64 streamed variant 5 % of its
// time in spills: nacl1m on 3 x 256 threads 21.5 -> 22.5 us a move.)
constexpr size_t pad16(size_t bytes) { return (bytes + 15) / 16 * 16; }
constexpr size_t kChainStaticBytes = pad16(sizeof(ChainShared)) + pad16(sizeof(float) * 2 * kWin) + pad16(sizeof(DevSys)) +
                                     pad16(sizeof(long long) * PH_COUNT);

// SPLIT = false: unbiased device-resident chain only (one fused pass per move, speculation);
// SPLIT = true: force-biased moves (old pass + new pass with forces).
template <int NT, int EPT, bool SPLIT, bool MX>
__global__ void __launch_bounds__(EPT < 0 ? kChainMaxThreadsWide : kChainMaxThreads, 1) k_chain(ChainArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ChainShared sh;
    __shared__ float rwin[2][kWin];

    cg::cluster_group cluster = cg::this_cluster();
    const int G = A.G;
    const int rank = G > 1 ? (int)cluster.block_rank() : 0;
    const int rep = blockIdx.x / G;
    // the system's parameters and array pointers in shared memory: every thread reads them from
    // there (a per-thread copy would live in local memory, which the staged atoms leave little L1 for)
    __shared__ DevSys D_s;
    {
        const int *src = reinterpret_cast<const int *>(A.sys + rep);
        int *dst = reinterpret_cast<int *>(&D_s);
        for (int i = threadIdx.x; i < (int)(sizeof(DevSys) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
        __syncthreads();
    }
    const DevSys &D = D_s;
    RunSlot *run = A.run + rep;
    const int B = blockDim.x;
    const int tid = threadIdx.x;
    const int KM = D.kmax + 1;
    const int S = D.S;
    const int nt = D.nt;
    const int nwork = B - kCtl;
    const int wtid = tid - kCtl;
    const bool ctl = tid < kCtl;
    const int lane = tid & 31;

    // shared memory carve-up (chain_smem_bytes on the host computes the same sizes)
    const int nblk_max = (A.nown_max + kBlk - 1) / kBlk;
    double2 *tab = reinterpret_cast<double2 *>(smem_raw);                     // [3][KM][kTabRow]
    float4 *box_s = reinterpret_cast<float4 *>(tab + kTabRow * 3 * KM);       // [nblk_max][2]
    double4 *atom_s = reinterpret_cast<double4 *>(box_s + 2 * nblk_max);      // [nown_max]
    int2 *meta_s = reinterpret_cast<int2 *>(atom_s + A.nown_max);             // [nown_max]
    int *wbuf = reinterpret_cast<int *>(meta_s + A.nown_max);                 // [wbuf_ints]: the warps' near atoms and pairs
    double *red = reinterpret_cast<double *>(wbuf + wbuf_ints(B, D.kmax));    // [B/32][kNV]
    // the mixed form's rho refresh reuses the warps' buffers as atom phase tables
    double2 *scr = reinterpret_cast<double2 *>((reinterpret_cast<uintptr_t>(wbuf) + 15) & ~uintptr_t(15));
    const int scr_atoms = (int)(((reinterpret_cast<char *>(red) - reinterpret_cast<char *>(scr))) /
                                (long)(sizeof(double2) * 3 * KM + sizeof(double) + sizeof(int)));
    double *xch = red + (B / 32) * kNV;                                       // [2][G][kNV]
    double *lj_s = xch + 2 * G * kNV;                                         // [2][nt*nt]
    double *dhs_ts = lj_s + 2 * nt * nt;                                      // [nt+1] hard core by LJ type

    // atoms of this CTA: j = rank + G * i (interleaved, so every CTA holds a spatial mix), in
    // the spatial order of k_stage_order (slot D.slot[j]), with the bounding box of every kBlk slots
    const int nown = (D.N - rank + G - 1) / G;
    for (int i = tid; i < nown; i += B) {
        const int j = rank + G * i, sl = (int)YAMC_IX(D.slot[j], A.nown_max);
        atom_s[sl] = D.atom[j]; meta_s[sl] = D.meta[j];
    }
    __syncthreads();
    for (int b = tid; b < (nown + kBlk - 1) / kBlk; b += B) block_box(atom_s, b, nown, box_s);
    for (int i = tid; i < nt * nt; i += B) { lj_s[i] = D.lj_sig6[i]; lj_s[nt * nt + i] = D.lj_feps[i]; }
    for (int i = tid; i <= nt; i += B) dhs_ts[i] = D.dhs_t[i];

    // the workers' k-vector entries; rho stays in registers for the whole launch
    using Rt = typename Prec<MX>::R;
    using R2 = typename Prec<MX>::R2;
    RegsOf<NT, EPT, MX> R;
    const int gwork = G * nwork;
    const int e0 = rank * nwork + wtid;  // this worker's entries: e0 + k * gwork
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
        const int e = ctl ? S : rank * nwork + wtid + k * gwork;
        R.e[k] = e < S ? e : -1;
        R.kx[k] = R.ky[k] = R.kz[k] = 0;
        R.beta[k] = 0;
        if (e < S) {
            const int4 kv = D.kvec[e];
            R.kx[k] = kv.x; R.ky[k] = kv.y; R.kz[k] = kv.z;
            R.beta[k] = (Rt)D.ebeta[e];
        }
#pragma unroll
        for (int p = 0; p < NPair<NT>::value; ++p) R.bl[k][p] = e < S ? (Rt)D.ebetalj[(size_t)p * S + e] : Rt(0);
#pragma unroll
        for (int t = 0; t <= NT; ++t) {
            R.rho[k][t] = e < S ? D.rho[(size_t)t * S + e] : make_double2(0, 0);
            R.mold[k][t] = mk2(Rt(0), Rt(0));
            R.dl[k][t] = mk2(Rt(0), Rt(0));
        }
    }
    const long long n_rng = run->n_rng;
    if (tid == 0) {
        for (int c = 0; c < SC_COUNT; ++c) sh.sc[c] = D.scal[c];
        sh.icycle = D.cnt[CN_ICYCLE];
        sh.mic = D.cnt[CN_MOVE_IN_CYCLE];
        sh.cursor = run->cursor;
        sh.last_mol = -1;
        sh.view = StageView{atom_s, meta_s, box_s, dhs_ts, lj_s, red, wbuf, nown, rank, G};
        sh.abort = 0;
        sh.wnext = 0;
        sh.icur = 0;
        sh.spec_ok = 0;
        // static atom data of each molecule species, taken from its first molecule
        sh.nspec = D.nspec <= kMaxSpecies ? D.nspec : 0;
        for (int sp = 0; sp < sh.nspec; ++sp) {
            const int4 c = D.spec[sp];
            sh.sp_m0[sp] = c.x; sh.sp_cnt[sp] = c.y; sh.sp_na[sp] = c.z; sh.sp_a0[sp] = c.w;
            for (int a = 0; a < c.z; ++a) {
                const int j = c.w + a;
                Slot t;
                t.x = t.y = t.z = 0.0;
                t.q = D.atom[j].w; t.iq = t.q != 0.0 ? 1.0 / t.q : 0.0;
                t.dhs = D.dhs[j]; t.type = D.meta[j].y; t.pad = 0;
                sh.sp_atom[sp][a] = t;
                sh.sp_mass[sp][a] = D.mass[j];
            }
        }
    }
    // first random window at the start cursor
    if (ctl) {
        const long long base = run->cursor;
        const long long avail = n_rng - base;
        const int nw = (int)(avail < (long long)kWin ? (avail > 0 ? avail : 0) : kWin);
        for (int i = lane; i < nw; i += 32) rwin[0][i] = run->rng[YAMC_IX(base + i - run->rng_off, n_rng - run->rng_off)];
        if (lane == 0) { sh.wbase[0] = base; sh.wn[0] = nw; sh.wbase[1] = -1; sh.wn[1] = 0; sh.wnext = 1; }
    }
    __syncthreads();
    constexpr bool biased = SPLIT;  // (the SPLIT variant runs exactly the systems with a force bias)
    // the next move is prepared while the workers run the current pass: chosen and proposed for
    // unbiased moves, only chosen for force-biased ones (their proposal needs the old forces)
    constexpr bool choose_only = biased;
    const ChooseCtx X{&D, run, rwin[0], rwin[1], atom_s, G};

    long long moves_done = 0;
    int n_acc = 0, rows = 0;
    // mixed form: accepted moves since the last FP64 recomputation of rho(k), known to every thread
    long long acc_since = D.cnt[CN_ACC_SINCE_REFRESH], refreshes = 0;
    const long long refresh_every = MX ? D.refresh_every : 0;
    int xpar = 0;  // parity of the cluster exchange buffer, flipped after every pass
    const long long n_moves = run->n_moves;
    // phase cycles are counted in shared memory (a counter in global memory costs a round trip per mark)
    __shared__ long long prof_s[PH_COUNT];
    long long *prof = (A.prof && rank == 0) ? prof_s : nullptr;
    if (prof && tid < PH_COUNT) prof_s[tid] = 0;
    if (prof) __syncthreads();
    const bool pc = prof && tid == 0;
    long long t_mark = 0;
#define YAMC_PH(ph) do { if (pc) { const long long t_now = clock64(); prof[ph] += t_now - t_mark; t_mark = t_now; } } while (0)

    // ---------------------------------------------------------------- the first move of the launch
    bool have_next = false;  // sh.cur already prepared by the previous iteration's speculation
    for (long long it = 0; it < n_moves; ++it) {
        if (pc) t_mark = clock64();
        R2 *mold_g = scratch_buf<MX>(D.scratch, 0, 1 + NT, S);  // the moved molecule's old phase sums
        if (!have_next) {
            __syncthreads();  // every thread has read what the last decision left in sh
            // choose the molecule and stage its atoms (no move in flight)
            if (tid == 0) {
                Cand &C = sh.cand[sh.icur];
                C.cur_start = sh.cursor;
                RngReader rng = make_reader(X, sh, sh.cursor);
                int imol = draw_molecule(D, rng, sh.mic == 0);
                C.valid = imol > 0;
                C.cur_prop = rng.cur();
                if (!imol) imol = 1;
                stage_molecule(X, sh, C, imol, -1, nullptr, cluster);
                sh.abort = C.valid ? 0 : kAbortStream;
            }
            __syncthreads();
            if (sh.abort) break;
            YAMC_PH(PH_CHOOSE);
        }
        if (!have_next || choose_only) {
            const int na0 = sh.cand[sh.icur].na;
            // old forces for force-biased moves (movemc Steps 3-4)
            if constexpr (biased) {
                if (!ctl) worker_pass<NT, EPT, PASS_OLD, MX>(D, sh, R, tab, e0, gwork, prof, mold_g);
                __syncthreads();
                reduce_pass(sh, red, xch, RV_F + 3 * na0, G, rank, xpar, cluster);
                xpar ^= 1;
                __syncthreads();
                YAMC_PH(PH_OLD_PASS);  // the force-biased old pass and its reduction (the control warp's view)
            }
            // the proposal (movemc Step 5)
            if constexpr (biased) {
                // on two warps: warp 0 draws the displacement (its Newton iteration is the long serial
                // part) while warp 1 skips the displacement's draws and draws the rotation; all lanes of
                // a warp run the same code on the same data, which lets them share the sum of the
                // rotation's bias term (shi_sans_exp_warp)
                if (tid < 64) {
                    const Cand &C = sh.cand[sh.icur];
                    double F[3], T[3];
                    const Slot *os = C.slot + na0;
                    // the old forces with the external field -2 kext q mu (MC.f90:988-997)
                    mol_force_torque_f(na0, [&](int i, int d) { return d == 0 ? os[i].x : (d == 1 ? os[i].y : os[i].z); },
                                       C.mass, [&](int i, int d) { return sh.tot[RV_F + 3 * i + d] + D.m2k * os[i].q * sh.sc[SC_MU_X + d]; },
                                       F, T);
                    RngReader rng = make_reader(X, sh, C.cur_prop);
                    MoveState m;
                    mcm_init_old(m, F, T);
                    if (tid < 32) {
                        mcm_choose_displacement(m, rng, D.xlf, D.dr);
                        if (lane == 0) {
                            sh.eold[0] = sh.tot[RV_EW]; sh.eold[1] = sh.tot[RV_LJ6]; sh.eold[2] = sh.tot[RV_LJ12];
                            MoveState &d = sh.cand[sh.icur].mv;
                            d.fxo = m.fxo; d.fyo = m.fyo; d.fzo = m.fzo; d.cxo = m.cxo; d.cyo = m.cyo; d.czo = m.czo; d.co = m.co;
                            d.umaxold = m.umaxold; d.cold = m.cold; d.deltx = m.deltx; d.delty = m.delty; d.deltz = m.deltz;
                            sh.disp_end = rng.cur();
                            sh.disp_out = rng.out;
                        }
                    } else {
                        mcm_skip_displacement(m, rng, D.xlf, D.dr);
                        const long long start = rng.cur();
                        if (!rng.out) mcm_choose_rotation(m, rng, D.xlc, D.d_angle, shi_sans_exp_warp, PickWarp());
                        if (lane == 0) {
                            copy_rotation(sh.mrot, m);
                            sh.rot_start = start;
                            sh.rot_end = rng.cur();
                            sh.rot_out = rng.out;
                        }
                    }
                }
                __syncthreads();
                if (ctl) {
                    Cand &C = sh.cand[sh.icur];
                    MoveState &m = C.mv;
                    bool out = sh.disp_out != 0;
                    long long cur = sh.disp_end;
                    if (!out) {
                        if (sh.rot_start == sh.disp_end) {
                            if (lane == 0) copy_rotation(m, sh.mrot);
                            cur = sh.rot_end;
                            out = sh.rot_out != 0;
                        } else {  // (the skip always draws what the displacement draws; kept as a guard)
                            RngReader rng = make_reader(X, sh, sh.disp_end);
                            MoveState r;
                            r.cxo = m.cxo; r.cyo = m.cyo; r.czo = m.czo; r.co = m.co;
                            mcm_choose_rotation(r, rng, D.xlc, D.d_angle, shi_sans_exp_warp, PickWarp());
                            if (lane == 0) copy_rotation(m, r);
                            cur = rng.cur();
                            out = rng.out != 0;
                        }
                        __syncwarp();
                    }
                    if (lane == 0) {
                        sh.prop_out = out;
                        if (out) {
                            C.valid = 0;
                        } else {
                            // old positions from slots [na0, 2 na0), new ones into [0, na0): no overlap
                            const Slot *os = C.slot + na0;
                            Slot *ns = C.slot;
                            place_molecule_f(m, na0, [&](int i, int d) { return d == 0 ? os[i].x : (d == 1 ? os[i].y : os[i].z); },
                                             C.mass, [&](int i, double x, double y, double z) { ns[i].x = x; ns[i].y = y; ns[i].z = z; });
                            C.cur_prop = cur;
                        }
                    }
                }
            } else if (tid == 0) {
                Cand &C = sh.cand[sh.icur];
                RngReader rng = make_reader(X, sh, C.cur_prop);
                propose(D, C, rng);
                C.cur_prop = rng.cur();
                // (not into sh.abort: a warp that has yet to read it after the choice above would
                // leave the loop alone, and the others wait for it at the next barrier)
                sh.prop_out = rng.out;
                if (rng.out) C.valid = 0;
            }
            __syncthreads();
            if (sh.prop_out) {
                if (tid == 0) sh.abort = kAbortStream;
                break;
            }
            YAMC_PH(PH_PROPOSE);
        }
        const int na = sh.cand[sh.icur].na;
        const bool split = SPLIT;

        // ------------------------------------------------ the pass over the new positions
        if (!ctl) {
            if constexpr (SPLIT) worker_pass<NT, EPT, PASS_NEW, MX>(D, sh, R, tab, e0, gwork, prof, mold_g);
            else worker_pass<NT, EPT, PASS_BOTH, MX>(D, sh, R, tab, e0, gwork, prof, mold_g);
        } else if (it + 1 < n_moves) {
            // prepare the next move's candidates while the workers run: lanes 1-2 after the
            // acceptance draw, lane 2 with the molecule in flight at its proposed positions (used
            // only if it is chosen again and accepted)
            const Cand &M = sh.cand[sh.icur];
            const long long c1 = M.cur_prop;
            const bool next_cycle = (sh.mic + 1 == D.M);
            // the window of the stream the candidates read: make sure it covers c1 onwards
            {
                const int b = sh.wnext;
                const bool covered0 = sh.wbase[0] >= 0 && c1 >= sh.wbase[0] && c1 + kWin / 2 <= sh.wbase[0] + sh.wn[0];
                const bool covered1 = sh.wbase[1] >= 0 && c1 >= sh.wbase[1] && c1 + kWin / 2 <= sh.wbase[1] + sh.wn[1];
                if (!covered0 && !covered1) {
                    const long long avail = n_rng - c1;
                    const int nw = (int)(avail < (long long)kWin ? (avail > 0 ? avail : 0) : kWin);
                    __syncwarp();
                    for (int i = lane; i < nw; i += 32) rwin[b][i] = run->rng[YAMC_IX(c1 + i - run->rng_off, n_rng - run->rng_off)];
                    __syncwarp();
                    if (lane == 0) { sh.wbase[b] = c1; sh.wn[b] = nw; sh.wnext = b ^ 1; }
                    __syncwarp();
                }
            }
            if (lane == 0) {
                // the candidate after an overlap is not prepared: overlaps are rare, and a third
                // lane on its own random numbers diverges from lanes 1-2 (which draw the same
                // numbers and run in step); an overlap takes the unspeculated path instead
                sh.spec[0] = (sh.icur + 1) & 3; sh.spec[1] = (sh.icur + 2) & 3; sh.spec[2] = (sh.icur + 3) & 3;
                sh.cand[(sh.icur + 1) & 3].valid = 0;
            } else if (lane < 3) {
                const int buf = (sh.icur + 1 + lane) & 3;
                Cand &C = sh.cand[buf];
                RngReader rng = make_reader(X, sh, c1);
                (void)rng.next();  // the acceptance draw (MonteCarloMove.f90:553)
                C.cur_start = rng.cur();
                const int imol = rng.out ? 0 : draw_molecule(D, rng, next_cycle);
                C.valid = imol > 0;
                const Slot *moving = (lane == 2) ? &M.slot[0] : &M.slot[M.na];
                stage_molecule(X, sh, C, imol > 0 ? imol : 1, M.imol - 1, moving, cluster);
                if constexpr (!SPLIT) if (C.valid) propose(D, C, rng);
                C.cur_prop = rng.cur();
                if (rng.out) C.valid = 0;
            }
            if (pc) { const long long t_now = clock64(); prof[PH_SPECULATE] += t_now - t_mark; t_mark = t_now; }
        }
        __syncthreads();
        reduce_pass(sh, red, xch, split ? RV_F + 3 * na : RV_F, G, rank, xpar, cluster);
        xpar ^= 1;
        YAMC_PH(PH_REDUCE);

        // ------------------------------------------------ Metropolis (Steps 7-13) and commit (Step 14)
        // The control warp decides (all lanes on the same data); what the next move waits for is written
        // before the barrier, the books are kept after it, beside the workers' commit and next pass.
        bool overlap = false;
        int flags = 0, acc = 0;
        double du_real = 0, du_kc = 0, du_kl = 0, du_ext = 0, dmx = 0, dmy = 0, dmz = 0, dew = 0, dlj6 = 0, dlj12 = 0;
        long long cur_after = 0;
        int imol_moved = 0;
        if (ctl) {
            __syncwarp();  // (the lanes have written sh.tot)
            const Cand &M = sh.cand[sh.icur];
            overlap = sh.tot[RV_OVL] > 0.0;
            flags = overlap ? 2 : 0;
            cur_after = M.cur_prop;
            imol_moved = M.imol;
            bool out = false, finite = true;
            if (!overlap) {
                RngReader rng = make_reader(X, sh, M.cur_prop);
                if constexpr (biased) {
                    dew = sh.tot[RV_EW] - sh.eold[0]; dlj6 = sh.tot[RV_LJ6] - sh.eold[1]; dlj12 = sh.tot[RV_LJ12] - sh.eold[2];
                    du_real = (sh.tot[RV_EW] + sh.tot[RV_LJ12] - sh.tot[RV_LJ6]) - (sh.eold[0] + sh.eold[2] - sh.eold[1]);
                } else {
                    dew = sh.tot[RV_EW]; dlj6 = sh.tot[RV_LJ6]; dlj12 = sh.tot[RV_LJ12];
                    du_real = dew + dlj12 - dlj6;
                }
                du_kc = sh.tot[RV_DUC];
                du_kl = sh.tot[RV_DUL];
                double mx = 0, my = 0, mz = 0;
                for (int a = 0; a < na; ++a) { mx = mx + M.slot[a].q * M.slot[a].x; my = my + M.slot[a].q * M.slot[a].y; mz = mz + M.slot[a].q * M.slot[a].z; }
                dmx = mx - M.mu_old[0]; dmy = my - M.mu_old[1]; dmz = mz - M.mu_old[2];
                const double mux = sh.sc[SC_MU_X], muy = sh.sc[SC_MU_Y], muz = sh.sc[SC_MU_Z];
                // EwaldSumExternal_calc_dU (EwaldSumExternal.f90:68-82)
                du_ext = D.kext * ((2 * mux + dmx) * dmx + (2 * muy + dmy) * dmy + (2 * muz + dmz) * dmz);
                const double du_total = du_real + (du_kc + du_kl) + du_ext;
                // a non-finite energy change or bias force (an input the arithmetic cannot take:
                // NaN positions or random numbers, coincident charges) stops the chain before
                // the move is decided, with the state as it was after the last completed move
                finite = isfinite(du_total);
                if constexpr (biased) {
                    double F[3], T[3];
                    const double mu[3] = {mux + dmx, muy + dmy, muz + dmz};
                    const Slot *ns = M.slot;
                    mol_force_torque_f(na, [&](int i, int d) { return d == 0 ? ns[i].x : (d == 1 ? ns[i].y : ns[i].z); }, M.mass,
                                       [&](int i, int d) { return sh.tot[RV_F + 3 * i + d] + D.m2k * ns[i].q * (d == 0 ? mu[0] : (d == 1 ? mu[1] : mu[2])); },
                                       F, T);
                    for (int c = 0; c < 3; ++c) finite = finite && isfinite(F[c]) && isfinite(T[c]);
                    if (finite) {
                        const BiasNew b = mcm_init_new(F, T, D.xlf, D.xlc, D.dr, D.d_angle, shi_sans_exp_warp);
                        acc = mcm_accept(M.mv, F, T, b, du_total, D.xlf, D.xlc, rng);
                    }
                } else if (finite) {
                    // MonteCarloMove_accept_or_decline without bias: every bias term is an exact 0
                    // or 1 (cold = qold = cnew = qnew = 1), so the factor is exp(-dU) bit for bit
                    const double factor = c_exp(-du_total);
                    acc = rng.next() > factor ? 0 : 1;
                }
                out = rng.out != 0;
                cur_after = rng.cur();
                flags |= acc;
            }
            if (out) acc = 0;
            __syncwarp();
            if (lane == 0) {
                sh.accepted = acc;
                if (!finite) sh.abort = kAbortNonFinite;
                else if (out) sh.abort = kAbortStream;  // the interrupted move restarts from its first draw (sh.cursor unchanged)
                else {
                    if (acc) {
                        sh.last_mol = M.imol - 1;
                        for (int a = 0; a < na; ++a) {
                            sh.lx[a] = M.slot[a].x; sh.ly[a] = M.slot[a].y; sh.lz[a] = M.slot[a].z;
                            sh.mv_slot[a] = M.slot[a].pad;
                        }
                        const MolK<MX> mk(M.slot, na);
                        sh.mv_first = M.first; sh.mv_na = na; sh.mv_tmask = mk.tmask; sh.mv_simple = mk.simple;
                    }
                    sh.cursor = cur_after;
                    // the next move: the prepared candidate that matches what happened
                    sh.spec_ok = 0;
                    if (it + 1 < n_moves) {
                        const int sel = overlap ? 0 : ((acc && sh.cand[sh.spec[2]].imol == M.imol) ? 2 : 1);
                        const int buf = sh.spec[sel];
                        const Cand &C = sh.cand[buf];
                        if (C.valid && C.cur_start == cur_after) {
                            sh.icur = buf;
                            sh.spec_ok = 1;
                        }
                    }
                }
            }
        }
        __syncthreads();
        YAMC_PH(PH_DECIDE);
        if (sh.abort) break;
        const bool accepted = sh.accepted != 0;
        if (ctl) {
            // the totals, the log, the cycle counters and energy.dat rows (runmc.f90:230-279)
            if (lane == 0) {
                if (acc) {
                    sh.sc[SC_UU_EW] += dew; sh.sc[SC_UU_LJ6] += dlj6; sh.sc[SC_UU_LJ12] += dlj12;
                    sh.sc[SC_EK_C] += du_kc; sh.sc[SC_EK_LJ] += du_kl;
                    sh.sc[SC_MU_X] += dmx; sh.sc[SC_MU_Y] += dmy; sh.sc[SC_MU_Z] += dmz;
                    sh.sc[SC_N_MV_ACC] += 1.0;
                    ++n_acc;
                }
                sh.sc[SC_N_MV_STEPS] += 1.0;
                if (rank == 0) {
                    if (acc)
                        for (int a = 0; a < na; ++a) {  // x, y, z of the double4 (q unchanged): no read
                            double *pa = reinterpret_cast<double *>(D.atom + sh.mv_first + a);
                            pa[0] = sh.lx[a]; pa[1] = sh.ly[a]; pa[2] = sh.lz[a];
                        }
                    if (run->log) {
                        yamc_move_record rec;
                        rec.imol = imol_moved; rec.flags = flags; rec.cursor = cur_after;
                        rec.du_real = du_real; rec.du_k_coul = du_kc; rec.du_k_lj = du_kl; rec.du_ext = du_ext;
                        run->log[it] = rec;
                    }
                }
                sh.mic += 1;
                if (sh.mic == D.M) {
                    sh.mic = 0;
                    const double fr = sh.sc[SC_N_MV_STEPS] / D.M + sh.sc[SC_N_VOL_STEPS];
                    if (fmod(fr, D.n_store_energy_interval) < 1e-10 && rank == 0 && run->rows && rows < run->max_rows) {
                        const double *sc = sh.sc;
                        const double uext = D.kext * (sc[SC_MU_X] * sc[SC_MU_X] + sc[SC_MU_Y] * sc[SC_MU_Y] + sc[SC_MU_Z] * sc[SC_MU_Z]);
                        const double utew = sc[SC_UU_EW] + sc[SC_EK_C] + sc[SC_TAIL_C] + uext;
                        const double utlj = sc[SC_UU_LJ12] - sc[SC_UU_LJ6] + sc[SC_EK_LJ] + sc[SC_TAIL_LJ12] - sc[SC_TAIL_LJ6];
                        double *row = run->rows + 9 * (size_t)rows;
                        row[0] = (double)sh.icycle; row[1] = utew + utlj; row[2] = utew; row[3] = utlj;
                        row[4] = sc[SC_UU_EW]; row[5] = sc[SC_UU_LJ6]; row[6] = sc[SC_UU_LJ12];
                        row[7] = sc[SC_EK_C]; row[8] = sc[SC_EK_LJ];
                        ++rows;
                    }
                    sh.icycle += 1;
                }
            }
            __syncwarp();
        } else if (accepted) {
            // this CTA's staged copy of the moved atoms, by one thread of the last warp (two atoms may
            // share a block's box); the workers read it after the phase tables' barrier, and another CTA
            // that stages the molecule meanwhile takes its positions from sh.lx (last_mol)
            if (wtid == nwork - 1)
                for (int a = 0; a < sh.mv_na; ++a) {
                    if ((sh.mv_first + a) % G != rank) continue;
                    const int sl = (int)YAMC_IX(sh.mv_slot[a], nown);  // the atom's staging slot
                    double4 p = atom_s[sl];
                    p.x = sh.lx[a]; p.y = sh.ly[a]; p.z = sh.lz[a];
                    atom_s[sl] = p;
                    box_expand(box_s, sl / kBlk, p.x, p.y, p.z);
                }
            // commit: rho += delta (MC.f90:1245), in registers or in memory by the entry's owner; the
            // rows of LJ types that the molecule does not carry have no delta
            const int tmask = sh.mv_tmask;
            const bool simple = sh.mv_simple != 0;
            static_for<0, EPT>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                R.rho[k][0].x += R.dl[k][0].x; R.rho[k][0].y += R.dl[k][0].y;
#pragma unroll
                for (int t = 1; t <= NT; ++t) {
                    const Rt dx = pick<Rt>(simple, R.dl[k][1].x, R.dl[k][t].x), dy = pick<Rt>(simple, R.dl[k][1].y, R.dl[k][t].y);
                    const bool hit = (tmask >> (t - 1)) & 1;
                    R.rho[k][t].x += hit ? (double)dx : 0.0; R.rho[k][t].y += hit ? (double)dy : 0.0;
                }
            });
            if constexpr (EPT <= 0) {
                const R2 *dl_g = scratch_buf<MX>(D.scratch, 1, 1 + NT, S);
                for (int e = e0; e < S; e += gwork)
#pragma unroll
                    for (int t = 0; t <= NT; ++t) {
                        if (t > 0 && !((tmask >> (t - 1)) & 1)) continue;
                        double2 r = D.rho[(size_t)t * S + e];
                        const double2 d = to_d2(dl_g[(size_t)t * S + e]);
                        r.x += d.x; r.y += d.y;
                        D.rho[(size_t)t * S + e] = r;
                        if constexpr (MX) D.rho_f[(size_t)t * S + e] = make_float2((float)r.x, (float)r.y);
                    }
            }
        }
        ++moves_done;
        have_next = sh.spec_ok != 0;
        YAMC_PH(PH_COMMIT);
        if constexpr (MX) {
            acc_since += accepted;  // the same decisions in every CTA: every thread agrees
            if (refresh_every > 0 && acc_since >= refresh_every) {
                refresh_in_chain<NT, EPT>(D, scr, scr_atoms, e0, gwork, G, rank, sh, red, xch, xpar, cluster);
                static_for<0, EPT>([&](auto kc) {
                    constexpr int k = decltype(kc)::value;
#pragma unroll
                    for (int t = 0; t <= NT; ++t)
                        if (R.e[k] >= 0) R.rho[k][t] = D.rho[(size_t)t * S + R.e[k]];
                });
                xpar ^= 1;
                acc_since = 0;
                ++refreshes;
            }
        }
    }
#undef YAMC_PH

    if (prof) {
        __syncthreads();
        if (tid < PH_COUNT) A.prof[tid] += prof_s[tid];
    }
    {  // write back the register and shared state
#pragma unroll
        for (int k = 0; k < EPT; ++k)
            if (R.e[k] >= 0) {
#pragma unroll
                for (int t = 0; t <= NT; ++t) D.rho[(size_t)t * S + R.e[k]] = R.rho[k][t];
            }
        if (tid == 0 && rank == 0) {
            for (int c = 0; c < SC_COUNT; ++c) D.scal[c] = run->sc[c] = sh.sc[c];
            run->cnt[CN_ICYCLE] = sh.icycle;
            run->cnt[CN_ACC_SINCE_REFRESH] = acc_since;
            run->cnt[CN_REFRESHES] = D.cnt[CN_REFRESHES] + refreshes;
            run->cnt[CN_MOVE_IN_CYCLE] = sh.mic;
            for (int c = 0; c < CN_COUNT; ++c) D.cnt[c] = run->cnt[c];
            run->cursor = sh.cursor;
            run->moves_done = moves_done;
            run->n_rows = rows;
            run->accepted = n_acc;
            run->status = sh.abort == kAbortNonFinite ? YAMC_ENAN : (sh.abort ? YAMC_ERNG_EXHAUSTED : YAMC_OK);
        }
    }
    if (G > 1) cluster.sync();  // no CTA leaves while another may still address its shared memory
}

// nrep chains of one launch shape: nrep clusters of L.G CTAs, chain r on cluster r
template <int NT, int EPT, bool SPLIT, bool MX>
int launch_chain_t(const LaunchCfg &L, cudaStream_t stream, int nrep, const ChainArgs &args) {
    auto kfn = k_chain<NT, EPT, SPLIT, MX>;
    if (const int r = grant_smem(kfn, L.smem)) return r;
    if (L.G > 8) CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(L.G * nrep, 1, 1);
    cfg.blockDim = dim3(L.B, 1, 1);
    cfg.dynamicSmemBytes = L.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = L.G;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CUDA_TRY(cudaLaunchKernelEx(&cfg, kfn, args));
    return YAMC_OK;
}

// clusters of shape L that can be resident at once (0 if the shape does not launch)
template <int NT, int EPT, bool SPLIT, bool MX>
int max_clusters_t(const LaunchCfg &L, int *out) {
    auto kfn = k_chain<NT, EPT, SPLIT, MX>;
    if (const int r = grant_smem(kfn, L.smem)) return r;
    if (L.G > 8) CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(L.G, 1, 1);
    cfg.blockDim = dim3(L.B, 1, 1);
    cfg.dynamicSmemBytes = L.smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = L.G;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CUDA_TRY(cudaOccupancyMaxActiveClusters(out, kfn, &cfg));
    return YAMC_OK;
}


// the launch entry points of each LJ type count, defined in yamc_chain_inst.cu (compiled once per
// count): every (entries per thread, split, mixed) variant of that count
template <int NT> int launch_chain_nt(const LaunchCfg &L, bool split, bool mx, cudaStream_t s, int nrep, const ChainArgs &a);
template <int NT> int max_clusters_nt(const LaunchCfg &L, bool split, bool mx, int *out);
#define YAMC_DECLARE_NT(N)                                                                                       \
    template <> int launch_chain_nt<N>(const LaunchCfg &, bool, bool, cudaStream_t, int, const ChainArgs &);     \
    template <> int max_clusters_nt<N>(const LaunchCfg &, bool, bool, int *);
YAMC_DECLARE_NT(1)
YAMC_DECLARE_NT(2)
YAMC_DECLARE_NT(3)
YAMC_DECLARE_NT(4)
#undef YAMC_DECLARE_NT

}  // namespace yamc
