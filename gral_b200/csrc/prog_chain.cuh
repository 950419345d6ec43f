// prog_chain.cuh -- the row-chain schedule of the slab family's Gauss-Seidel sweeps: what its kernels
// share (prog_chain.cu: pressure and model 1; prog_chain_scalar.cu: models 0 and 2).
//
// A sweep is two launches.  A parallel kernel evaluates every column's coefficients and sources
// (all that does not read values the sweep itself changes), runs the forward elimination and writes
// one contiguous record per column.  The chain kernel then walks the sweep rows i1, a row's columns
// j1 in order, and passes finished columns on as stamped words (float bits and a stamp in one 8-byte
// access): through rings in shared memory inside a block and to the next block of the cluster,
// through global memory from one cluster's claim to the next.
//
// What bounds it: the chain of (rows + columns) column steps.  A step's time is two first-order
// vertical recurrences over about 40 levels, whose every operation is rounded as in the reference.
// Run one level after the other they take about 20 (back-substitution) and 12 (Q) cycles a level.
// Here a lane holds levels 2*lane and 2*lane+1 and the warp iterates x_k = f_k(x_k-1) on all
// levels at once, each round passing values two levels on through one shuffle, until a whole round
// changes no bit.  A state that f maps to itself, starting from the exact first level, is the
// sequential recurrence's result bit for bit (by induction over the levels), whatever the number of
// rounds; the recurrences are contractions (the influence of a level fades by relax*P <= 0.1 or
// by C*T, well below 1), so a few rounds reach it instead of forty levels.
//
// A claim (the strips of one cluster) is taken from an atomic counter in order and waits only on the
// claim before, so clusters need not be resident together; the blocks of a cluster are.  Every wait
// is bounded and gives up when another warp has set the error word.
#pragma once

#include "prog_common.cuh"
#include "prog_kernels.cuh"
#include "prog_level.cuh"

namespace gral {

using KFn = void (*)(KArgs, SweepGeom, ChainBufs);

// chain and coefficient kernels of models 0 and 2 (kind = PH_U, PH_V, PH_W, PH_TKE), pairs of a record
KFn chain_scalar_kernel(int kind, int model);
KFn chain_scalar_terms(int kind, int model);
int chain_scalar_pairs(int model);
// grid of a chain kernel: whole clusters, at most one per claim
cudaError_t chain_grid_of(const void *kernel, int threads, long long claims, int *grid);
bool chain_pow2(float x);

namespace {

constexpr int CH_RING = 8;    // hand-off slots between a row and the row below it in the block
constexpr int CH_AHEAD = 4;   // columns of a warp whose records are asked into L2 ahead
constexpr int CT_COLS = 32;   // columns of a tile of the coefficient kernels
constexpr int CT_THREADS = 256;

enum { COMP_U = 0, COMP_V = 1, COMP_W = 2 };

__device__ __forceinline__ void chain_dir(int it, int &IS, int &JS) {
    // PrognosticFlowfield.cs:770-802
    const int m = it % 4;
    IS = (m == 0 || m == 1) ? -1 : 1;
    JS = (m == 1 || m == 2) ? -1 : 1;
}

// Tile of a coefficient launch: CT_COLS columns along j of one sweep row of one unit.
struct Tile {
    int u, s, i, j0, nc, IS, JS;
    bool ok;
};
__device__ __forceinline__ Tile make_tile(const KArgs &a, const SweepGeom &g, const ChainBufs &b, bool reverse) {
    Tile t;
    chain_dir(*a.it_global, t.IS, t.JS);
    if (reverse) { t.IS = -t.IS; t.JS = -t.JS; }
    const int per = (g.nj + CT_COLS - 1) / CT_COLS;
    const int q = blockIdx.x / per;
    const int c0 = (blockIdx.x - q * per) * CT_COLS;
    t.u = q / g.ni;
    const int i1 = g.ia + (q - t.u * g.ni);
    t.i = (t.IS == 1) ? i1 : a.nii - i1 + 1;
    t.nc = min(CT_COLS, g.nj - c0);
    // the tile's columns in ascending j: sweep columns j1 = ja + c0 ... of either direction
    t.j0 = (t.JS == 1) ? g.ja + c0 : a.njj - (g.ja + c0 + t.nc - 1) + 1;
    t.ok = b.unit_lo + t.u < *a.nact;
    t.s = t.ok ? a.act[b.unit_lo + t.u] : 0;
    t.ok = t.ok && a.sit[t.s].active;
    return t;
}

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Stamped words of two neighbouring levels.
struct Words2 {
    unsigned long long a, b;
};
__device__ __forceinline__ unsigned long long word(float v, unsigned stamp) {
    return ((unsigned long long)stamp << 32) | __float_as_uint(v);
}
__device__ __forceinline__ float word_val(unsigned long long w) { return __uint_as_float((unsigned)w); }
__device__ __forceinline__ bool stamped(const Words2 &w, unsigned stamp) {
    return (unsigned)(w.a >> 32) == stamp && (unsigned)(w.b >> 32) == stamp;
}
// The accesses of a lane without levels (`on` false) are predicated off rather than branched over:
// a branch costs the chain a reconvergence.
__device__ __forceinline__ Words2 ld_words(const unsigned long long *p, bool on) {
    Words2 w;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u64 %0, 0;\n\tmov.u64 %1, 0;\n\t"
        "@q ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n\t}"
        : "=&l"(w.a), "=&l"(w.b)
        : "l"(p), "r"((unsigned)on)
        : "memory");
    return w;
}
__device__ __forceinline__ void st_words(unsigned long long *p, const Words2 &w, bool on) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n\t}" ::"l"(p),
        "l"(w.a), "l"(w.b), "r"((unsigned)on)
        : "memory");
}
__device__ __forceinline__ void st_pair(float2 *p, float2 v, bool on) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q st.global.cg.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(p),
                 "f"(v.x), "f"(v.y), "r"((unsigned)on)
                 : "memory");
}
__device__ __forceinline__ Words2 lds_words(unsigned p) {
    Words2 w;
    asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(w.a), "=l"(w.b) : "r"(p) : "memory");
    return w;
}
__device__ __forceinline__ void sts_words(unsigned p, const Words2 &w) {
    asm volatile("st.volatile.shared.v2.u64 [%0], {%1, %2};" ::"r"(p), "l"(w.a), "l"(w.b) : "memory");
}
__device__ __forceinline__ void l2_ahead(const void *p, bool on) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t@q prefetch.global.L2 [%0];\n\t}" ::"l"(p),
                 "r"((unsigned)on));
}
// d = a + b or a * b where `on`, as one predicated instruction: the compiler's own forms of a
// conditional assignment (a select after the operation, or a branch over it) lengthen the recurrences
// (a round of the momentum step took 109 cycles with `if`, 80 with a select, 68 this way).
__device__ __forceinline__ void add_if(float &d, float a, float b, unsigned on) {
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q add.rn.f32 %0, %1, %2;\n\t}" : "+f"(d) : "f"(a), "f"(b), "r"(on));
}
__device__ __forceinline__ void mul_if(float &d, float a, float b, unsigned on) {
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q mul.rn.f32 %0, %1, %2;\n\t}" : "+f"(d) : "f"(a), "f"(b), "r"(on));
}
__device__ __forceinline__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }

// Bound of a spin: every 32nd call looks at the error word and the clock; true when the wait must
// end (warp-uniform).
struct SpinBound {
    unsigned long long t0 = 0;
    unsigned n = 0;
    __device__ __forceinline__ bool expired(const KArgs &a) {
        if (n == 0) t0 = globaltimer_ns();
        if ((++n & 31) != 0) return false;
        bool stop = *(volatile int *)a.err != ERR_NONE;
        if (!stop && globaltimer_ns() - t0 > a.wait_limit_ns) {
            atomicCAS(a.err, ERR_NONE, ERR_TIMEOUT);
            stop = true;
        }
        return __any_sync(0xffffffffu, stop);
    }
};

// Rounds of the two recurrences before the first test; a failed test continues round by round.  One
// round less or more: 400x400 U chain 0.45 / 0.42 / 0.45 ms for 4 / 3 / 2, pressure 0.58 / 0.57 / 0.60 for
// 5 / 6 / 4 (the pressure's influence fades by 0.17 a level where the layers are as thick as wide).
constexpr int ROUNDS_MOM = 3, ROUNDS_PRESS = 6;

// Bytes of a ring slot (every lane's words of one column) and of a ring in shared memory.
template <int NV>
__host__ __device__ constexpr unsigned slot_bytes() { return NV * 32u * 16u; }
template <int NV>
__host__ __device__ constexpr unsigned ring_bytes() { return CH_RING * slot_bytes<NV>(); }

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// address of this block's shared-memory location p in block `rank` of the cluster
__device__ __forceinline__ unsigned remote(unsigned p, unsigned rank) {
    unsigned q;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"(p), "r"(rank));
    return q;
}
__device__ __forceinline__ void st_remote(unsigned p, const Words2 &w, bool on) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q st.relaxed.cluster.shared::cluster.v2.u64 [%0], {%1, %2};\n\t}" ::"r"(p),
        "l"(w.a), "l"(w.b), "r"((unsigned)on)
        : "memory");
}
__device__ __forceinline__ void st_remote(unsigned p, int v, bool on) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.relaxed.cluster.shared::cluster.s32 [%0], %1;\n\t}" ::"r"(p),
                 "r"(v), "r"((unsigned)on)
                 : "memory");
}
__device__ __forceinline__ unsigned ld_remote(unsigned p) {
    unsigned v;
    asm volatile("ld.relaxed.cluster.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}

// Shared memory of a block: the rings 0..SR (ring r: what row r takes from above; ring SR: what the
// strip's last row finished), the claim, and how many columns each ring's reader has taken.
template <int SR, int NV>
struct ChainSmem {
    alignas(16) unsigned long long ring[(SR + 1) * ring_bytes<NV>() / 8];
    unsigned claim;
    int taken[SR + 1];
};

// One cluster of CL blocks takes CL strips of SR rows each (a claim), M warps per row: warp m of a
// row runs the columns m, m+M, ..., so that while one warp is in its step the row's other warps
// store, ask for their next record and load it.  A finished column goes into the ring of the row
// below, where that row and the next column's warp of this row read it; from the last row of a
// strip also into ring 0 of the next block of the cluster, and from the last row of the claim into
// the words in global memory, which the feeder warp of the next claim's first block turns into its
// ring 0 (for the sweep's first row: the values the sweep does not change).
template <class Job, int PH, int SR, int M, int CL, int IS, int JS>
__device__ __forceinline__ void run_chain(const KArgs &a, const SweepGeom &g, const ChainBufs &b,
                                          ChainSmem<SR, Job::NV> &sm, Job job = Job()) {
    constexpr int NV = Job::NV;                   // values of a column handed to the row below,
    constexpr int NJ = Job::NJ;                   // the first NJ of them also to the row's next column
    constexpr int NF = Job::NF;                   // and the first NF stored in fields
    constexpr int WCOL = NV * KMAX_LEVELS;        // words of a column in global memory
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ks = a.ks, nj = g.nj, l2 = 2 * lane;
    const bool mine = l2 < ks;       // this lane holds levels of the column
    const unsigned rank = cluster_rank();
    const unsigned ring0 = smem_u32(sm.ring) + lane * 16u;
    job.init(a, lane);
    const unsigned gstamp = (unsigned)*b.epoch * 8u + PH;      // of the words in global memory
    const unsigned units = (unsigned)min(b.unit_n, max(0, *a.nact - b.unit_lo));
    const unsigned ngroups = (unsigned)((g.ni + SR * CL - 1) / (SR * CL));
    const unsigned total = ngroups * units;
    unsigned *ctr = a.counters + 8 * b.ctr_slot + PH;
    unsigned seq = 0;                // claims run by this block: part of the ring stamps
    const int jfirst = (JS == 1) ? g.ja : a.njj - g.ja + 1;
    const size_t wrow = (size_t)nj * WCOL;
    for (;;) {
        cluster_sync();
        if (rank == 0 && threadIdx.x == 0)
            sm.claim = (*(volatile int *)a.err != ERR_NONE) ? 0xffffffffu : atomicAdd(ctr, 1u);
        if (threadIdx.x <= SR) sm.taken[threadIdx.x] = 0;
        cluster_sync();
        const unsigned t = ld_remote(remote(smem_u32(&sm.claim), 0));
        if (t >= total) break;
        ++seq;
        const int u = (int)(t % units), group = (int)(t / units);
        const int s = a.act[b.unit_lo + u];
        const int first = g.ia + (group * CL + (int)rank) * SR, rows = min(SR, g.ia + g.ni - first);
        if (!a.sit[s].active || rows <= 0) continue;
        auto row_i = [&](int r) { return (IS == 1) ? first + r : a.nii - (first + r) + 1; };
        unsigned long long *gout = b.words + ((size_t)(b.unit_lo + u) * ngroups + group) * wrow + l2;
        const unsigned sbase = seq << 16;
        // waits until ring r's reader has taken n columns (their slots are free)
        int seen = 0;
        auto room = [&](int r, int n) {
            if (seen >= n) return true;
            SpinBound sb;
            for (;;) {
                seen = __shfl_sync(0xffffffffu, *(volatile int *)(sm.taken + r), 0);
                if (seen >= n) return true;
                if (sb.expired(a)) return false;
            }
        };
        auto slot = [&](int c) { return (unsigned)(c & (CH_RING - 1)) * slot_bytes<NV>(); };
        auto push = [&](unsigned ring, int c, const typename Job::Val &v) {
            const unsigned st = sbase + (unsigned)(c + 1), p = ring + slot(c);
#pragma unroll
            for (int q = 0; q < NV; ++q) sts_words(p + q * 512u, Words2{word(v.v[q].x, st), word(v.v[q].y, st)});
        };
        if (warp == SR * M) {                                      // the feeder
            constexpr int NA = 4;                                  // columns in flight
            bool ok = true;
            if (rank > 0) {
            } else if (group > 0) {
                const unsigned long long *gin = gout - wrow;
                Words2 w[NA][NV];
                auto peek = [&](int c, Words2 (&x)[NV]) {
#pragma unroll
                    for (int q = 0; q < NV; ++q) x[q] = ld_words(gin + (size_t)c * WCOL + q * KMAX_LEVELS, mine && c < nj);
                };
                auto feed = [&](int c, Words2 (&x)[NV]) {
                    SpinBound sb;
                    for (;;) {
                        bool got = true;
#pragma unroll
                        for (int q = 0; q < NV; ++q) got = got && stamped(x[q], gstamp);
                        if (__all_sync(0xffffffffu, got || !mine)) break;
                        if (sb.expired(a)) return false;
                        peek(c, x);
                    }
                    typename Job::Val v;
#pragma unroll
                    for (int q = 0; q < NV; ++q) v.v[q] = make_float2(word_val(x[q].a), word_val(x[q].b));
                    if (!room(0, c - CH_RING + 1)) return false;
                    push(ring0, c, v);
                    peek(c + NA, x);
                    return true;
                };
#pragma unroll
                for (int q = 0; q < NA; ++q) peek(q, w[q]);
                for (int c = 0; c < nj && ok; c += NA)
#pragma unroll
                    for (int q = 0; q < NA; ++q)
                        if (ok && c + q < nj) ok = feed(c + q, w[q]);
            } else {
                const int cb = (row_i(0) - IS) * a.nj2 + jfirst;
                auto value = [&](int c) {
                    return job.still(a, ((size_t)s * a.ncols + (size_t)(cb + JS * min(c, nj - 1))) * ks, lane);
                };
                typename Job::Val v[NA];
#pragma unroll
                for (int q = 0; q < NA; ++q) v[q] = value(q);
                for (int c = 0; c < nj && ok; c += NA)
#pragma unroll
                    for (int q = 0; q < NA; ++q)
                        if (ok && c + q < nj) {
                            ok = room(0, c + q - CH_RING + 1);
                            push(ring0, c + q, v[q]);
                            v[q] = value(c + q + NA);
                        }
            }
            continue;
        }
        const int r = warp / M, m = warp - r * M;
        if (r >= rows) continue;
        const bool more_rows = first + rows < g.ia + g.ni;             // a strip follows this one
        const bool last = r + 1 == rows;                               // the strip's last row
        const bool next_block = last && more_rows && rank + 1 < CL;    // ... read by the cluster's next block
        const bool next_claim = last && more_rows && rank + 1 == CL && mine;
        const unsigned ring_in = ring0 + (unsigned)r * ring_bytes<NV>(), ring_out = ring_in + ring_bytes<NV>();
        const unsigned ring_far = remote(ring0, min(rank + 1, CL - 1u));
        const unsigned taken_far = remote(smem_u32(sm.taken + SR), max((int)rank, 1) - 1);
        const bool far_above = r == 0 && rank > 0 && lane == 0;        // this row reads the block before
        const bool watch = !last || next_block;                        // somebody reads this row's columns
        const int taker = last ? SR : r + 1;
        const int col0 = row_i(r) * a.nj2 + jfirst;
        const size_t e0 = ((size_t)s * a.ncols + (size_t)col0) * ks;
        float2 *out_f[NF];
#pragma unroll
        for (int q = 0; q < NF; ++q) out_f[q] = reinterpret_cast<float2 *>(job.F[q] + e0) + lane + (long long)m * JS * (ks / 2);
        unsigned long long *wout = gout + (size_t)m * WCOL;
        job.template begin<M>(a, b, u, s, col0 + JS * m, lane);
        if (m == 0) push(ring_out, -1, job.still(a, e0 - (long long)JS * ks, lane));   // left of the first column
        typename Job::Rec rec;
        for (int c = m; c < m + CH_AHEAD * M; c += M) job.ahead(c < nj);
        if (m < nj) job.load(rec);
        for (int c = m; c < nj; c += M) {
            Words2 wI[NV], wJ[NJ];
            const unsigned want = sbase + (unsigned)(c + 1), pI = ring_in + slot(c), pJ = ring_out + slot(c - 1);
            SpinBound sb;
            bool ok = true;
            for (;;) {
#pragma unroll
                for (int q = 0; q < NJ; ++q) wJ[q] = lds_words(pJ + q * 512u);
#pragma unroll
                for (int q = 0; q < NV; ++q) wI[q] = lds_words(pI + q * 512u);
                bool got = true;
#pragma unroll
                for (int q = 0; q < NJ; ++q) got = got && stamped(wJ[q], want - 1u);
#pragma unroll
                for (int q = 0; q < NV; ++q) got = got && stamped(wI[q], want);
                if (__all_sync(0xffffffffu, got)) break;
                if (sb.expired(a)) { ok = false; break; }
            }
            typename Job::Val vI;
#pragma unroll
            for (int q = 0; q < NV; ++q) vI.v[q] = make_float2(word_val(wI[q].a), word_val(wI[q].b));
            float2 vJ[NJ];
#pragma unroll
            for (int q = 0; q < NJ; ++q) vJ[q] = make_float2(word_val(wJ[q].a), word_val(wJ[q].b));
            const typename Job::Val v = job.step(rec, vI, vJ);
            if (!ok) break;
            push(ring_out, c, v);
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                const unsigned st = sbase + (unsigned)(c + 1);
                st_remote(ring_far + slot(c) + q * 512u, Words2{word(v.v[q].x, st), word(v.v[q].y, st)}, next_block);
            }
            // the rest runs while the row's next column is in its step
            *(volatile int *)(sm.taken + r) = c + 1;
            st_remote(taken_far, c + 1, far_above);
            if (c + M < nj) job.load(rec);
#pragma unroll
            for (int q = 0; q < NV; ++q)
                st_words(wout + q * KMAX_LEVELS, Words2{word(v.v[q].x, gstamp), word(v.v[q].y, gstamp)}, next_claim);
#pragma unroll
            for (int q = 0; q < NF; ++q) {    // levels the sweep does not change keep their value
                st_pair(out_f[q], v.v[q], mine);
                out_f[q] += M * JS * (ks / 2);
            }
            wout += (size_t)M * WCOL;
            job.ahead(c + CH_AHEAD * M < nj);
            if (watch && !room(taker, c + M - CH_RING + 1)) break;
        }
    }
    cluster_sync();      // no block leaves while another may still write into its shared memory
}

// Strip shape: rows of a block, warps of a row, blocks of a cluster.  Measured on the 400x400 grid,
// ms of an iteration: (4,2,8) 3.44, (3,2,8) 3.51, (2,3,8) 3.61, (4,3,8) 3.48; one warp per row and every
// hand-off between blocks through global memory 4.25.
constexpr int CH_SR = 4, CH_M = 2, CH_CL = 8;
constexpr int CH_THREADS = (CH_SR * CH_M + 1) * 32;

}  // namespace

}  // namespace gral
