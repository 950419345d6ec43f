// prog_chain_diag.cu -- row chains (prog_chain.cuh) of DiagnosticFlowfield.Calculate's pressure sweeps
// (DiagnosticFlowfield.cs:86-315) on the full-height fields after a prognostic solve.
//
// Every column of the sweep range, levels KKART+1..NKK-1, the four neighbours' DPM of this sweep or the
// last one, PIMP/QIMP at NKK zero, no quantisation and no residual.  The forward elimination is the
// same for all columns (a table) but for P at KKART+1, so a column's record is only DIV/DTIME; the
// successors' DPM is read from the field one column ahead.  A lane holds L levels (2 up to NKK 64, 6 up
// to 192); DPM and DIV/DTIME live in L/2 planes [situation][col][64] of level pairs, so that a lane's
// pair is one aligned access: level k = L*lane + 2*q + r is element 2*lane + r of plane q.
#include <algorithm>

#include "prog_chain.cuh"

namespace gral {

namespace {

struct DiagChainArgs {
    DiagTabs t;
    float *div;          // planes of the units in flight, DIV/DTIME
    size_t div_plane;    // floats of a plane
    float *dpm;          // planes of all situations
    size_t dpm_plane;
};

// Sweep orders by IterationLoops % 4 (DiagnosticFlowfield.cs:94-315): 0 rows and columns ascending,
// 1 rows descending, 2 both descending, 3 columns descending.
__device__ __forceinline__ void diag_dir(int it, int &IS, int &JS) {
    const int m = it % 4;
    IS = (m == 2 || m == 3) ? -1 : 1;
    JS = (m == 1 || m == 2) ? -1 : 1;
}

template <int L>
__device__ __forceinline__ size_t plane_at(size_t plane, size_t cell, int k) {
    const int lane = k / L, o = k - lane * L;
    return (size_t)(o >> 1) * plane + cell * 64 + 2 * lane + (o & 1);
}

// a: full-height slab (KS = NKK+2)
template <int L>
__global__ void __launch_bounds__(256) k_diag_div(KArgs a, DiagChainArgs d, int unit_lo) {
    const int u = blockIdx.y, s = a.act[unit_lo + u];
    const int col = blockIdx.x * 8 + (threadIdx.x >> 5), i = col / a.nj2, j = col - i * a.nj2;
    if (i < 2 || i > a.nii - 1 || j < 2 || j > a.njj - 1) return;
    const int KK = a.meta[col].kkart, top = a.nkk - 1;
    const Acc<false> x = make_acc<false>(a, s, col);
    const long long E = a.nj2, N = 1;
    const float DXK = a.dxk, DYK = a.dyk, DT = d.t.dtime[s];
    for (int k = KK + 1 + (threadIdx.x & 31); k <= top; k += 32) {
        const float u0 = a.uk[x.at(0, k)], uE = a.uk[x.at(E, k)], v0 = a.vk[x.at(0, k)], vN = a.vk[x.at(N, k)];
        const float w0 = a.wk[x.at(0, k)], wT = a.wk[x.at(0, k + 1)];
        const float dz = d.t.dzk[k];
        const float DIV = (k > KK + 1) ? (u0 - uE) * DYK * dz + (v0 - vN) * DXK * dz + (w0 - wT) * DXK * DYK
                                       : (u0 - uE) * DYK * dz + (v0 - vN) * DXK * dz - wT * DXK * DYK;
        d.div[plane_at<L>(d.div_plane, (size_t)u * a.ncols + col, k)] = DIV / DT;
    }
}

// velocity correction without quantisation on levels 1..NKK-1 (:320-382)
template <int L>
__global__ void __launch_bounds__(256) k_diag_velcorr_planes(KArgs a, DiagChainArgs d) {
    const int s = a.act[blockIdx.y];
    const int col = blockIdx.x * 8 + (threadIdx.x >> 5), i = col / a.nj2, j = col - i * a.nj2;
    if (i < 2 || i > a.nii - 1 || j < 2 || j > a.njj - 1) return;
    const int KK = a.meta[col].kkart, KKW = a.meta[col - a.nj2].kkart, KKS = a.meta[col - 1].kkart;
    const float DXK = a.dxk, DYK = a.dyk, DT = d.t.dtime[s];
    const Acc<false> x = make_acc<false>(a, s, col);
    const size_t cell = (size_t)s * a.ncols + col;
    auto dpm = [&](size_t c, int k) { return d.dpm[plane_at<L>(d.dpm_plane, c, k)]; };
    for (int k = 1 + (threadIdx.x & 31); k <= a.nkk - 1; k += 32) {
        const float c = dpm(cell, k);
        const float DDPX = dpm(cell - a.nj2, k) - c, DDPY = dpm(cell - 1, k) - c;
        const float DDPZ = (k > KK + 1) ? dpm(cell, k - 1) - c : 0.0f;
        float &u = a.uk[x.at(0, k)], &v = a.vk[x.at(0, k)], &w = a.wk[x.at(0, k)];
        u = ((KK < k) && (KKW < k)) ? u + (DDPX / DXK * DT) : 0.0f;
        v = ((KK < k) && (KKS < k)) ? v + (DDPY / DYK * DT) : 0.0f;
        w = (KK + 1 < k) ? w + (DDPZ * 2 / (d.t.dzk[k] + d.t.dzk[k - 1]) * DT) : 0.0f;
    }
}

// a: KS = 64 (a plane's column)
template <int L, int IS, int JS, bool P2>
struct DiagChain {
    static constexpr int NP = L / 2, NV = NP, NJ = NP, NF = NP;
    struct Rec {
        float2 t[NP], si[NP], sj[NP];
        int kk;
    };
    struct Val {
        float2 v[NP];
    };
    const DiagChainArgs &d;
    float atp[L], T[L], P1[L], P0[L], dz[L];
    float dxk, dyk, rx, ry;
    float *F[NF];
    int top, lo;               // lo: this lane's first level
    const float2 *div, *own;   // this lane's pair of plane 0 at the next column to load
    const ColMeta *meta;
    int hstep, rowstep, mstep;

    __device__ __forceinline__ DiagChain(const DiagChainArgs &args) : d(args) {}
    __device__ __forceinline__ void init(const KArgs &a, int lane) {
        dxk = a.dxk; dyk = a.dyk;
        rx = 1.0f / dxk; ry = 1.0f / dyk;
        top = a.nkk - 1;
        lo = L * lane;
#pragma unroll
        for (int q = 0; q < NF; ++q) F[q] = d.dpm + (size_t)q * d.dpm_plane;
#pragma unroll
        for (int q = 0; q < L; ++q) {
            const int k = min(lo + q, top);
            atp[q] = d.t.atp[k]; dz[q] = d.t.dzk[k];
            T[q] = d.t.tab[k]; P1[q] = d.t.tab[a.nkk + 2 + k]; P0[q] = d.t.tab[2 * (a.nkk + 2) + k];
        }
    }
    template <int M>
    __device__ __forceinline__ void begin(const KArgs &a, const ChainBufs &, int u, int s, int col, int lane) {
        div = reinterpret_cast<const float2 *>(d.div + ((size_t)u * a.ncols + col) * 64) + lane;
        own = reinterpret_cast<const float2 *>(d.dpm + ((size_t)s * a.ncols + col) * 64) + lane;
        meta = a.meta + col;
        hstep = JS * M * 32;
        mstep = JS * M;
        rowstep = IS * a.nj2 * 32;
    }
    __device__ __forceinline__ void ahead(bool) {}
    __device__ __forceinline__ void load(Rec &r) {
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const size_t p = (size_t)q * (d.dpm_plane / 2);
            r.t[q] = __ldcg(div + (size_t)q * (d.div_plane / 2));
            r.si[q] = __ldcg(own + p + rowstep);
            r.sj[q] = __ldcg(own + p + JS * 32);
        }
        r.kk = meta->kkart;
        div += hstep;
        own += hstep;
        meta += mstep;
    }
    __device__ __forceinline__ Val still(const KArgs &, size_t base, int lane) const {
        Val o;
#pragma unroll
        for (int q = 0; q < NP; ++q) o.v[q] = __ldcg(reinterpret_cast<const float2 *>(F[q] + base) + lane);
        return o;
    }
    __device__ __forceinline__ float dim(float t, float dzk, float si, float sj, float pi, float pj) const {
        const float a = (IS == 1) ? pi + si : si + pi, b = (JS == 1) ? pj - sj : sj - pj;
        const float qi = P2 ? a * rx : div_by(a, dxk, rx), qj = P2 ? b * ry : div_by(b, dyk, ry);
        return t + qi * dyk * dzk + qj * dxk * dzk;
    }
    __device__ __forceinline__ Val step(const Rec &r, const Val &vI, const float2 (&vJ)[NJ]) const {
        float D[L], Q[L], v[L], P[L];
        unsigned on[L];
#pragma unroll
        for (int q = 0; q < L; ++q) {
            const int p = q / 2;
            const bool y = q & 1;
            on[q] = lo + q > r.kk && lo + q <= top;
            P[q] = (lo + q > r.kk + 1) ? P1[q] : P0[q];
            D[q] = dim(y ? r.t[p].y : r.t[p].x, dz[q], y ? r.si[p].y : r.si[p].x, y ? r.sj[p].y : r.sj[p].x,
                       y ? vI.v[p].y : vI.v[p].x, y ? vJ[p].y : vJ[p].x);
            Q[q] = 0.0f;
            v[q] = 0.0f;
        }
        float inQ = 0.0f, inV = 0.0f;
        // Q downwards from the zero at NKK, DPM upwards from the zero at KKART
        auto down = [&]() {
#pragma unroll
            for (int q = L - 1; q >= 0; --q) mul_if(Q[q], atp[q] * (q == L - 1 ? inQ : Q[q < L - 1 ? q + 1 : q]) + D[q], T[q], on[q]);
        };
        auto up = [&]() {
#pragma unroll
            for (int q = 0; q < L; ++q) add_if(v[q], P[q] * (q == 0 ? inV : v[q > 0 ? q - 1 : q]), Q[q], on[q]);
        };
        down();
#pragma unroll
        for (int n = 0; n < (L == 2 ? ROUNDS_PRESS : 2); ++n) {
            inV = __shfl_up_sync(0xffffffffu, v[L - 1], 1);
            inQ = __shfl_down_sync(0xffffffffu, Q[0], 1);
            up();
            down();
        }
        for (;;) {
            const float nV = __shfl_up_sync(0xffffffffu, v[L - 1], 1), nQ = __shfl_down_sync(0xffffffffu, Q[0], 1);
            const bool more = __any_sync(0xffffffffu, differ(nQ, inQ));
            inV = nV; inQ = nQ;
            up();
            if (!more) break;
            down();
        }
        for (;;) {
            const float nV = __shfl_up_sync(0xffffffffu, v[L - 1], 1);
            const bool more = __any_sync(0xffffffffu, differ(nV, inV));
            inV = nV;
            up();
            if (!more) break;
        }
        Val o;
#pragma unroll
        for (int q = 0; q < NP; ++q) o.v[q] = make_float2(v[2 * q], v[2 * q + 1]);
        return o;
    }
};

// rows of a block: with six levels a lane the rings of four rows would pass 48 KB
template <int L>
__host__ __device__ constexpr int diag_sr() { return L == 2 ? CH_SR : 2; }
template <int L>
__host__ __device__ constexpr int diag_threads() { return (diag_sr<L>() * CH_M + 1) * 32; }
int diag_claims(int ni, int levels) {
    const int per = (levels == 2 ? diag_sr<2>() : diag_sr<6>()) * CH_CL;
    return (ni + per - 1) / per;
}

template <int L, bool P2>
__global__ void __cluster_dims__(CH_CL, 1, 1) __launch_bounds__(diag_threads<L>(), 1)
    k_diag_chain(KArgs a, SweepGeom g, ChainBufs b, DiagChainArgs d) {
    constexpr int SR = diag_sr<L>(), M = CH_M, CL = CH_CL;
    __shared__ ChainSmem<SR, L / 2> sm;
    for (unsigned q = threadIdx.x; q < sizeof(sm.ring) / 8; q += diag_threads<L>()) sm.ring[q] = 0ull;
    int is, js;
    diag_dir(a.diag_iter, is, js);
    if (is == 1) {
        if (js == 1) run_chain<DiagChain<L, 1, 1, P2>, PH_DIAG, SR, M, CL, 1, 1>(a, g, b, sm, DiagChain<L, 1, 1, P2>(d));
        else run_chain<DiagChain<L, 1, -1, P2>, PH_DIAG, SR, M, CL, 1, -1>(a, g, b, sm, DiagChain<L, 1, -1, P2>(d));
    } else {
        if (js == 1) run_chain<DiagChain<L, -1, 1, P2>, PH_DIAG, SR, M, CL, -1, 1>(a, g, b, sm, DiagChain<L, -1, 1, P2>(d));
        else run_chain<DiagChain<L, -1, -1, P2>, PH_DIAG, SR, M, CL, -1, -1>(a, g, b, sm, DiagChain<L, -1, -1, P2>(d));
    }
}

template <int L>
void diag_chain_sweep(const KArgs &a, const SweepGeom &g, const DiagTabs &t, const DiagChainBufs &buf, cudaStream_t st) {
    DiagChainArgs d{t, buf.div, (size_t)buf.units * a.ncols * 64, buf.dpm, (size_t)a.nb * a.ncols * 64};
    const bool p2 = chain_pow2(a.dxk) && chain_pow2(a.dyk);
    KArgs c = a;
    c.ks = 64;
    ChainBufs b{};
    b.words = buf.words;
    b.epoch = buf.stamps + (a.diag_iter - 1);
    b.unit_n = buf.units;
    for (b.unit_lo = 0; b.unit_lo < a.nb; b.unit_lo += buf.units, ++b.ctr_slot) {
        const int n = std::min(buf.units, a.nb - b.unit_lo);
        k_diag_div<L><<<dim3((a.ncols + 7) / 8, n), 256, 0, st>>>(a, d, b.unit_lo);
        if (p2) k_diag_chain<L, true><<<buf.grid, diag_threads<L>(), 0, st>>>(c, g, b, d);
        else k_diag_chain<L, false><<<buf.grid, diag_threads<L>(), 0, st>>>(c, g, b, d);
    }
    k_diag_velcorr_planes<L><<<dim3((a.ncols + 7) / 8, a.nb), 256, 0, st>>>(a, d);
}

}  // namespace

int diag_chain_levels(int nkk) { return nkk <= 64 ? 2 : (nkk <= 192 ? 6 : 0); }

size_t diag_chain_words(int nii, int njj, int levels) {
    return (size_t)diag_claims(nii - 2, levels) * (njj - 2) * (levels / 2) * KMAX_LEVELS;
}

cudaError_t diag_chain_grid(int levels, int ni, int units, int *grid) {
    const long long claims = (long long)diag_claims(ni, levels) * units;
    if (levels == 2) return chain_grid_of((const void *)k_diag_chain<2, true>, diag_threads<2>(), claims, grid);
    return chain_grid_of((const void *)k_diag_chain<6, true>, diag_threads<6>(), claims, grid);
}

void launch_diag_chain(const KArgs &a, const SweepGeom &g, const DiagTabs &t, const DiagChainBufs &buf, cudaStream_t st) {
    if (buf.levels == 2) diag_chain_sweep<2>(a, g, t, buf, st);
    else diag_chain_sweep<6>(a, g, t, buf, st);
}

}  // namespace gral
