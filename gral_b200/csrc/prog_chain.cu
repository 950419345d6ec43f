// prog_chain.cu -- row chains of the pressure correction and the model-1 momentum sweeps, and the
// launches of the schedule (prog_chain.cuh).
#include <algorithm>
#include <cmath>

#include "prog_chain.cuh"

namespace gral {

namespace {

// A column record of the momentum sweeps: pairs of values per level, [pair][KMAX_LEVELS] float2, so
// that a lane reads its two levels of a pair with one 16-byte load at a constant offset (levels from
// KS up are never touched).  The sweep's direction is known when
// the record is written, so it names the neighbours by what the chain knows of them: cI, cJ are the
// coefficients of the predecessors (i-IS, j) and (i, j-JS), kI and kJ what the successors contribute.
template <int COMP, int SW>
__host__ __device__ constexpr int mom_pairs() { return COMP == COMP_W ? 7 : ((COMP == COMP_V && SW == 8) ? 9 : 10); }
constexpr int MOM_PAIRS_MAX = 10;
// level flags of a record (bits of a float)
enum : unsigned { L_Q = 1u, L_U = 2u, L_X = 4u, L_VEG = 8u };

// What a chain step needs of one level: the sums of DIM in the reference's order, split into the
// parts the predecessors enter (see MomChain::dim).
struct LevelRec {
    float cI, cJ, kI, kJ, t1, t2, t3, w, vdx, K, e0, e1, e2, e3, phi, C, T, P, sI;
    unsigned fl;
};
// pair q of a record as the two values stored at a level
template <int COMP, int SW>
__device__ __forceinline__ float2 rec_pair(const LevelRec &r, int q) {
    const float fl = __uint_as_float(r.fl);
    if (COMP == COMP_W) {
        switch (q) {
            case 0: return make_float2(r.cI, r.cJ);
            case 1: return make_float2(r.kI, r.kJ);
            case 2: return make_float2(r.t1, r.t2);
            case 3: return make_float2(r.t3, r.e0);
            case 4: return make_float2(r.phi, fl);
            case 5: return make_float2(r.C, r.sI);
            default: return make_float2(r.T, r.P);
        }
    }
    switch (q) {
        case 0: return make_float2(r.cI, r.cJ);
        case 1: return make_float2(r.kI, r.kJ);
        case 2: return make_float2(r.t1, r.t2);
        case 3: return make_float2(r.t3, r.w);
        case 4: return make_float2(r.vdx, r.K);
        case 5: return make_float2(r.e0, r.e1);
        case 6: return make_float2(r.e2, r.C);
        case 7: return make_float2(r.phi, fl);
        case 8: return make_float2(r.T, r.P);
        default: return make_float2(r.e3, r.sI);
    }
}
template <int COMP, int SW>
__device__ __forceinline__ void rec_unpair(LevelRec &r, int q, float2 v) {
    if (COMP == COMP_W) {
        switch (q) {
            case 0: r.cI = v.x; r.cJ = v.y; break;
            case 1: r.kI = v.x; r.kJ = v.y; break;
            case 2: r.t1 = v.x; r.t2 = v.y; break;
            case 3: r.t3 = v.x; r.e0 = v.y; break;
            case 4: r.phi = v.x; r.fl = __float_as_uint(v.y); break;
            case 5: r.C = v.x; r.sI = v.y; break;
            default: r.T = v.x; r.P = v.y; break;
        }
        return;
    }
    switch (q) {
        case 0: r.cI = v.x; r.cJ = v.y; break;
        case 1: r.kI = v.x; r.kJ = v.y; break;
        case 2: r.t1 = v.x; r.t2 = v.y; break;
        case 3: r.t3 = v.x; r.w = v.y; break;
        case 4: r.vdx = v.x; r.K = v.y; break;
        case 5: r.e0 = v.x; r.e1 = v.y; break;
        case 6: r.e2 = v.x; r.C = v.y; break;
        case 7: r.phi = v.x; r.fl = __float_as_uint(v.y); break;
        case 8: r.T = v.x; r.P = v.y; break;
        default: r.e3 = v.x; r.sI = v.y; break;
    }
}
template <int COMP>
__host__ __device__ constexpr int tp_pair() { return COMP == COMP_W ? 6 : 8; }   // the pair that holds T and P

// ------------------------------------ coefficients ------------------------------------------

// The record of one level from its coefficients: products and sums that involve only the successors'
// old values are formed here, each where the reference's association order allows it.
template <int COMP, int SW>
__device__ __forceinline__ void level_rec(LevelRec &r, const MomPre &p, int IS, int JS, float sI, float sJ, bool veg,
                                          bool extra) {
    const float cs = IS == 1 ? p.ae : p.aw;          // coefficient of the successor in i
    r.cI = IS == 1 ? p.aw : p.ae;
    r.cJ = JS == 1 ? p.as : p.an;
    r.kI = cs * sI;
    r.kJ = (JS == 1 ? p.an : p.as) * sJ;
    if (SW == 16 && (COMP != COMP_V || veg)) {       // pairs by fused multiply-add (the Vector512 twins)
        if (IS == JS) r.kI = fmaf(cs, sI, r.kJ);     // the pair of both successors
        else r.kI = cs;                              // the successor in i pairs with the predecessor in j
    } else if (IS == -1 && JS == -1) {
        r.kI = r.kI + r.kJ;                          // AW1*PHI + AS1*PHI, the first two of the sum
    }
    r.sI = sI;
    r.t1 = p.t1; r.t2 = p.t2; r.t3 = p.t3;
    if (COMP == COMP_U && SW == 16 && !veg) {        // + fma(DDPX, DYKDZK, t3); adding -0 changes nothing
        r.t2 = fmaf(p.t2, p.hz, p.t3);
        r.t3 = -0.0f;
    }
    r.phi = p.phi; r.C = p.C;
    r.e0 = extra ? p.e0 : 0.0f;
    if (COMP != COMP_W) {
        r.w = p.w; r.vdx = p.vdx;
        r.e1 = extra ? p.e1 : 0.0f;
        r.e2 = extra ? p.e2 : 0.0f;
        if (COMP == COMP_U) {
            r.e3 = extra ? p.e3 : 0.0f;
            r.K = IS == 1 ? (sI - p.phi) * p.hz : (p.phi - sI) * p.hz;      // DUDXE or DUDXW
        } else {
            r.K = JS == 1 ? r.e0 + (sJ - p.phi) * p.hz : (p.phi - sJ) * p.hz;   // e0 + DVDYN, or DVDYS
        }
    }
}

// Coefficients of one model-1 momentum sweep.  Threads map to (column, level) pairs of the tile's level
// range in the slab's memory order, so loads and record stores are contiguous and few lanes idle; then a warp
// per column runs the forward elimination P_k = B_k*T_k, T_k = 1/(A_k - C_k*P_k-1) like the chain's
// recurrences (its influence fades by C*P*T a level; a lane per column, level by level, left seven
// of the block's eight warps waiting).
template <int COMP, int SW>
__global__ void __launch_bounds__(CT_THREADS, 4) k_mom1_terms(KArgs a, SweepGeom g, ChainBufs b) {
    grid_wait();
    __shared__ float sA[CT_COLS][KMAX_LEVELS + 1], sB[CT_COLS][KMAX_LEVELS + 1], sC[CT_COLS][KMAX_LEVELS + 1];
    __shared__ ColCtx s_col[CT_COLS];
    __shared__ float s_ust[CT_COLS];
    __shared__ int s_lo, s_n;
    const Tile t = make_tile(a, g, b, COMP == COMP_V);
    if (!t.ok) return;
    constexpr int NP = mom_pairs<COMP, SW>(), TP = tp_pair<COMP>();
    constexpr int KL = KMAX_LEVELS;
    const int ks = a.ks;
    const SitCtx sc = make_sit(a, t.s);
    const float *F = COMP == COMP_U ? a.uk : (COMP == COMP_V ? a.vk : a.wk);
    constexpr size_t rs = (size_t)NP * KL;     // float2 of a record
    float2 *base = b.rec + ((size_t)t.u * a.ncols + (size_t)(t.i * a.nj2 + t.j0)) * rs;
    // the columns' constants and wall-law friction velocity once per tile
    if (threadIdx.x < t.nc) {
        const ColCtx c = make_col(a, t.i, t.j0 + threadIdx.x);
        s_col[threadIdx.x] = c;
        s_ust[threadIdx.x] = (COMP != COMP_W && (c.fl & F_ADV)) ? ml_ustern<false>(a, make_acc<false>(a, t.s, c.col), c) : 0.0f;
    }
    // the tile's level range: its full items are (column, level in the range), the others only pass
    // the field's value on
    if (threadIdx.x < 32) {
        __syncwarp();
        const bool on = threadIdx.x < t.nc && (s_col[threadIdx.x].fl & F_ADV);
        const int lo = __reduce_min_sync(0xffffffffu, on ? s_col[threadIdx.x].K0 : ks);
        const int hi = __reduce_max_sync(0xffffffffu, on ? s_col[threadIdx.x].VI : -1);
        if (threadIdx.x == 0) { s_lo = hi < 0 ? 0 : lo; s_n = hi < 0 ? 0 : hi - lo + 1; }
    }
    __syncthreads();
    constexpr int PP = COMP == COMP_W ? 4 : 7;             // the pair of phi and the flags
    const int klo = s_lo, nlev = s_n, nrest = ks - nlev;
    auto pass_on = [&](int cl, int k) {
        LevelRec r;
        r.phi = F[make_acc<false>(a, t.s, s_col[cl].col).at(0, k)];
        r.fl = 0u;
        base[(size_t)cl * rs + k + PP * KL] = rec_pair<COMP, SW>(r, PP);
    };
    for (int q = threadIdx.x; q < t.nc * nrest; q += CT_THREADS) {
        const int cl = q / nrest, k = q - cl * nrest;
        pass_on(cl, k < klo ? k : k + nlev);
    }
    for (int q = threadIdx.x; q < t.nc * nlev; q += CT_THREADS) {
        const int cl = q / nlev, k = klo + q - cl * nlev;
        const ColCtx &c = s_col[cl];
        if (!(c.fl & F_ADV) || k < c.K0 || k > c.VI) {     // a level the sweep does not change
            pass_on(cl, k);
            continue;
        }
        const Acc<false> x = make_acc<false>(a, t.s, c.col);
        float2 *rec = base + (size_t)cl * rs + k;
        LevelRec r;
        MomPre p;
        if (COMP == COMP_U) p = u1_pre<false, SW>(a, x, c, sc, k, s_ust + cl);
        else if (COMP == COMP_V) p = v1_pre<false, SW>(a, x, c, sc, k, s_ust + cl);
        else p = w1_pre<false, SW>(a, x, c, sc, k);
        sA[cl][k] = p.A; sB[cl][k] = p.B; sC[cl][k] = p.C;
        const float sI = F[x.at((long long)t.IS * c.nj2, k)], sJ = F[x.at((long long)t.JS, k)];
        const bool veg = (c.fl & F_VEG) != 0, extra = k >= c.kad;
        level_rec<COMP, SW>(r, p, t.IS, t.JS, sI, sJ, veg, extra);
        const int kkm = COMP == COMP_U ? c.kkm_u : (COMP == COMP_V ? c.kkm_v : -1);
        r.fl = (k > c.KK + 1 ? L_Q : 0u) | (k > kkm ? L_U : 0u) | (extra ? L_X : 0u) | (veg ? L_VEG : 0u);
#pragma unroll
        for (int n = 0; n < NP; ++n)
            if (n != TP) rec[n * KL] = rec_pair<COMP, SW>(r, n);
    }
    __syncthreads();
    // forward elimination, a warp per column and two levels per lane, in rounds until no bit changes
    const int lane = threadIdx.x & 31;
    for (int cl = threadIdx.x >> 5; cl < t.nc; cl += CT_THREADS / 32) {
        const ColCtx &c = s_col[cl];
        if (!(c.fl & F_ADV)) continue;
        const int ka = 2 * lane, kb = ka + 1;
        const bool inA = ka >= c.K0 && ka <= c.VI, inB = kb >= c.K0 && kb <= c.VI;
        const float A0 = inA ? sA[cl][ka] : 1.0f, B0 = inA ? sB[cl][ka] : 0.0f;
        const float A1 = inB ? sA[cl][kb] : 1.0f, B1 = inB ? sB[cl][kb] : 0.0f;
        const bool qA = inA && ka > c.KK + 1, qB = inB && kb > c.KK + 1;
        const float C0 = qA ? sC[cl][ka] : 0.0f, C1 = qB ? sC[cl][kb] : 0.0f;
        float T0 = 1.0f / A0, T1 = 1.0f / A1, P0 = B0 * T0, P1 = B1 * T1, in = 0.0f;
        if (qB) { T1 = 1.0f / (A1 - C1 * P0); P1 = B1 * T1; }
        for (;;) {
            const float nx = __shfl_up_sync(0xffffffffu, P1, 1);
            const bool more = __any_sync(0xffffffffu, __float_as_uint(nx) != __float_as_uint(in));
            if (!more) break;
            in = nx;
            T0 = 1.0f / (qA ? A0 - C0 * in : A0); P0 = B0 * T0;
            T1 = 1.0f / (qB ? A1 - C1 * P0 : A1); P1 = B1 * T1;
        }
        float4 *rec = reinterpret_cast<float4 *>(base + (size_t)cl * rs + TP * KL) + lane;
        if (inA || inB) *rec = make_float4(T0, P0, T1, P1);
    }
}

// Divergence term DIV/DTIME of the pressure sweep, [unit][col][KS] (pressure_pre per level).  A thread per
// level of PT_COLS columns, all operands loaded before a column's flags decide anything.
constexpr int PT_COLS = 2;
__global__ void __launch_bounds__(256) k_pressure_terms(KArgs a, ChainBufs b) {
    grid_wait();
    const int u = blockIdx.y, k = threadIdx.x, ks = a.ks;
    if (b.unit_lo + u >= *a.nact) return;
    const int s = a.act[b.unit_lo + u];
    const size_t E = (size_t)a.nj2 * ks;
    float u0[PT_COLS], uE[PT_COLS], v0[PT_COLS], vN[PT_COLS], w0[PT_COLS], wT[PT_COLS];
    uint32_t fl[PT_COLS];
    ColMeta m[PT_COLS];
    int col[PT_COLS];
    bool in[PT_COLS];
#pragma unroll
    for (int q = 0; q < PT_COLS; ++q) {
        const int c = (blockIdx.x * PT_COLS + q) * blockDim.y + threadIdx.y, i = c / a.nj2, j = c - i * a.nj2;
        in[q] = i >= 2 && i <= a.nii - 1 && j >= 2 && j <= a.njj - 1;
        col[q] = in[q] ? c : 2 * a.nj2 + 2;
        const size_t e = ((size_t)s * a.ncols + col[q]) * ks + k;
        u0[q] = a.uk[e]; uE[q] = a.uk[e + E]; v0[q] = a.vk[e]; vN[q] = a.vk[e + ks];
        w0[q] = a.wk[e]; wT[q] = a.wk[e + 1];      // level KS of a column is level 0 of the next
        fl[q] = a.cflags[col[q]];
        m[q] = a.meta[col[q]];
    }
    const float DXK = a.dxk, DYK = a.dyk, AREA = a.areaxy, dz = a.dzk[k], dt = a.sit[s].dtime, rdt = a.sit[s].rdtime;
    const bool active = a.sit[s].active != 0;
    float *out = reinterpret_cast<float *>(b.rec) + (size_t)u * a.ncols * ks + k;
#pragma unroll
    for (int q = 0; q < PT_COLS; ++q) {
        if (!in[q] || !active || !(fl[q] & F_ADV) || k <= m[q].kkart || k > m[q].vi) continue;
        const float h = (u0[q] - uE[q]) * DYK * dz + (v0[q] - vN[q]) * DXK * dz;
        const float DIV = (k > m[q].kkart + 1) ? h + (w0[q] - wT[q]) * AREA : h - wT[q] * AREA;
        out[(size_t)col[q] * ks] = div_by(DIV, dt, rdt);
    }
}

// Forward elimination of the pressure sweep, T = 1/(APP - ATP*P) and P = ABP*T from VerticalIndex
// down to KKART+1, per i-direction: [dir][col][KS] {T, P}, zero on the levels the sweep does not
// change.  It depends on the grid alone, so it is built once per load.  A column starts from the P
// that its row-carry writer (rcw) left at VerticalIndex+1, zero without one.  Every thread takes a
// column and passes are repeated until one changes nothing; the start's influence fades by P*P a
// level, so two or three passes suffice.  A pass after the first only recomputes the top level and
// stops there if it is unchanged.
__global__ void __launch_bounds__(128) k_pressure_tab(KArgs a, float2 *tab, int *changed, int pass) {
    if (pass > 0 && changed[pass - 1] == 0) return;
    const int dir = blockIdx.y, ks = a.ks;
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= a.ncols) return;
    const int i = col / a.nj2, j = col - i * a.nj2;
    if (i < 2 || i > a.nii - 1 || j < 2 || j > a.njj - 1 || !(a.cflags[col] & F_ADV)) return;
    const ColMeta m = a.meta[col];
    float2 *tp = tab + ((size_t)dir * a.ncols + col) * ks;
    const short2 w = a.rcw[col];
    const int wi = dir == 0 ? w.x : w.y;
    float P = 0.0f;
    if (wi >= 0) P = *(volatile float *)&tab[((size_t)dir * a.ncols + (size_t)wi * a.nj2 + j) * ks + m.vi + 1].y;
    for (int k = m.vi; k > m.kkart; --k) {
        const float T = 1.0f / (a.app[k] - a.atp[k] * P);
        P = a.abp[k] * T;
        if (pass > 0 && __float_as_uint(T) == __float_as_uint(tp[k].x)) return;   // the rest follows from T
        tp[k] = make_float2(T, P);
        if (k == m.vi) changed[pass] = 1;
    }
}

// ------------------------------------ row chains --------------------------------------------

// Model-1 momentum: record of one column in registers (two levels per lane) and the step, for one
// sweep direction (branches on it would stall the chain).
template <int COMP, int SW, int IS, int JS>
struct MomChain {
    static constexpr int NV = 1, NJ = 1, NF = 1;    // see run_chain
    static constexpr int NP = mom_pairs<COMP, SW>();
    struct Rec {
        float4 f[NP];      // {x(2l), y(2l), x(2l+1), y(2l+1)} of each pair
    };
    struct Val {
        float2 v[NV];
    };
    float relax;
    float2 hz;
    float *F[NF];
    const float4 *rec;     // this lane's part of the next record to load
    const char *line;      // this lane's 128-byte line of the next record to ask into L2
    bool on0, on1;         // whether the line exists (and the one 32 lines on)

    __device__ __forceinline__ void init(const KArgs &a, int lane) {
        relax = a.relax;
        F[0] = COMP == COMP_U ? a.uk : (COMP == COMP_V ? a.vk : a.wk);
        const float face = COMP == COMP_U ? a.dyk : a.dxk;
        const int l = min(lane, a.ks / 2 - 1);
        hz = make_float2(face * a.dzk[2 * l], face * a.dzk[2 * l + 1]);
        on0 = (lane & 3) * 16 < a.ks && (lane >> 2) < NP;
        on1 = (lane & 3) * 16 < a.ks && (lane >> 2) + 8 < NP;
    }
    int step_rec;          // float4 to this warp's next record
    template <int M>
    __device__ __forceinline__ void begin(const KArgs &a, const ChainBufs &b, int u, int, int col, int lane) {
        step_rec = JS * M * (NP * (KMAX_LEVELS / 2));
        const float2 *p = b.rec + ((size_t)u * a.ncols + col) * (NP * KMAX_LEVELS);
        rec = reinterpret_cast<const float4 *>(p) + min(lane, a.ks / 2 - 1);
        line = reinterpret_cast<const char *>(p) + 128 * lane;
    }
    // asks the next column's record into L2; loads the next column's record
    __device__ __forceinline__ void ahead(bool on) {
        l2_ahead(line, on && on0);
        if (NP > 8) l2_ahead(line + 4096, on && on1);
        line += step_rec * 16;
    }
    __device__ __forceinline__ void load(Rec &r) {
#pragma unroll
        for (int q = 0; q < NP; ++q) r.f[q] = __ldcg(rec + q * (KMAX_LEVELS / 2));
        rec += step_rec;
    }
    // the field's values of a column that this sweep does not change
    __device__ __forceinline__ Val still(const KArgs &a, size_t base, int lane) const {
        Val o;
        o.v[0] = __ldcg(reinterpret_cast<const float2 *>(F[0] + base) + min(lane, a.ks / 2 - 1));
        return o;
    }
    // DIM of one level: the neighbour products and sources in the reference's association order
    __device__ __forceinline__ float dim(const LevelRec &r, float hzk, float vI, float vJ) const {
        float D;
        const float pJ = r.cJ * vJ;
        float Df = 0.0f;
        if (SW == 16) {   // U-prognostic-microscale_1_Vec512.cs:399-421
            float S1, S2;
            if (IS == JS) {
                S1 = fmaf(r.cI, vI, pJ);
                S2 = r.kI;                                    // a + b == b + a: either pair may come first
            } else {
                S1 = fmaf(r.cI, vI, r.kJ);
                S2 = fmaf(r.kI, r.sI, pJ);
            }
            Df = S1 + S2;
        }
        if (SW == 8 || COMP == COMP_V) {
            const float pI = r.cI * vI;
            if (IS == 1) D = (JS == 1) ? pI + pJ + r.kI + r.kJ : pI + r.kJ + r.kI + pJ;
            else D = (JS == 1) ? r.kI + pJ + pI + r.kJ : r.kI + pI + pJ;
            if (SW == 16 && (r.fl & L_VEG)) D = Df;
        } else {
            D = Df;
        }
        D = D + r.t1 + r.t2;
        if (COMP == COMP_W) {
            D = D - r.t3;
            add_if(D, D, r.e0, r.fl & L_X);
            return D;
        }
        D = D + r.t3 - r.w;
        float X;
        if (COMP == COMP_U) {
            const float d = (IS == 1) ? r.K - (r.phi - vI) * hzk : (vI - r.phi) * hzk - r.K;
            X = d + r.e0 - r.e1 + r.e2 - r.e3;
        } else {
            const float d = (JS == 1) ? r.K - (r.phi - vJ) * hzk : r.e0 + (vJ - r.phi) * hzk - r.K;
            X = d + r.e1 - r.e2;
        }
        add_if(D, D, r.vdx * X, r.fl & L_X);
        return D;
    }
    __device__ __forceinline__ Val step(const Rec &rc, const Val &vI, const float2 (&vJ)[NJ]) const {
        LevelRec A, B;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            rec_unpair<COMP, SW>(A, q, make_float2(rc.f[q].x, rc.f[q].y));
            rec_unpair<COMP, SW>(B, q, make_float2(rc.f[q].z, rc.f[q].w));
        }
        const float Da = dim(A, hz.x, vI.v[0].x, vJ[0].x), Db = dim(B, hz.y, vI.v[0].y, vJ[0].y);
        // Q_k = D_k*T_k up to KKART+1, above it Q_k = (D_k + C_k*Q_k-1)*T_k
        const unsigned qA = A.fl & L_Q, qB = B.fl & L_Q, uA = A.fl & L_U, uB = B.fl & L_U;
        float Qa = Da * A.T, Qb = Db * B.T, inQ = 0.0f, inU = 0.0f;
        mul_if(Qb, Db + B.C * Qa, B.T, qB);
        auto up = [&]() {
            mul_if(Qa, Da + A.C * inQ, A.T, qA);
            mul_if(Qb, Db + B.C * Qa, B.T, qB);
        };
        // relaxed back-substitution from VerticalIndex down; the other levels keep their value
        float va = A.phi, vb = B.phi;
        auto down = [&]() {
            add_if(vb, B.phi, relax * (B.P * inU + Qb - B.phi), uB);
            add_if(va, A.phi, relax * (A.P * vb + Qa - A.phi), uA);
        };
        // while Q settles, the back-substitution already iterates on the Q of the round before: its
        // chain runs beside Q's, and little is left for it once Q is final
#pragma unroll
        for (int n = 0; n < ROUNDS_MOM; ++n) {
            inU = __shfl_down_sync(0xffffffffu, va, 1);
            inQ = __shfl_up_sync(0xffffffffu, Qb, 1);
            down();
            up();
        }
        for (;;) {
            const float nU = __shfl_down_sync(0xffffffffu, va, 1), nQ = __shfl_up_sync(0xffffffffu, Qb, 1);
            const bool more = __any_sync(0xffffffffu, differ(nQ, inQ));
            inU = nU; inQ = nQ;
            down();
            if (!more) break;      // Q is final and has been used
            up();
        }
        for (;;) {
            const float nU = __shfl_down_sync(0xffffffffu, va, 1);
            const bool more = __any_sync(0xffffffffu, differ(nU, inU));
            inU = nU;
            down();
            if (!more) break;
        }
        Val o;
        o.v[0] = make_float2(va, vb);
        return o;
    }
};

// Pressure correction (PrognosticFlowfield.cs:804-901).  Values handed on: DPM and the row carry's Q
// (the reference's QIMP buffer lives per sweep row j and is not cleared between columns, :865-868:
// a column's Q starts from what an earlier column of its row j left at VerticalIndex+1), which
// therefore travels along i with the DPM.  DPMNEW and the residual follow in the velocity correction.
template <int IS, int JS, bool P2>
struct PressChain {
    static constexpr int NV = 2, NJ = 1, NF = 1;
    struct Rec {
        float4 tp;      // {T, P} of the two levels
        float2 d;       // DIV/DTIME
    };
    struct Val {
        float2 v[NV];
    };
    float2 atp, dz;
    float dxk, dyk, rx, ry;
    float *F[NF];
    const float2 *div;
    const float4 *tab;
    const char *line;
    long long step_line;
    int hstep;
    bool on0;

    __device__ __forceinline__ void init(const KArgs &a, int lane) {
        F[0] = a.dpm;
        dxk = a.dxk; dyk = a.dyk;
        rx = 1.0f / dxk; ry = 1.0f / dyk;
        const int l = min(lane, a.ks / 2 - 1);
        atp = make_float2(a.atp[2 * l], a.atp[2 * l + 1]);
        dz = make_float2(a.dzk[2 * l], a.dzk[2 * l + 1]);
    }
    template <int M>
    __device__ __forceinline__ void begin(const KArgs &a, const ChainBufs &b, int u, int, int col, int lane) {
        hstep = JS * M * (a.ks / 2);
        const int l = min(lane, a.ks / 2 - 1);
        const float *d = reinterpret_cast<const float *>(b.rec) + ((size_t)u * a.ncols + col) * a.ks;
        const float2 *t = b.ptab + ((size_t)(IS == 1 ? 0 : 1) * a.ncols + col) * a.ks;
        div = reinterpret_cast<const float2 *>(d) + l;
        tab = reinterpret_cast<const float4 *>(t) + l;
        // lines of 128 bytes of the two runs, lanes 0-3 and 4-7 (a run that does not start on a line leaves the
        // last bit of it to the load)
        line = lane < 4 ? reinterpret_cast<const char *>(d) + 128 * lane : reinterpret_cast<const char *>(t) + 128 * (lane - 4);
        on0 = lane < 4 ? 128 * lane < a.ks * 4 : (lane < 8 && 128 * (lane - 4) < a.ks * 8);
        step_line = (long long)JS * M * a.ks * (lane < 4 ? 4 : 8);
    }
    __device__ __forceinline__ void ahead(bool on) {
        l2_ahead(line, on && on0);
        line += step_line;
    }
    __device__ __forceinline__ void load(Rec &r) {
        r.tp = __ldcg(tab);
        r.d = __ldcg(div);
        tab += hstep;
        div += hstep;
    }
    // outside the sweep DPM is zero, and a sweep row's carry starts from zero
    __device__ __forceinline__ Val still(const KArgs &, size_t, int) const {
        Val o;
        o.v[0] = o.v[1] = make_float2(0.0f, 0.0f);
        return o;
    }
    // pressure_post_v of one level
    __device__ __forceinline__ float dim(float t0, float dzk, float pi, float pj) const {
        const float si = (IS == 1) ? (pi + 0.0f) : (0.0f + pi);
        const float sj = (JS == 1) ? (pj - 0.0f) : (0.0f - pj);
        // x / 2^n == x * 2^-n in every rounding, so power-of-two spacings (P2) need no division
        const float qi = P2 ? si * rx : si / dxk, qj = P2 ? sj * ry : sj / dyk;
        return t0 + qi * dyk * dzk + qj * dxk * dzk;
    }
    __device__ __forceinline__ Val step(const Rec &r, const Val &vI, const float2 (&vJ)[NJ]) const {
        const float Ta = r.tp.x, Pa = r.tp.y, Tb = r.tp.z, Pb = r.tp.w;
        const unsigned lA = Ta != 0.0f, lB = Tb != 0.0f;
        const float Da = dim(r.d.x, dz.x, vI.v[0].x, vJ[0].x), Db = dim(r.d.y, dz.y, vI.v[0].y, vJ[0].y);
        // Q downwards from the carry at VerticalIndex+1
        float Qa = vI.v[1].x, Qb = vI.v[1].y, inQ = 0.0f, inD = 0.0f;
        mul_if(Qb, Db, Tb, lB);
        mul_if(Qa, atp.x * Qb + Da, Ta, lA);
        auto down = [&]() {
            mul_if(Qb, atp.y * inQ + Db, Tb, lB);
            mul_if(Qa, atp.x * Qb + Da, Ta, lA);
        };
        // DPM upwards from the zero at KKART
        float da = 0.0f, db = 0.0f;
        auto up = [&]() {
            add_if(da, Pa * inD, Qa, lA);
            add_if(db, Pb * da, Qb, lB);
        };
        // the two recurrences side by side, as in the momentum step
#pragma unroll
        for (int n = 0; n < ROUNDS_PRESS; ++n) {
            inD = __shfl_up_sync(0xffffffffu, db, 1);
            inQ = __shfl_down_sync(0xffffffffu, Qa, 1);
            up();
            down();
        }
        for (;;) {
            const float nD = __shfl_up_sync(0xffffffffu, db, 1), nQ = __shfl_down_sync(0xffffffffu, Qa, 1);
            const bool more = __any_sync(0xffffffffu, differ(nQ, inQ));
            inD = nD; inQ = nQ;
            up();
            if (!more) break;      // Q is final and has been used
            down();
        }
        for (;;) {
            const float nD = __shfl_up_sync(0xffffffffu, db, 1);
            const bool more = __any_sync(0xffffffffu, differ(nD, inD));
            inD = nD;
            up();
            if (!more) break;
        }
        Val o;
        o.v[0] = make_float2(da, db);
        o.v[1] = make_float2(Qa, Qb);
        return o;
    }
};

// The kernels take the sweep's direction from the iteration count and run the code built for it.
template <int COMP, int SW>
__global__ void __cluster_dims__(CH_CL, 1, 1) __launch_bounds__(CH_THREADS, 2) k_mom_chain(KArgs a, SweepGeom g, ChainBufs b) {
    __shared__ ChainSmem<CH_SR, 1> sm;
    constexpr int PH = COMP == COMP_U ? PH_U : (COMP == COMP_V ? PH_V : PH_W);
    constexpr int SR = CH_SR, M = CH_M, CL = CH_CL;
    for (unsigned q = threadIdx.x; q < sizeof(sm.ring) / 8; q += CH_THREADS) sm.ring[q] = 0ull;
    int is, js;
    chain_dir(*a.it_global, is, js);
    if (COMP == COMP_V) { is = -is; js = -js; }     // model-1 V sweeps with (-IS,-JS)
    if (is == 1) {
        if (js == 1) run_chain<MomChain<COMP, SW, 1, 1>, PH, SR, M, CL, 1, 1>(a, g, b, sm);
        else run_chain<MomChain<COMP, SW, 1, -1>, PH, SR, M, CL, 1, -1>(a, g, b, sm);
    } else {
        if (js == 1) run_chain<MomChain<COMP, SW, -1, 1>, PH, SR, M, CL, -1, 1>(a, g, b, sm);
        else run_chain<MomChain<COMP, SW, -1, -1>, PH, SR, M, CL, -1, -1>(a, g, b, sm);
    }
}

template <bool P2>
__global__ void __cluster_dims__(CH_CL, 1, 1) __launch_bounds__(CH_THREADS, 2) k_pressure_chain(KArgs a, SweepGeom g, ChainBufs b) {
    __shared__ ChainSmem<CH_SR, 2> sm;
    constexpr int PH = PH_PRESSURE, SR = CH_SR, M = CH_M, CL = CH_CL;
    for (unsigned q = threadIdx.x; q < sizeof(sm.ring) / 8; q += CH_THREADS) sm.ring[q] = 0ull;
    int is, js;
    chain_dir(*a.it_global, is, js);
    if (is == 1) {
        if (js == 1) run_chain<PressChain<1, 1, P2>, PH, SR, M, CL, 1, 1>(a, g, b, sm);
        else run_chain<PressChain<1, -1, P2>, PH, SR, M, CL, 1, -1>(a, g, b, sm);
    } else {
        if (js == 1) run_chain<PressChain<-1, 1, P2>, PH, SR, M, CL, -1, 1>(a, g, b, sm);
        else run_chain<PressChain<-1, -1, P2>, PH, SR, M, CL, -1, -1>(a, g, b, sm);
    }
}


KFn chain_kernel(int kind, const KArgs &a) {
    const bool w = a.simd == 16;
    if (kind != PH_PRESSURE && a.model != 1) return chain_scalar_kernel(kind, a.model);
    switch (kind) {
        case PH_PRESSURE: return (chain_pow2(a.dxk) && chain_pow2(a.dyk)) ? k_pressure_chain<true> : k_pressure_chain<false>;
        case PH_U: return w ? k_mom_chain<COMP_U, 16> : k_mom_chain<COMP_U, 8>;
        case PH_V: return w ? k_mom_chain<COMP_V, 16> : k_mom_chain<COMP_V, 8>;
        default: return w ? k_mom_chain<COMP_W, 16> : k_mom_chain<COMP_W, 8>;
    }
}

KFn terms_kernel(int kind, const KArgs &a) {
    const bool w = a.simd == 16;
    if (a.model != 1) return chain_scalar_terms(kind, a.model);
    switch (kind) {
        case PH_U: return w ? k_mom1_terms<COMP_U, 16> : k_mom1_terms<COMP_U, 8>;
        case PH_V: return w ? k_mom1_terms<COMP_V, 16> : k_mom1_terms<COMP_V, 8>;
        default: return w ? k_mom1_terms<COMP_W, 16> : k_mom1_terms<COMP_W, 8>;
    }
}

}  // namespace

size_t chain_record_bytes(int model) {
    return (size_t)(model == 1 ? MOM_PAIRS_MAX : chain_scalar_pairs(model)) * KMAX_LEVELS * sizeof(float2);
}

size_t chain_unit_words(int nii, int njj) {
    return (size_t)chain_claims(nii - 2) * (njj - 2) * 2 * KMAX_LEVELS;   // two values a level at most
}

int chain_claims(int ni) { return (ni + CH_SR * CH_CL - 1) / (CH_SR * CH_CL); }

bool chain_pow2(float x) {
    int e;
    return std::frexp(x, &e) == 0.5f && e > -100 && e < 100;
}

cudaError_t chain_grid(int kind, const KArgs &a, long long claims, int *grid) {
    return chain_grid_of((const void *)chain_kernel(kind, a), CH_THREADS, claims, grid);
}

cudaError_t chain_grid_of(const void *kernel, int threads, long long claims, int *grid) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CH_CL);
    cfg.blockDim = dim3(threads);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CH_CL;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (e != cudaSuccess) return e;
    *grid = CH_CL * (int)std::max<long long>(1, std::min<long long>(std::max(1, clusters), claims));
    return cudaSuccess;
}

void launch_chain(int kind, const KArgs &a, const SweepGeom &g, const ChainBufs &bufs, int grid, cudaStream_t st) {
    if (g.ni <= 0 || g.nj <= 0) return;
    ChainBufs b = bufs;
    b.ctr_slot = 0;
    for (b.unit_lo = 0; b.unit_lo < a.nb; b.unit_lo += bufs.unit_n, ++b.ctr_slot) {
        const int n = std::min(bufs.unit_n, a.nb - b.unit_lo);
        const long long tiles = (long long)n * g.ni * ((g.nj + CT_COLS - 1) / CT_COLS);
        if (kind == PH_PRESSURE) {
            const int rows = std::max(1, 256 / a.ks), per = rows * PT_COLS;
            launch_after(k_pressure_terms, dim3((a.ncols + per - 1) / per, n), dim3(a.ks, rows), st, a, b);
        } else {
            launch_after(terms_kernel(kind, a), (unsigned)tiles, CT_THREADS, st, a, g, b);
        }
        chain_kernel(kind, a)<<<grid, CH_THREADS, 0, st>>>(a, g, b);
    }
}

void launch_pressure_tab(const KArgs &a, float2 *tab, int *changed, int first, int passes, cudaStream_t st) {
    for (int p = first; p < first + passes; ++p)
        k_pressure_tab<<<dim3((a.ncols + 127) / 128, 2), 128, 0, st>>>(a, tab, changed, p);
}

}  // namespace gral
