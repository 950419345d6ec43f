// prog_chain_scalar.cu -- row chains (prog_chain.cuh) of turbulence models 0 and 2: U, V, W and the
// k-eps transport.
//
// Their recurrences divide by A - C*P at every level (U-prognostic-microscale_2.cs:247-256).  The
// divisor does not depend on the sweep, so its reciprocal is in the record and a quotient is the
// correctly rounded form of prog_quot.cuh (5 dependent operations instead of a division); a column
// in which a dividend, quotient or divisor leaves that form's range is redone with divisions.
#include "prog_chain.cuh"

namespace gral {

namespace {

// Values of a record level, two to a pair.  W has no T3 and keeps its whole viscous increment in W;
// model 0 has no viscous terms (the values from VDX on).
enum : int { S_CI, S_CJ, S_KI, S_KJ, S_T1, S_T2, S_T3, S_W, S_PHI, S_FL, S_C, S_DEN, S_Y, S_P, S_VDX, S_K, S_E0, S_E1, S_E2, S_E3, S_N };
template <int MODEL, int COMP>
__host__ __device__ constexpr int scal_pairs() { return (MODEL == 2 && COMP != COMP_W) ? S_N / 2 : (S_P + 1) / 2; }
// model-0 W: P, the divisor and its reciprocal are doubles, one to a pair
enum : int { Z_CI, Z_CJ, Z_KI, Z_KJ, Z_T1, Z_T2, Z_PHI, Z_FL, Z_C, Z_A, Z_N, Z_DEN = 5, Z_Y, Z_P, Z_PAIRS };
// k-eps: neighbour coefficients, the successors' part for TURB (1) and TDISS (2), sources, recurrences
enum : int { T_CI, T_CJ, T_KI1, T_KJ1, T_KI2, T_KJ2, T_T1, T_T2, T_T3, T_S1, T_S2, T_FL, T_C1, T_DEN1, T_Y1, T_P1, T_C2, T_DEN2, T_Y2, T_P2, T_K, T_E, T_N };
constexpr int TKE_PAIRS = T_N / 2;

// level flags: Q recurrence, updated, viscous terms, divisor outside the quotient's range; Q in use: the level
// is updated or, from KKART+1 on (which a taller neighbour keeps from being updated), the next one's Q reads it
enum : unsigned { L_Q = 1u, L_U = 2u, L_X = 4u, L_D = 8u, L_R = 16u };
// a level's quot_worst as far as its Q is in use, with the divisor's flag on top
__device__ __forceinline__ unsigned in_use(unsigned w, unsigned fl) { return (fl & L_R) ? (w | (fl & L_D) << 28) : 0u; }

template <int I>
__device__ __forceinline__ float lev_a(const float4 *f) { return (I & 1) ? f[I / 2].y : f[I / 2].x; }
template <int I>
__device__ __forceinline__ float lev_b(const float4 *f) { return (I & 1) ? f[I / 2].w : f[I / 2].z; }

// ------------------------------------ coefficients ------------------------------------------

// Tile prologue: the columns' constants in shared memory and the tile's level range.
struct TileSmem {
    ColCtx col[CT_COLS];
    int lo, n;
};
__device__ __forceinline__ void tile_columns(const KArgs &a, const Tile &t, TileSmem &sm) {
    if (threadIdx.x < t.nc) sm.col[threadIdx.x] = make_col(a, t.i, t.j0 + threadIdx.x);
    if (threadIdx.x < 32) {
        __syncwarp();
        const bool on = threadIdx.x < t.nc && (sm.col[threadIdx.x].fl & F_ADV);
        const int lo = __reduce_min_sync(0xffffffffu, on ? sm.col[threadIdx.x].K0 : a.ks);
        const int hi = __reduce_max_sync(0xffffffffu, on ? sm.col[threadIdx.x].VI : -1);
        if (threadIdx.x == 0) { sm.lo = hi < 0 ? 0 : lo; sm.n = hi < 0 ? 0 : hi - lo + 1; }
    }
    __syncthreads();
}
// Calls rest(column of the tile, level) for the levels no column of the tile sweeps (they only pass the
// field's value on) and full(column, level) for the range.
template <class Full, class Rest>
__device__ __forceinline__ void tile_items(const KArgs &a, const Tile &t, const TileSmem &sm, Full &&full, Rest &&rest) {
    const int klo = sm.lo, nlev = sm.n, nrest = a.ks - nlev;
    for (int q = threadIdx.x; q < t.nc * nrest; q += CT_THREADS) {
        const int cl = q / nrest, k = q - cl * nrest;
        rest(cl, k < klo ? k : k + nlev);
    }
    for (int q = threadIdx.x; q < t.nc * nlev; q += CT_THREADS) {
        const int cl = q / nlev, k = klo + q - cl * nlev;
        const ColCtx &c = sm.col[cl];
        if (!(c.fl & F_ADV) || k < c.K0 || k > c.VI) rest(cl, k);
        else full(cl, k);
    }
}

// Divisors and P of one column's forward elimination on a warp (two levels per lane), in rounds until no
// bit changes: den_k = A_k - C_k*P_k-1 above KKART+1, A_k up to it; P_k = B_k/den_k.
template <class T>
struct Elim {
    T den0, den1, P0, P1;
};
template <class T>
__device__ __forceinline__ Elim<T> eliminate(float A0, float B0, float C0, bool q0, float A1, float B1, float C1, bool q1) {
    Elim<T> e;
    // up to KKART+1 the quotient is a float's, also in the double routine
    const T f0 = (T)(B0 / A0), f1 = (T)(B1 / A1);
    T in = (T)0;
    e.den0 = (T)A0; e.den1 = (T)A1;
    e.P0 = f0; e.P1 = f1;
    for (bool first = true;; first = false) {
        const T nx = __shfl_up_sync(0xffffffffu, e.P1, 1);
        const bool more = __any_sync(0xffffffffu, sizeof(T) == 4 ? __float_as_uint((float)nx) != __float_as_uint((float)in)
                                                                 : __double_as_longlong((double)nx) != __double_as_longlong((double)in));
        if (!more && !first) break;
        in = nx;
        if (q0) { e.den0 = (T)A0 - (T)C0 * in; e.P0 = (T)B0 / e.den0; }
        if (q1) { e.den1 = (T)A1 - (T)C1 * e.P0; e.P1 = (T)B1 / e.den1; }
    }
    return e;
}

// the level's neighbour terms as the chain takes them: predecessors by coefficient, successors by product
__device__ __forceinline__ void neighbours(const MomPre &p, int IS, int JS, float sI, float sJ, float &cI, float &cJ,
                                           float &kI, float &kJ) {
    cI = IS == 1 ? p.aw : p.ae;
    cJ = JS == 1 ? p.as : p.an;
    kI = (IS == 1 ? p.ae : p.aw) * sI;
    kJ = (JS == 1 ? p.an : p.as) * sJ;
    if (IS == -1 && JS == -1) kI = kI + kJ;          // AW1*PHI + AS1*PHI, the first two of the sum
}

template <int MODEL, int COMP>
__global__ void __launch_bounds__(CT_THREADS, 3) k_scal_terms(KArgs a, SweepGeom g, ChainBufs b) {
    grid_wait();
    constexpr bool Z = MODEL == 0 && COMP == COMP_W, DIFF = MODEL == 2;
    constexpr int NP = Z ? (int)Z_PAIRS : scal_pairs<MODEL, COMP>(), KL = KMAX_LEVELS;
    __shared__ float sA[CT_COLS][KL + 1], sB[CT_COLS][KL + 1], sC[CT_COLS][KL + 1];
    __shared__ TileSmem sm;
    const Tile t = make_tile(a, g, b, false);
    if (!t.ok) return;
    const SitCtx sc = make_sit(a, t.s);
    const float *F = COMP == COMP_U ? a.uk : (COMP == COMP_V ? a.vk : a.wk);
    constexpr size_t rs = (size_t)NP * KL;     // float2 of a record
    float2 *base = b.rec + ((size_t)t.u * a.ncols + (size_t)(t.i * a.nj2 + t.j0)) * rs;
    tile_columns(a, t, sm);
    auto full = [&](int cl, int k) {
        const ColCtx &c = sm.col[cl];
        const Acc<false> x = make_acc<false>(a, t.s, c.col);
        float2 *rec = base + (size_t)cl * rs + k;
        const MomPre p = [&] {
            if constexpr (COMP == COMP_W) return w_scalar_pre<DIFF, false>(a, x, c, sc, k);
            else return uv_scalar_pre<DIFF, COMP, false>(a, x, c, sc, k);
        }();
        sA[cl][k] = p.A; sB[cl][k] = p.B; sC[cl][k] = p.C;
        const float sI = F[x.at((long long)t.IS * c.nj2, k)], sJ = F[x.at((long long)t.JS, k)];
        float cI, cJ, kI, kJ;
        neighbours(p, t.IS, t.JS, sI, sJ, cI, cJ, kI, kJ);
        const int kkm = COMP == COMP_U ? c.kkm_u : (COMP == COMP_V ? c.kkm_v : -1);
        const float fl = __uint_as_float((k > c.KK + 1 ? L_Q : 0u) | (k > kkm ? L_U : 0u) | ((DIFF && k > c.KK + 1) ? L_X : 0u) |
                                         ((k > c.KK || k > kkm) ? L_R : 0u));
        auto put = [&](int q, float v0, float v1) { rec[q * KL] = make_float2(v0, v1); };
        put(S_CI / 2, cI, cJ);
        put(S_KI / 2, kI, kJ);
        put(S_T1 / 2, p.t1, p.t2);
        if constexpr (Z) {
            put(Z_PHI / 2, p.phi, fl);
            put(Z_C / 2, p.C, p.A);
        } else {
            if constexpr (COMP == COMP_W) put(S_T3 / 2, 0.0f, p.e0);
            else put(S_T3 / 2, p.t3, p.w);
            put(S_PHI / 2, p.phi, fl);
            if constexpr (DIFF && COMP != COMP_W) {
                float K;      // the viscous difference on the successor's side
                if (COMP == COMP_U) K = t.IS == 1 ? (sI - p.phi) * p.hz : (p.phi - sI) * p.hz;
                else K = t.JS == 1 ? p.e0 + (sJ - p.phi) * p.hz : (p.phi - sJ) * p.hz;
                put(S_VDX / 2, p.vdx, K);
                put(S_E0 / 2, p.e0, p.e1);
                put(S_E2 / 2, p.e2, COMP == COMP_U ? p.e3 : 0.0f);
            }
        }
    };
    auto rest = [&](int cl, int k) {
        base[(size_t)cl * rs + k + (Z ? Z_PHI / 2 : S_PHI / 2) * KL] =
            make_float2(F[make_acc<false>(a, t.s, sm.col[cl].col).at(0, k)], __uint_as_float(0u));
    };
    tile_items(a, t, sm, full, rest);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int cl = threadIdx.x >> 5; cl < t.nc; cl += CT_THREADS / 32) {
        const ColCtx &c = sm.col[cl];
        if (!(c.fl & F_ADV)) continue;
        const int ka = 2 * lane, kb = ka + 1;
        const bool inA = ka >= c.K0 && ka <= c.VI, inB = kb >= c.K0 && kb <= c.VI;
        const bool qA = inA && ka > c.KK + 1, qB = inB && kb > c.KK + 1;
        const float A0 = inA ? sA[cl][ka] : 1.0f, B0 = inA ? sB[cl][ka] : 0.0f, C0 = qA ? sC[cl][ka] : 0.0f;
        const float A1 = inB ? sA[cl][kb] : 1.0f, B1 = inB ? sB[cl][kb] : 0.0f, C1 = qB ? sC[cl][kb] : 0.0f;
        float4 *rec = reinterpret_cast<float4 *>(base + (size_t)cl * rs) + lane;
        constexpr int H = KL / 2;
        if constexpr (Z) {
            const Elim<double> e = eliminate<double>(A0, B0, C0, qA, A1, B1, C1, qB);
            if (inA || inB) {
                auto two = [&](int q, double v0, double v1) {
                    rec[q * H] = make_float4(__int_as_float(__double2loint(v0)), __int_as_float(__double2hiint(v0)),
                                             __int_as_float(__double2loint(v1)), __int_as_float(__double2hiint(v1)));
                };
                two(Z_DEN, e.den0, e.den1);
                two(Z_Y, 1.0 / e.den0, 1.0 / e.den1);
                two(Z_P, e.P0, e.P1);
            }
        } else {
            const Elim<float> e = eliminate<float>(A0, B0, C0, qA, A1, B1, C1, qB);
            if (inA || inB) {
                // C and the divisor, the reciprocal and P; the divisor's range goes into the flags
                rec[(S_C / 2) * H] = make_float4(C0, e.den0, C1, e.den1);
                rec[(S_Y / 2) * H] = make_float4(1.0f / e.den0, e.P0, 1.0f / e.den1, e.P1);
                float4 f = rec[(S_PHI / 2) * H];
                if (inA && odd_divisor(e.den0)) f.y = __uint_as_float(__float_as_uint(f.y) | L_D);
                if (inB && odd_divisor(e.den1)) f.w = __uint_as_float(__float_as_uint(f.w) | L_D);
                if ((inA && odd_divisor(e.den0)) || (inB && odd_divisor(e.den1))) rec[(S_PHI / 2) * H] = f;
            }
        }
    }
}

// Coefficients of the k-eps sweep.  A level with a wall function (and one at or below KKART) is a
// constant of the sweep: its value goes into the record and nothing updates it.
__global__ void __launch_bounds__(CT_THREADS, 2) k_tke_terms(KArgs a, SweepGeom g, ChainBufs b) {
    grid_wait();
    constexpr int KL = KMAX_LEVELS;
    __shared__ float sm_f[5][CT_COLS][KL + 1];     // A, B1, C1, B2, C2
    __shared__ TileSmem sm;
    const Tile t = make_tile(a, g, b, false);
    if (!t.ok) return;
    const SitCtx sc = make_sit(a, t.s);
    constexpr size_t rs = (size_t)TKE_PAIRS * KL;
    float2 *base = b.rec + ((size_t)t.u * a.ncols + (size_t)(t.i * a.nj2 + t.j0)) * rs;
    tile_columns(a, t, sm);
    auto full = [&](int cl, int k) {
        const ColCtx &c = sm.col[cl];
        const Acc<false> x = make_acc<false>(a, t.s, c.col);
        float2 *rec = base + (size_t)cl * rs + k;
        const KePre p = tke_pre<false>(a, x, c, sc, k);
        sm_f[0][cl][k] = p.A; sm_f[1][cl][k] = p.B1; sm_f[2][cl][k] = p.C1; sm_f[3][cl][k] = p.B2; sm_f[4][cl][k] = p.C2;
        const long long dI = (long long)t.IS * c.nj2, dJ = t.JS;
        const float cs = t.IS == 1 ? p.ae : p.aw, ct = t.JS == 1 ? p.an : p.as;
        float kI1 = cs * a.turb[x.at(dI, k)], kJ1 = ct * a.turb[x.at(dJ, k)];
        float kI2 = cs * a.tdiss[x.at(dI, k)], kJ2 = ct * a.tdiss[x.at(dJ, k)];
        if (t.IS == -1 && t.JS == -1) { kI1 = kI1 + kJ1; kI2 = kI2 + kJ2; }
        float kn = p.k1, en = p.e1;
        unsigned fl = (k > c.KK + 1 ? L_Q : 0u) | (k > c.KK ? L_R : 0u);
        if (k > c.KK) {
            const float *vf[3] = {a.uk, a.vk, a.wk};
            if (tke_wall(a, c, a.colke[c.col], k, kn, en, [&](int f, long long dc, int kk) { return vf[f][x.at(dc, kk)]; })) {
                kn = (float)net_maxd((double)kn, 0.001);
                en = (float)net_maxd((double)en, 0.0000001);
            } else {
                fl |= L_U;
            }
        }
        auto put = [&](int q, float v0, float v1) { rec[q * KL] = make_float2(v0, v1); };
        put(T_CI / 2, t.IS == 1 ? p.aw : p.ae, t.JS == 1 ? p.as : p.an);
        put(T_KI1 / 2, kI1, kJ1);
        put(T_KI2 / 2, kI2, kJ2);
        put(T_T1 / 2, p.t1, p.t2);
        put(T_T3 / 2, p.t3, p.s1);
        put(T_S2 / 2, p.s2, __uint_as_float(fl));
        put(T_K / 2, kn, en);
    };
    auto rest = [&](int cl, int k) {
        const size_t e = make_acc<false>(a, t.s, sm.col[cl].col).at(0, k);
        float2 *rec = base + (size_t)cl * rs + k;
        rec[(T_K / 2) * KL] = make_float2(a.turb[e], a.tdiss[e]);
        rec[(T_S2 / 2) * KL] = make_float2(0.0f, __uint_as_float(0u));
    };
    tile_items(a, t, sm, full, rest);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int cl = threadIdx.x >> 5; cl < t.nc; cl += CT_THREADS / 32) {
        const ColCtx &c = sm.col[cl];
        if (!(c.fl & F_ADV)) continue;
        const int ka = 2 * lane, kb = ka + 1;
        const bool inA = ka >= c.K0 && ka <= c.VI, inB = kb >= c.K0 && kb <= c.VI;
        const bool qA = inA && ka > c.KK + 1, qB = inB && kb > c.KK + 1;
        float4 *rec = reinterpret_cast<float4 *>(base + (size_t)cl * rs) + lane;
        constexpr int H = KL / 2;
        const float A0 = inA ? sm_f[0][cl][ka] : 1.0f, A1 = inB ? sm_f[0][cl][kb] : 1.0f;
        bool oddA = false, oddB = false;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const float B0 = inA ? sm_f[1 + 2 * v][cl][ka] : 0.0f, C0 = qA ? sm_f[2 + 2 * v][cl][ka] : 0.0f;
            const float B1 = inB ? sm_f[1 + 2 * v][cl][kb] : 0.0f, C1 = qB ? sm_f[2 + 2 * v][cl][kb] : 0.0f;
            const Elim<float> e = eliminate<float>(A0, B0, C0, qA, A1, B1, C1, qB);
            if (inA || inB) {
                rec[(v == 0 ? T_C1 : T_C2) / 2 * H] = make_float4(C0, e.den0, C1, e.den1);
                rec[(v == 0 ? T_Y1 : T_Y2) / 2 * H] = make_float4(1.0f / e.den0, e.P0, 1.0f / e.den1, e.P1);
            }
            oddA |= inA && odd_divisor(e.den0);
            oddB |= inB && odd_divisor(e.den1);
        }
        if (oddA || oddB) {
            float4 f = rec[(T_S2 / 2) * H];
            if (oddA) f.y = __uint_as_float(__float_as_uint(f.y) | L_D);
            if (oddB) f.w = __uint_as_float(__float_as_uint(f.w) | L_D);
            rec[(T_S2 / 2) * H] = f;
        }
    }
}

// ------------------------------------ row chains --------------------------------------------

// Record access shared by the jobs of this file: NP pairs, a record one column ahead in registers, lines
// of the records asked into L2.
template <int NP, int JS>
struct RecReader {
    const float4 *rec;
    const char *line;
    int step_rec;
    bool on0, on1;
    template <int M>
    __device__ __forceinline__ void begin(const KArgs &a, const ChainBufs &b, int u, int col, int lane) {
        step_rec = JS * M * (NP * (KMAX_LEVELS / 2));
        const float2 *p = b.rec + ((size_t)u * a.ncols + col) * (NP * KMAX_LEVELS);
        rec = reinterpret_cast<const float4 *>(p) + min(lane, a.ks / 2 - 1);
        line = reinterpret_cast<const char *>(p) + 128 * lane;
        on0 = (lane & 3) * 16 < a.ks && (lane >> 2) < NP;
        on1 = (lane & 3) * 16 < a.ks && (lane >> 2) + 8 < NP;
    }
    __device__ __forceinline__ void ahead(bool on) {
        l2_ahead(line, on && on0);
        if (NP > 8) l2_ahead(line + 4096, on && on1);
        line += step_rec * 16;
    }
    __device__ __forceinline__ void load(float4 (&f)[NP]) {
#pragma unroll
        for (int q = 0; q < NP; ++q) f[q] = __ldcg(rec + q * (KMAX_LEVELS / 2));
        rec += step_rec;
    }
};

// neighbour products in the reference's order AW1, AS1, AE1, AN1
template <int IS, int JS>
__device__ __forceinline__ float nbr_sum(float cI, float cJ, float kI, float kJ, float vI, float vJ) {
    const float pI = cI * vI, pJ = cJ * vJ;
    if (IS == 1) return (JS == 1) ? pI + pJ + kI + kJ : pI + kJ + kI + pJ;
    return (JS == 1) ? kI + pJ + pI + kJ : kI + pI + pJ;
}

// U, V of models 0 and 2, W of model 2.
template <int MODEL, int COMP, int IS, int JS>
struct ScalChain {
    static constexpr int NV = 1, NJ = 1, NF = 1;
    static constexpr int NP = scal_pairs<MODEL, COMP>();
    struct Rec {
        float4 f[NP];
    };
    struct Val {
        float2 v[NV];
    };
    RecReader<NP, JS> rd;
    float relax;
    float2 hz, ap0;
    float *F[NF];

    __device__ __forceinline__ void init(const KArgs &a, int lane) {
        relax = a.relax;
        F[0] = COMP == COMP_U ? a.uk : (COMP == COMP_V ? a.vk : a.wk);
        const float face = COMP == COMP_U ? a.dyk : a.dxk;
        const int l = min(lane, a.ks / 2 - 1);
        hz = make_float2(face * a.dzk[2 * l], face * a.dzk[2 * l + 1]);
    }
    template <int M>
    __device__ __forceinline__ void begin(const KArgs &a, const ChainBufs &b, int u, int s, int col, int lane) {
        rd.template begin<M>(a, b, u, col, lane);
        const int l = min(lane, a.ks / 2 - 1);
        const float *p = a.ap0 + (size_t)s * a.ks + 2 * l;
        ap0 = make_float2(p[0], p[1]);
    }
    __device__ __forceinline__ void ahead(bool on) { rd.ahead(on); }
    __device__ __forceinline__ void load(Rec &r) { rd.load(r.f); }
    __device__ __forceinline__ Val still(const KArgs &a, size_t base, int lane) const {
        Val o;
        o.v[0] = __ldcg(reinterpret_cast<const float2 *>(F[0] + base) + min(lane, a.ks / 2 - 1));
        return o;
    }
    struct Lev {
        float cI, cJ, kI, kJ, t1, t2, t3, w, vdx, K, e0, e1, e2, e3, phi, C, den, y, P;
        unsigned fl;
    };
#define GRAL_LEV(G)                                                                                             \
    Lev{G<S_CI>(f), G<S_CJ>(f), G<S_KI>(f), G<S_KJ>(f), G<S_T1>(f), G<S_T2>(f), G<S_T3>(f), G<S_W>(f),             \
        V ? G<V ? S_VDX : 0>(f) : 0.0f, V ? G<V ? S_K : 0>(f) : 0.0f, V ? G<V ? S_E0 : 0>(f) : 0.0f,               \
        V ? G<V ? S_E1 : 0>(f) : 0.0f, V ? G<V ? S_E2 : 0>(f) : 0.0f, V ? G<V ? S_E3 : 0>(f) : 0.0f, G<S_PHI>(f),  \
        G<S_C>(f), G<S_DEN>(f), G<S_Y>(f), G<S_P>(f), __float_as_uint(G<S_FL>(f))}
    __device__ __forceinline__ float dim(const Lev &r, float ap, float hzk, float vI, float vJ) const {
        const float S = nbr_sum<IS, JS>(r.cI, r.cJ, r.kI, r.kJ, vI, vJ);
        // uv_scalar_post, w_scalar_post: float products, then the sum in double
        double z = (double)S + (double)ap * 0.5 * (double)r.t1;
        z = z + (double)r.t2;
        if (COMP == COMP_W) {
            float D = (float)z;
            add_if(D, D, r.w, r.fl & L_X);
            return D;
        }
        z = z + (double)r.t3;
        float D = (float)z - r.w;
        if (MODEL == 2) {
            float X;
            if (COMP == COMP_U) {
                const float d = (IS == 1) ? r.K - (r.phi - vI) * hzk : (vI - r.phi) * hzk - r.K;
                X = d + r.e0 - r.e1 + r.e2 - r.e3;
            } else {
                const float d = (JS == 1) ? r.K - (r.phi - vJ) * hzk : r.e0 + (vJ - r.phi) * hzk - r.K;
                X = d + r.e1 - r.e2;
            }
            add_if(D, D, r.vdx * X, r.fl & L_X);
        }
        return D;
    }
    __device__ __forceinline__ Val step(const Rec &rc, const Val &vI, const float2 (&vJ)[NJ]) const {
        constexpr bool V = MODEL == 2 && COMP != COMP_W;
        const float4 *f = rc.f;
        const Lev A = GRAL_LEV(lev_a), B = GRAL_LEV(lev_b);
        const float Da = dim(A, ap0.x, hz.x, vI.v[0].x, vJ[0].x), Db = dim(B, ap0.y, hz.y, vI.v[0].y, vJ[0].y);
        const unsigned qA = A.fl & L_Q, qB = B.fl & L_Q, uA = A.fl & L_U, uB = B.fl & L_U;
        float Qa = 0.0f, Qb = 0.0f, inQ = 0.0f, inU = 0.0f;
        quot_if(Qa, Da, A.den, A.y, 1u);
        quot_if(Qb, Db, B.den, B.y, 1u);
        quot_if(Qb, Db + B.C * Qa, B.den, B.y, qB);
        auto up = [&]() {
            quot_if(Qa, Da + A.C * inQ, A.den, A.y, qA);
            quot_if(Qb, Db + B.C * Qa, B.den, B.y, qB);
        };
        float va = A.phi, vb = B.phi;
        auto down = [&]() {
            add_if(vb, B.phi, relax * (B.P * inU + Qb - B.phi), uB);
            add_if(va, A.phi, relax * (A.P * vb + Qa - A.phi), uA);
        };
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
            if (!more) break;
            up();
        }
        // dividends and quotients of the settled Q, where they are in use
        const float xa = qA ? Da + A.C * inQ : Da, xb = qB ? Db + B.C * Qa : Db;
        const bool odd = max(in_use(quot_worst(xa, Qa), A.fl), in_use(quot_worst(xb, Qb), B.fl)) >= QUOT_SPAN;
        // the vote's result is looked at only after the back-substitution, whose rounds hide it
        const bool redo = __any_sync(0xffffffffu, odd);
        auto settle = [&]() {
            for (;;) {
                const float nU = __shfl_down_sync(0xffffffffu, va, 1);
                const bool more = __any_sync(0xffffffffu, differ(nU, inU));
                inU = nU;
                down();
                if (!more) break;
            }
        };
        settle();
        if (redo) {
            Qa = Da / A.den;
            Qb = Db / B.den;
            for (bool first = true;; first = false) {
                const float nQ = __shfl_up_sync(0xffffffffu, Qb, 1);
                const bool more = __any_sync(0xffffffffu, differ(nQ, inQ));
                if (!more && !first) break;
                inQ = nQ;
                if (qA) Qa = (Da + A.C * inQ) / A.den;
                if (qB) Qb = (Db + B.C * Qa) / B.den;
            }
            inU = __shfl_down_sync(0xffffffffu, va, 1);
            down();
            settle();
        }
        Val o;
        o.v[0] = make_float2(va, vb);
        return o;
    }
#undef GRAL_LEV
};

// W of model 0: P, Q and the divisor in double (W-prognostic-microscale_0.cs:35-36, 124-139).
template <int IS, int JS>
struct W0Chain {
    static constexpr int NV = 1, NJ = 1, NF = 1;
    struct Rec {
        float4 f[Z_PAIRS];
    };
    struct Val {
        float2 v[NV];
    };
    RecReader<Z_PAIRS, JS> rd;
    double relax;
    float2 ap0;
    float *F[NF];

    __device__ __forceinline__ void init(const KArgs &a, int) {
        relax = (double)a.relax;
        F[0] = a.wk;
    }
    template <int M>
    __device__ __forceinline__ void begin(const KArgs &a, const ChainBufs &b, int u, int s, int col, int lane) {
        rd.template begin<M>(a, b, u, col, lane);
        const float *p = a.ap0 + (size_t)s * a.ks + 2 * min(lane, a.ks / 2 - 1);
        ap0 = make_float2(p[0], p[1]);
    }
    __device__ __forceinline__ void ahead(bool on) { rd.ahead(on); }
    __device__ __forceinline__ void load(Rec &r) { rd.load(r.f); }
    __device__ __forceinline__ Val still(const KArgs &a, size_t base, int lane) const {
        Val o;
        o.v[0] = __ldcg(reinterpret_cast<const float2 *>(F[0] + base) + min(lane, a.ks / 2 - 1));
        return o;
    }
    __device__ __forceinline__ Val step(const Rec &rc, const Val &vI, const float2 (&vJ)[NJ]) const {
        const float4 *f = rc.f;
        auto dbl = [](float lo, float hi) { return __hiloint2double(__float_as_int(hi), __float_as_int(lo)); };
        const float Sa = nbr_sum<IS, JS>(f[0].x, f[0].y, f[1].x, f[1].y, vI.v[0].x, vJ[0].x);
        const float Sb = nbr_sum<IS, JS>(f[0].z, f[0].w, f[1].z, f[1].w, vI.v[0].y, vJ[0].y);
        const float Da = (float)((double)Sa + (double)ap0.x * 0.5 * (double)f[2].x + (double)f[2].y);
        const float Db = (float)((double)Sb + (double)ap0.y * 0.5 * (double)f[2].z + (double)f[2].w);
        const float fa = f[3].x, fb = f[3].z;
        const unsigned la = __float_as_uint(f[3].y), lb = __float_as_uint(f[3].w);
        const unsigned qA = la & L_Q, qB = lb & L_Q, uA = la & L_U, uB = lb & L_U;
        const double Ca = f[4].x, Cb = f[4].z;
        const double dA = dbl(f[Z_DEN].x, f[Z_DEN].y), dB = dbl(f[Z_DEN].z, f[Z_DEN].w);
        const double yA = dbl(f[Z_Y].x, f[Z_Y].y), yB = dbl(f[Z_Y].z, f[Z_Y].w);
        const double PA = dbl(f[Z_P].x, f[Z_P].y), PB = dbl(f[Z_P].z, f[Z_P].w);
        // up to KKART+1 the quotient is a float's
        double Qa = (double)(Da / f[4].y), Qb = (double)(Db / f[4].w), inQ = 0.0;
        float va = fa, vb = fb, inU = 0.0f;
        auto up = [&]() {
            quot_if(Qa, (double)Da + Ca * inQ, dA, yA, qA);
            quot_if(Qb, (double)Db + Cb * Qa, dB, yB, qB);
        };
        auto down = [&]() {
            add_if(vb, fb, (float)(relax * (PB * (double)inU + Qb - (double)fb)), uB);
            add_if(va, fa, (float)(relax * (PA * (double)vb + Qa - (double)fa)), uA);
        };
        auto same = [](double x, double y) { return __double_as_longlong(x) == __double_as_longlong(y); };
        quot_if(Qb, (double)Db + Cb * Qa, dB, yB, qB);
#pragma unroll
        for (int n = 0; n < ROUNDS_MOM; ++n) {
            inU = __shfl_down_sync(0xffffffffu, va, 1);
            inQ = __shfl_up_sync(0xffffffffu, Qb, 1);
            down();
            up();
        }
        for (;;) {
            const double nQ = __shfl_up_sync(0xffffffffu, Qb, 1);
            const bool more = __any_sync(0xffffffffu, !same(nQ, inQ));
            inQ = nQ;
            if (!more) break;
            up();
        }
        const double xa = (double)Da + Ca * inQ, xb = (double)Db + Cb * Qa;
        const unsigned wA = quot_worst(xa, Qa) | (odd_divisor(dA) ? 0x80000000u : 0u);
        const unsigned wB = quot_worst(xb, Qb) | (odd_divisor(dB) ? 0x80000000u : 0u);
        const bool odd = max(qA ? wA : 0u, qB ? wB : 0u) >= QUOT_SPAN_DOUBLE;
        const bool redo = __any_sync(0xffffffffu, odd);
        auto settle = [&]() {
            inU = __shfl_down_sync(0xffffffffu, va, 1);
            down();
            for (;;) {
                const float nU = __shfl_down_sync(0xffffffffu, va, 1);
                const bool more = __any_sync(0xffffffffu, differ(nU, inU));
                inU = nU;
                down();
                if (!more) break;
            }
        };
        settle();
        if (redo) {
            for (bool first = true;; first = false) {
                const double nQ = __shfl_up_sync(0xffffffffu, Qb, 1);
                const bool more = __any_sync(0xffffffffu, !same(nQ, inQ));
                if (!more && !first) break;
                inQ = nQ;
                if (qA) Qa = ((double)Da + Ca * inQ) / dA;
                if (qB) Qb = ((double)Db + Cb * Qa) / dB;
            }
            settle();
        }
        Val o;
        o.v[0] = make_float2(va, vb);
        return o;
    }
};

// k and eps (TKE-prognostic-microscale.cs:255-347): two recurrences each, side by side.
template <int IS, int JS>
struct TkeChain {
    static constexpr int NV = 2, NJ = 2, NF = 2;
    struct Rec {
        float4 f[TKE_PAIRS];
    };
    struct Val {
        float2 v[NV];
    };
    RecReader<TKE_PAIRS, JS> rd;
    float *F[NF];

    __device__ __forceinline__ void init(const KArgs &a, int) {
        F[0] = a.turb;
        F[1] = a.tdiss;
    }
    template <int M>
    __device__ __forceinline__ void begin(const KArgs &a, const ChainBufs &b, int u, int, int col, int lane) {
        rd.template begin<M>(a, b, u, col, lane);
    }
    __device__ __forceinline__ void ahead(bool on) { rd.ahead(on); }
    __device__ __forceinline__ void load(Rec &r) { rd.load(r.f); }
    __device__ __forceinline__ Val still(const KArgs &a, size_t base, int lane) const {
        Val o;
#pragma unroll
        for (int q = 0; q < 2; ++q) o.v[q] = __ldcg(reinterpret_cast<const float2 *>(F[q] + base) + min(lane, a.ks / 2 - 1));
        return o;
    }
    // P*up + Q clamped from below, as net_maxd((double)x, 0.001) rounded to float (and 1e-7): a float is
    // below the double bound exactly when it is below the bound's float, and NaN stays
    static __device__ __forceinline__ float clamped(float x, float lo) { return x < lo ? lo : x; }
    __device__ __forceinline__ Val step(const Rec &rc, const Val &vI, const float2 (&vJ)[NJ]) const {
        const float4 *f = rc.f;
        const unsigned la = __float_as_uint(lev_a<T_FL>(f)), lb = __float_as_uint(lev_b<T_FL>(f));
        const unsigned qA = la & L_Q, qB = lb & L_Q, uA = la & L_U, uB = lb & L_U;
        float Da[2], Db[2], Qa[2], Qb[2], va[2], vb[2], inQ[2] = {0.0f, 0.0f}, inV[2] = {0.0f, 0.0f};
        const float Ca[2] = {lev_a<T_C1>(f), lev_a<T_C2>(f)}, Cb[2] = {lev_b<T_C1>(f), lev_b<T_C2>(f)};
        const float dA[2] = {lev_a<T_DEN1>(f), lev_a<T_DEN2>(f)}, dB[2] = {lev_b<T_DEN1>(f), lev_b<T_DEN2>(f)};
        const float yA[2] = {lev_a<T_Y1>(f), lev_a<T_Y2>(f)}, yB[2] = {lev_b<T_Y1>(f), lev_b<T_Y2>(f)};
        const float PA[2] = {lev_a<T_P1>(f), lev_a<T_P2>(f)}, PB[2] = {lev_b<T_P1>(f), lev_b<T_P2>(f)};
        constexpr float LO[2] = {0.001f, 0.0000001f};
        Da[0] = nbr_sum<IS, JS>(lev_a<T_CI>(f), lev_a<T_CJ>(f), lev_a<T_KI1>(f), lev_a<T_KJ1>(f), vI.v[0].x, vJ[0].x) +
                lev_a<T_T1>(f) + lev_a<T_T2>(f) + lev_a<T_T3>(f);
        Db[0] = nbr_sum<IS, JS>(lev_b<T_CI>(f), lev_b<T_CJ>(f), lev_b<T_KI1>(f), lev_b<T_KJ1>(f), vI.v[0].y, vJ[0].y) +
                lev_b<T_T1>(f) + lev_b<T_T2>(f) + lev_b<T_T3>(f);
        Da[1] = nbr_sum<IS, JS>(lev_a<T_CI>(f), lev_a<T_CJ>(f), lev_a<T_KI2>(f), lev_a<T_KJ2>(f), vI.v[1].x, vJ[1].x) +
                lev_a<T_S1>(f) + lev_a<T_S2>(f);
        Db[1] = nbr_sum<IS, JS>(lev_b<T_CI>(f), lev_b<T_CJ>(f), lev_b<T_KI2>(f), lev_b<T_KJ2>(f), vI.v[1].y, vJ[1].y) +
                lev_b<T_S1>(f) + lev_b<T_S2>(f);
        va[0] = lev_a<T_K>(f); vb[0] = lev_b<T_K>(f);
        va[1] = lev_a<T_E>(f); vb[1] = lev_b<T_E>(f);
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            Qa[v] = Qb[v] = 0.0f;
            quot_if(Qa[v], Da[v], dA[v], yA[v], 1u);
            quot_if(Qb[v], Db[v], dB[v], yB[v], 1u);
            quot_if(Qb[v], Db[v] + Cb[v] * Qa[v], dB[v], yB[v], qB);
        }
        auto up = [&](int v) {
            quot_if(Qa[v], Da[v] + Ca[v] * inQ[v], dA[v], yA[v], qA);
            quot_if(Qb[v], Db[v] + Cb[v] * Qa[v], dB[v], yB[v], qB);
        };
        auto down = [&](int v) {
            const float x = clamped(PB[v] * inV[v] + Qb[v], LO[v]);
            vb[v] = uB ? x : vb[v];
            const float y = clamped(PA[v] * vb[v] + Qa[v], LO[v]);
            va[v] = uA ? y : va[v];
        };
#pragma unroll
        for (int n = 0; n < ROUNDS_PRESS; ++n)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                inV[v] = __shfl_down_sync(0xffffffffu, va[v], 1);
                inQ[v] = __shfl_up_sync(0xffffffffu, Qb[v], 1);
                down(v);
                up(v);
            }
        for (;;) {
            float nQ[2];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                nQ[v] = __shfl_up_sync(0xffffffffu, Qb[v], 1);
                inV[v] = __shfl_down_sync(0xffffffffu, va[v], 1);
            }
            const bool more = __any_sync(0xffffffffu, differ(nQ[0], inQ[0]) || differ(nQ[1], inQ[1]));
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                inQ[v] = nQ[v];
                down(v);
            }
            if (!more) break;
            up(0);
            up(1);
        }
        unsigned worst = 0;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const float xa = qA ? Da[v] + Ca[v] * inQ[v] : Da[v], xb = qB ? Db[v] + Cb[v] * Qa[v] : Db[v];
            worst = max(worst, max(in_use(quot_worst(xa, Qa[v]), la), in_use(quot_worst(xb, Qb[v]), lb)));
        }
        const bool redo = __any_sync(0xffffffffu, worst >= QUOT_SPAN);
        auto settle = [&]() {
            for (;;) {
                float nV[2];
#pragma unroll
                for (int v = 0; v < 2; ++v) nV[v] = __shfl_down_sync(0xffffffffu, va[v], 1);
                const bool more = __any_sync(0xffffffffu, differ(nV[0], inV[0]) || differ(nV[1], inV[1]));
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    inV[v] = nV[v];
                    down(v);
                }
                if (!more) break;
            }
        };
        settle();
        if (redo) {
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                Qa[v] = Da[v] / dA[v];
                Qb[v] = Db[v] / dB[v];
                for (bool first = true;; first = false) {
                    const float nQ = __shfl_up_sync(0xffffffffu, Qb[v], 1);
                    const bool more = __any_sync(0xffffffffu, differ(nQ, inQ[v]));
                    if (!more && !first) break;
                    inQ[v] = nQ;
                    if (qA) Qa[v] = (Da[v] + Ca[v] * inQ[v]) / dA[v];
                    if (qB) Qb[v] = (Db[v] + Cb[v] * Qa[v]) / dB[v];
                }
                inV[v] = __shfl_down_sync(0xffffffffu, va[v], 1);
                down(v);
            }
            settle();
        }
        Val o;
#pragma unroll
        for (int v = 0; v < 2; ++v) o.v[v] = make_float2(va[v], vb[v]);
        return o;
    }
};

template <int MODEL, int KIND, int IS, int JS>
struct JobOf {
    using T = ScalChain<MODEL, KIND == PH_U ? COMP_U : (KIND == PH_V ? COMP_V : COMP_W), IS, JS>;
};
template <int IS, int JS>
struct JobOf<0, PH_W, IS, JS> {
    using T = W0Chain<IS, JS>;
};
template <int IS, int JS>
struct JobOf<2, PH_TKE, IS, JS> {
    using T = TkeChain<IS, JS>;
};

template <int MODEL, int KIND>
__global__ void __cluster_dims__(CH_CL, 1, 1) __launch_bounds__(CH_THREADS, 2) k_scal_chain(KArgs a, SweepGeom g, ChainBufs b) {
    __shared__ ChainSmem<CH_SR, JobOf<MODEL, KIND, 1, 1>::T::NV> sm;
    constexpr int SR = CH_SR, M = CH_M, CL = CH_CL;
    for (unsigned q = threadIdx.x; q < sizeof(sm.ring) / 8; q += CH_THREADS) sm.ring[q] = 0ull;
    int is, js;
    chain_dir(*a.it_global, is, js);
    if (is == 1) {
        if (js == 1) run_chain<typename JobOf<MODEL, KIND, 1, 1>::T, KIND, SR, M, CL, 1, 1>(a, g, b, sm);
        else run_chain<typename JobOf<MODEL, KIND, 1, -1>::T, KIND, SR, M, CL, 1, -1>(a, g, b, sm);
    } else {
        if (js == 1) run_chain<typename JobOf<MODEL, KIND, -1, 1>::T, KIND, SR, M, CL, -1, 1>(a, g, b, sm);
        else run_chain<typename JobOf<MODEL, KIND, -1, -1>::T, KIND, SR, M, CL, -1, -1>(a, g, b, sm);
    }
}

}  // namespace

KFn chain_scalar_kernel(int kind, int model) {
    switch (kind) {
        case PH_U: return model == 2 ? k_scal_chain<2, PH_U> : k_scal_chain<0, PH_U>;
        case PH_V: return model == 2 ? k_scal_chain<2, PH_V> : k_scal_chain<0, PH_V>;
        case PH_W: return model == 2 ? k_scal_chain<2, PH_W> : k_scal_chain<0, PH_W>;
        default: return k_scal_chain<2, PH_TKE>;
    }
}

KFn chain_scalar_terms(int kind, int model) {
    switch (kind) {
        case PH_U: return model == 2 ? k_scal_terms<2, COMP_U> : k_scal_terms<0, COMP_U>;
        case PH_V: return model == 2 ? k_scal_terms<2, COMP_V> : k_scal_terms<0, COMP_V>;
        case PH_W: return model == 2 ? k_scal_terms<2, COMP_W> : k_scal_terms<0, COMP_W>;
        default: return k_tke_terms;
    }
}

int chain_scalar_pairs(int model) { return model == 2 ? TKE_PAIRS : (int)Z_PAIRS; }

}  // namespace gral
