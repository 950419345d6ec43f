// adj_chain.cuh -- the reverse sweeps of the adjoint on the row-chain schedule (prog_chain.cuh);
// included by prog_adjoint.cu inside its namespace.
//
// A reverse sweep is the forward's chain walked the other way: a column's cotangents need those of
// its two sweep successors and nothing else of the sweep.  Three launches: a parallel kernel forms the
// row, its Thomas recurrence and one record per column; the chain kernel runs only the recurrences
// between the columns (two per column, contractions as in the forward, see prog_chain.cuh); a
// parallel kernel turns the row's cotangents into those of its inputs.
//
// What bounds it: in the chain the column steps, 0.41 us each (a wavefront step of rev_tasks, a hand-off
// through global memory and about 100 levels of serial recurrence, took 3.1 us); in the parallel kernels
// latency: 55-60 % of the issue slots stay empty behind 32-35 loads a level at 16-20 warps an SM.  200x200, levels 25, us of a
// momentum sweep: terms 165, chain 163, rest 170 (rev_tasks 1250); pressure: 12, 221 (1250).

// Warps (columns) of a block of the parallel kernels.  Their five blocks an SM (96 registers, a few spilled)
// measured 21.5 ms for the reverse of 12 iterations on 200x200, four without spills 22.6, six 21.9, eight 23.6.
constexpr int AC_BLOCK = 4;
constexpr int AM_PAIRS = 3, AP_PAIRS = 2;

struct AdjChain {
    float2 *rec;        // [col][pair][KMAX_LEVELS]
    float *plane;       // PL_N fields [col][KS]
    const float2 *ptab; // the forward's elimination table [dir][col][KS] {TERMP, P}
    size_t fsz;         // floats of a field
    __device__ __forceinline__ float *at(int q) const { return plane + (size_t)q * fsz; }
};
enum : int { PL_T, PL_B, PL_E, PL_TTC, PL_QPT, PL_PP, PL_LQ, PL_MU, PL_N };

// sweep coordinates of warp w of a column launch, forward order
__device__ __forceinline__ bool sweep_col(const KArgs &a, const SweepGeom &g, int IS, int JS, int &i1, int &j1, int &i,
                                          int &j) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= (long long)g.ni * g.nj) return false;
    // the sweep's rows contiguous along j, as they lie in memory
    i1 = g.ia + (int)(w / g.nj);
    j1 = g.ja + (int)(w % g.nj);
    i = (IS == 1) ? i1 : a.nii - i1 + 1;
    j = (JS == 1) ? j1 : a.njj - j1 + 1;
    return true;
}

template <int COMP>
struct MomSplit : MomRev<COMP> {
    using B = MomRev<COMP>;
    using B::a, B::d, B::M, B::S, B::c, B::act, B::kkm, B::top_carry;

    // Record pairs of a level: (cotangent L0 of the new value left by the later phases, 1 where the
    // sweep updates the level), (T*C1 of the successor in i, T*C2 of the one in j: this column's
    // coefficients in their rows), (relax*P_{k-1}, C_{k+1}*T_{k+1}).  The second pair is written by
    // the successors' warps; a column at the sweep's end writes its own zeros.
    __device__ void record(const AdjChain &h, int IS, int JS, bool p1, bool p2, bool s1, bool s2) {
        const int lane = threadIdx.x & 31, ks = a.ks;
        const int K0 = c.K0, VI = c.VI, KK = c.KK;
        if (act) {
            // Thomas recurrence: two levels per lane, in rounds until no bit changes
            const int ka = 2 * lane, kb = ka + 1;
            const bool iA = ka >= K0 && ka <= VI, iB = kb >= K0 && kb <= VI;
            const float A0 = iA ? S[R_A][ka] : 1.0f, B0 = iA ? S[R_B][ka] : 0.0f, D0 = iA ? S[R_D][ka] : 0.0f;
            const float A1 = iB ? S[R_A][kb] : 1.0f, B1 = iB ? S[R_B][kb] : 0.0f, D1 = iB ? S[R_D][kb] : 0.0f;
            const bool qA = iA && ka > KK + 1, qB = iB && kb > KK + 1;
            const float C0 = qA ? S[R_C][ka] : 0.0f, C1 = qB ? S[R_C][kb] : 0.0f;
            float T0, T1, P0, P1, Q0, Q1, inP = 0.0f, inQ = 0.0f;
            for (;;) {
                T0 = 1.0f / (qA ? A0 - C0 * inP : A0);
                P0 = B0 * T0;
                Q0 = (qA ? D0 + C0 * inQ : D0) * T0;
                T1 = 1.0f / (qB ? A1 - C1 * P0 : A1);
                P1 = B1 * T1;
                Q1 = (qB ? D1 + C1 * Q0 : D1) * T1;
                const float nP = __shfl_up_sync(0xffffffffu, P1, 1), nQ = __shfl_up_sync(0xffffffffu, Q1, 1);
                if (!__any_sync(0xffffffffu, lane > 0 && (differ(nP, inP) || differ(nQ, inQ)))) break;
                inP = nP;
                inQ = nQ;
            }
            if (iA) { S[R_T][ka] = T0; S[R_P][ka] = P0; S[R_Q][ka] = Q0; }
            if (iB) { S[R_T][kb] = T1; S[R_P][kb] = P1; S[R_Q][kb] = Q1; }
        }
        __syncwarp();
        constexpr size_t rs = (size_t)AM_PAIRS * KMAX_LEVELS;
        float2 *r0 = h.rec + (size_t)c.col * rs;
        float *t1 = reinterpret_cast<float *>(h.rec + (size_t)(c.col - IS * a.nj2) * rs + KMAX_LEVELS);
        float *t2 = reinterpret_cast<float *>(h.rec + (size_t)(c.col - JS) * rs + KMAX_LEVELS) + 1;
        float *own = reinterpret_cast<float *>(r0 + KMAX_LEVELS);
        float *L = d.lam[COMP];
        for (int k = lane; k < ks; k += 32) {
            const size_t e = cell(a, c.col, k);
            float2 x = make_float2(0.0f, 0.0f), w = x, tc = x;
            if (act && k == VI + 1) h.at(PL_PP)[e] = S[R_P][VI];
            if (act && k >= K0 && k <= VI) {
                const bool ch = k > KK + 1;
                const float C = S[R_C][k], D = S[R_D][k], T = S[R_T][k];
                const float Qp = ch ? S[R_Q][k - 1] : 0.0f;
                h.at(PL_T)[e] = T;
                h.at(PL_B)[e] = S[R_B][k];
                h.at(PL_E)[e] = ch ? D + C * Qp : D;
                h.at(PL_TTC)[e] = ch ? T * T * C : 0.0f;
                h.at(PL_QPT)[e] = Qp * T;
                h.at(PL_PP)[e] = ch ? S[R_P][k - 1] : 0.0f;
                // an updated level's cotangent is handed over from its new to its old value
                if (kkm < k) {
                    x = make_float2(__ldcg(L + e), 1.0f);
                    L[e] = 0.0f;
                }
                if (k > K0) w.x = a.relax * S[R_P][k - 1];
                if (k < VI && k >= KK + 1) w.y = S[R_C][k + 1] * S[R_T][k + 1];
                tc = make_float2(T * S[R_C1][k], T * S[R_C2][k]);
            }
            r0[k] = x;
            r0[k + 2 * KMAX_LEVELS] = w;
            if (p1) t1[2 * k] = tc.x;
            if (p2) t2[2 * k] = tc.y;
            if (!s1) own[2 * k] = 0.0f;
            if (!s2) own[2 * k + 1] = 0.0f;
        }
    }

    // the levels of a predecessor that the chain has served: those its sweep step updated
    __device__ LevelSpan served(int di, int dj, bool in) const {
        LevelSpan s{1, 0};
        if (!in) return s;
        const ColCtx p = make_col(a, c.i + di, c.j + dj);
        if (!(p.fl & F_ADV)) return s;
        const int km = (COMP == 0) ? p.kkm_u : (COMP == 1 ? p.kkm_v : -32768);
        s.lo = max(p.K0, km + 1);
        s.hi = p.VI;
        return s;
    }

    // from the chain's cotangents mu (new value) and lQ: the recurrence of lP (top down, in rounds as
    // above), then the cotangents of A, B, C, D and of the old value
    __device__ void rest(const AdjChain &h, int IS, int JS, bool p1, bool p2) {
        if (!act) return;
        const int lane = threadIdx.x & 31;
        const int K0 = c.K0, VI = c.VI, ka = 2 * lane;
        const float relax = a.relax, r1 = 1.0f - relax;
        const size_t e0 = cell(a, c.col, 0);
        const float *up = d.end[COMP] + e0;
        float T[2], Bc[2], E[2], TTC[2], q[2], mu[2], qpt[2], pp[2], s[2];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int k = ka + n;
            const bool in = k >= K0 && k <= VI;
            const size_t e = e0 + k;
            T[n] = in ? h.at(PL_T)[e] : 0.0f;
            Bc[n] = in ? h.at(PL_B)[e] : 0.0f;
            E[n] = in ? h.at(PL_E)[e] : 0.0f;
            TTC[n] = in ? h.at(PL_TTC)[e] : 0.0f;
            qpt[n] = in ? h.at(PL_QPT)[e] : 0.0f;
            pp[n] = in ? h.at(PL_PP)[e] : 0.0f;
            q[n] = in ? h.at(PL_LQ)[e] : 0.0f;
            mu[n] = in ? h.at(PL_MU)[e] : 0.0f;
            s[n] = in ? relax * __ldcg(up + k + 1) * mu[n] : 0.0f;
        }
        top_carry = relax * h.at(PL_PP)[e0 + VI + 1] * h.at(PL_MU)[e0 + VI];
        float lT[2], lP[2], in = 0.0f;
        const float eb = q[1] * E[1], ea = q[0] * E[0];
        for (;;) {
            lP[1] = s[1] + in;
            lT[1] = fmaf(lP[1], Bc[1], eb);
            lP[0] = s[0] + TTC[1] * lT[1];
            lT[0] = fmaf(lP[0], Bc[0], ea);
            const float n = __shfl_down_sync(0xffffffffu, TTC[0] * lT[0], 1);
            if (!__any_sync(0xffffffffu, lane < 31 && differ(n, in))) break;
            if (lane < 31) in = n;
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int k = ka + n;
            const float lden = -(lT[n] * (T[n] * T[n]));
            S[R_A][k] = lden;
            S[R_B][k] = lP[n] * T[n];
            S[R_C][k] = q[n] * qpt[n] - lden * pp[n];
            S[R_D][k] = q[n] * T[n];
            S[R_LO][k] = r1 * mu[n];
        }
        __syncwarp();
        this->after(IS, JS, served(-IS, 0, p1), served(0, -JS, p2));
    }
};

template <int COMP>
__device__ __forceinline__ void mom_dir(int it, int &IS, int &JS) {
    sweep_dir_of(it, IS, JS);
    if (COMP == 1) { IS = -IS; JS = -JS; }   // model-1 V sweeps with (-IS, -JS)
}

template <int COMP>
__global__ void __launch_bounds__(AC_BLOCK * 32, 5) k_adj_mom_terms(KArgs a, AdjArgs d, SweepGeom g, AdjChain h) {
    __shared__ MomShared sm[AC_BLOCK];
    MomShared &M = sm[threadIdx.x >> 5];
    int IS, JS, i1, j1, i, j;
    mom_dir<COMP>(d.it, IS, JS);
    if (!sweep_col(a, g, IS, JS, i1, j1, i, j)) return;
    MomSplit<COMP> job{{a, d, M, M.rows}};
    job.rows(i, j, IS, JS);
    job.record(h, IS, JS, i1 > g.ia, j1 > g.ja, i1 < g.ia + g.ni - 1, j1 < g.ja + g.nj - 1);
}

template <int COMP>
__global__ void __launch_bounds__(AC_BLOCK * 32, 5) k_adj_mom_rest(KArgs a, AdjArgs d, SweepGeom g, AdjChain h) {
    __shared__ MomShared sm[AC_BLOCK];
    MomShared &M = sm[threadIdx.x >> 5];
    int IS, JS, i1, j1, i, j;
    mom_dir<COMP>(d.it, IS, JS);
    if (!sweep_col(a, g, IS, JS, i1, j1, i, j)) return;
    MomSplit<COMP> job{{a, d, M, M.rows}};
    job.column(i, j);
    job.rest(h, IS, JS, i1 > g.ia, j1 > g.ja);
}

// Pressure records: (cotangent of DPM and relaxp times that of DPMNEW, P_{k+1}), (ATP_{k-1}*TERMP_{k-1},
// TERMP); a thread per level.  TERMP is zero on the levels the sweep does not solve; at
// VerticalIndex+1 the third entry carries the top level's share of the row carry.
__global__ void __launch_bounds__(256) k_adj_press_terms(KArgs a, AdjArgs d, AdjChain h) {
    const int k = threadIdx.x, col = blockIdx.x * blockDim.y + threadIdx.y;
    if (col >= a.ncols) return;
    int IS, JS;
    sweep_dir_of(d.it, IS, JS);
    const int dirx = (IS == 1) ? 0 : 1;
    const ColMeta m = a.meta[col];
    const bool act = (a.cflags[col] & F_ADV) != 0;
    const float2 *tp = h.ptab + (size_t)dirx * h.fsz;
    const size_t e = cell(a, col, k);
    float2 x = make_float2(0.0f, 0.0f), y = x;
    if (act && k > m.kkart && k <= m.vi) {
        x.x = d.lam[L_DPM][e] + a.relaxp * d.lam[FDP][e];
        if (k < m.vi) x.y = tp[e + 1].y;
        y.y = tp[e].x;
    }
    if (act && k > m.kkart + 1 && k <= m.vi + 1) y.x = a.atp[k - 1] * tp[e - 1].x;
    float2 *r = h.rec + (size_t)col * AP_PAIRS * KMAX_LEVELS + k;
    r[0] = x;
    r[KMAX_LEVELS] = y;
}

// What the two chains share: the column records and the values outside the sweep (zero).
template <int NP, int NV_, int NF_, int JS>
struct AdjChainBase {
    static constexpr int NV = NV_, NJ = 1, NF = NF_;
    struct Rec {
        float4 f[NP];
    };
    struct Val {
        float2 v[NV_ > NF_ ? NV_ : NF_];
    };
    float *F[NF];
    const float4 *rec;
    const char *line;
    int step_rec;
    bool on0;
    __device__ __forceinline__ void lines(const KArgs &a, int lane) { on0 = (lane & 3) * 16 < a.ks && (lane >> 2) < NP; }
    template <int M>
    __device__ __forceinline__ void begin(const KArgs &a, const ChainBufs &b, int, int, int col, int lane) {
        step_rec = JS * M * (NP * (KMAX_LEVELS / 2));
        const float2 *p = b.rec + (size_t)col * (NP * KMAX_LEVELS);
        rec = reinterpret_cast<const float4 *>(p) + min(lane, a.ks / 2 - 1);
        line = reinterpret_cast<const char *>(p) + 128 * lane;
    }
    __device__ __forceinline__ void ahead(bool on) {
        l2_ahead(line, on && on0);
        line += step_rec * 16;
    }
    __device__ __forceinline__ void load(Rec &r) {
#pragma unroll
        for (int q = 0; q < NP; ++q) r.f[q] = __ldcg(rec + q * (KMAX_LEVELS / 2));
        rec += step_rec;
    }
    __device__ __forceinline__ Val still(const KArgs &, size_t, int) const { return Val{}; }
};

// Momentum: mu_k = L0_k + relax*P_{k-1}*mu_{k-1} (bottom up, the back-substitution reversed) and
// lQ_k = relax*mu_k + C_{k+1}*T_{k+1}*lQ_{k+1} (top down, the recurrence of Q reversed), L0 with the successors' parts
// lQ*(T*C1) at the updated levels.  lQ is handed on; mu is kept for the last kernel.
template <int JS>
struct MomAdjChain : AdjChainBase<AM_PAIRS, 1, 2, JS> {
    using B = AdjChainBase<AM_PAIRS, 1, 2, JS>;
    using typename B::Rec;
    using typename B::Val;
    float relax;
    __device__ __forceinline__ void init(const KArgs &a, int lane) {
        relax = a.relax;
        this->lines(a, lane);
    }
    __device__ __forceinline__ Val step(const Rec &r, const Val &vI, const float2 (&vJ)[1]) const {
        const float4 x = r.f[0], t = r.f[1], w = r.f[2];
        float xa = x.x, xb = x.z;
        add_if(xa, x.x, fmaf(vI.v[0].x, t.x, vJ[0].x * t.y), x.y != 0.0f);
        add_if(xb, x.z, fmaf(vI.v[0].y, t.z, vJ[0].y * t.w), x.w != 0.0f);
        float ma = xa, mb = fmaf(w.z, ma, xb), qa, qb, inM = 0.0f, inQ = 0.0f;
        auto up = [&]() {
            ma = fmaf(w.x, inM, xa);
            mb = fmaf(w.z, ma, xb);
        };
        auto down = [&]() {
            qb = fmaf(w.w, inQ, relax * mb);
            qa = fmaf(w.y, qb, relax * ma);
        };
        down();
        // lanes at the ends take their own value back from the shuffle; their coefficient is zero
#pragma unroll
        for (int n = 0; n < ROUNDS_MOM; ++n) {
            inM = __shfl_up_sync(0xffffffffu, mb, 1);
            inQ = __shfl_down_sync(0xffffffffu, qa, 1);
            up();
            down();
        }
        for (;;) {
            const float nM = __shfl_up_sync(0xffffffffu, mb, 1), nQ = __shfl_down_sync(0xffffffffu, qa, 1);
            const bool more = __any_sync(0xffffffffu, differ(nM, inM) || differ(nQ, inQ));
            if (!more) break;
            inM = nM;
            inQ = nQ;
            up();
            down();
        }
        Val o;
        o.v[0] = make_float2(qa, qb);
        o.v[1] = make_float2(ma, mb);
        return o;
    }
};

// Pressure: mu_k = S_k + P_{k+1}*mu_{k+1} (top down), lam_k = mu_k + R_k + ATP_{k-1}*TERMP_{k-1}*lam_{k-1} (bottom
// up), S with the successors' parts.  Handed on: the cotangent lam*TERMP of DIM, and along i the
// cotangents R of the row carry's Q that no column of the row has taken yet (a level that this column
// solves takes them; the level above its top receives this column's share).
template <int IS, int JS>      // of the reverse walk
struct PresAdjChain : AdjChainBase<AP_PAIRS, 2, 1, JS> {
    using B = AdjChainBase<AP_PAIRS, 2, 1, JS>;
    using typename B::Rec;
    using typename B::Val;
    float2 gi, gj;             // factor of the successors' DIM in i and in j
    __device__ __forceinline__ void init(const KArgs &a, int lane) {
        this->lines(a, lane);
        const int l = min(lane, a.ks / 2 - 1);
        const float za = a.dzk[2 * l], zb = a.dzk[2 * l + 1];
        gi = make_float2(a.dyk * za / a.dxk, a.dyk * zb / a.dxk);
        // DPM_jm enters with +, DPM_jp with - (the reference's sign, :853-854)
        const float sg = (JS == -1) ? 1.0f : -1.0f;
        gj = make_float2(sg * (a.dxk * za / a.dyk), sg * (a.dxk * zb / a.dyk));
    }
    __device__ __forceinline__ Val step(const Rec &r, const Val &vI, const float2 (&vJ)[1]) const {
        const float4 x = r.f[0], y = r.f[1];
        const unsigned lA = y.y != 0.0f, lB = y.w != 0.0f;
        float sa = 0.0f, sb = 0.0f, ra = 0.0f, rb = 0.0f;
        add_if(sa, x.x, fmaf(vI.v[0].x, gi.x, vJ[0].x * gj.x), lA);
        add_if(sb, x.z, fmaf(vI.v[0].y, gi.y, vJ[0].y * gj.y), lB);
        add_if(ra, vI.v[1].x, 0.0f, lA);
        add_if(rb, vI.v[1].y, 0.0f, lB);
        float mb = sb, ma = fmaf(x.y, mb, sa), la = 0.0f, lb = 0.0f, inM = 0.0f, inL = 0.0f;
        auto down = [&]() {
            mb = fmaf(x.w, inM, sb);
            ma = fmaf(x.y, mb, sa);
        };
        auto up = [&]() {
            add_if(la, y.x * inL, ma + ra, lA);
            add_if(lb, y.z * la, mb + rb, lB);
        };
        up();
#pragma unroll
        for (int n = 0; n < ROUNDS_PRESS; ++n) {
            inM = __shfl_down_sync(0xffffffffu, ma, 1);
            inL = __shfl_up_sync(0xffffffffu, lb, 1);
            down();
            up();
        }
        for (;;) {
            const float nM = __shfl_down_sync(0xffffffffu, ma, 1), nL = __shfl_up_sync(0xffffffffu, lb, 1);
            const bool more = __any_sync(0xffffffffu, differ(nM, inM) || differ(nL, inL));
            if (!more) break;
            inM = nM;
            inL = nL;
            down();
            up();
        }
        Val o;
        o.v[0] = make_float2(la * y.y, lb * y.w);
        o.v[1] = make_float2(fmaf(y.x, inL, vI.v[1].x), fmaf(y.z, la, vI.v[1].y));
        if (lA) o.v[1].x = 0.0f;
        if (lB) o.v[1].y = 0.0f;
        return o;
    }
};

// IS, JS of the forward sweep; the chain walks the other way
template <int COMP>
__global__ void __cluster_dims__(CH_CL, 1, 1) __launch_bounds__(CH_THREADS, 2)
    k_adj_mom_chain(KArgs a, SweepGeom g, ChainBufs b, int it, float *lq, float *mu) {
    __shared__ ChainSmem<CH_SR, 1> sm;
    constexpr int PH = COMP == 0 ? PH_U : (COMP == 1 ? PH_V : PH_W), SR = CH_SR, M = CH_M, CL = CH_CL;
    for (unsigned q = threadIdx.x; q < sizeof(sm.ring) / 8; q += CH_THREADS) sm.ring[q] = 0ull;
    int is, js;
    mom_dir<COMP>(it, is, js);
    MomAdjChain<1> f;
    MomAdjChain<-1> n;
    f.F[0] = n.F[0] = lq;
    f.F[1] = n.F[1] = mu;
    if (is == -1) {
        if (js == -1) run_chain<MomAdjChain<1>, PH, SR, M, CL, 1, 1>(a, g, b, sm, f);
        else run_chain<MomAdjChain<-1>, PH, SR, M, CL, 1, -1>(a, g, b, sm, n);
    } else {
        if (js == -1) run_chain<MomAdjChain<1>, PH, SR, M, CL, -1, 1>(a, g, b, sm, f);
        else run_chain<MomAdjChain<-1>, PH, SR, M, CL, -1, -1>(a, g, b, sm, n);
    }
}

template <int IS, int JS>
__device__ __forceinline__ void run_pres_adj(const KArgs &a, const SweepGeom &g, const ChainBufs &b,
                                             ChainSmem<CH_SR, 2> &sm, float *ldim) {
    PresAdjChain<IS, JS> job;
    job.F[0] = ldim;
    run_chain<PresAdjChain<IS, JS>, PH_PRESSURE, CH_SR, CH_M, CH_CL, IS, JS>(a, g, b, sm, job);
}
__global__ void __cluster_dims__(CH_CL, 1, 1) __launch_bounds__(CH_THREADS, 2)
    k_adj_press_chain(KArgs a, SweepGeom g, ChainBufs b, int it, float *ldim) {
    __shared__ ChainSmem<CH_SR, 2> sm;
    for (unsigned q = threadIdx.x; q < sizeof(sm.ring) / 8; q += CH_THREADS) sm.ring[q] = 0ull;
    int is, js;
    sweep_dir_of(it, is, js);
    if (is == -1) {
        if (js == -1) run_pres_adj<1, 1>(a, g, b, sm, ldim);
        else run_pres_adj<1, -1>(a, g, b, sm, ldim);
    } else {
        if (js == -1) run_pres_adj<-1, 1>(a, g, b, sm, ldim);
        else run_pres_adj<-1, -1>(a, g, b, sm, ldim);
    }
}

// Launch set of the reverse sweeps: the solver's arguments with a unit list, counters and epochs of their
// own (the recomputation of the next segment uses the context's at the same time), the sweeps'
// geometry seen from the other end, the grids.
struct RevChains {
    KArgs a;
    ChainBufs b;
    AdjChain h;
    int grid[8];
};
inline SweepGeom reversed(const KArgs &a, SweepGeom g) {
    g.ia = a.nii + 2 - g.ia - g.ni;
    g.ja = a.njj + 2 - g.ja - g.nj;
    return g;
}
inline int sweep_blocks(const SweepGeom &g) { return (int)(((long long)g.ni * g.nj + AC_BLOCK - 1) / AC_BLOCK); }

template <int COMP>
void launch_adj_mom(const RevChains &r, const AdjArgs &d, const SweepGeom &g, cudaStream_t st) {
    if (g.ni <= 0 || g.nj <= 0) return;
    constexpr int PH = COMP == 0 ? PH_U : (COMP == 1 ? PH_V : PH_W);
    k_adj_mom_terms<COMP><<<sweep_blocks(g), AC_BLOCK * 32, 0, st>>>(r.a, d, g, r.h);
    k_adj_mom_chain<COMP><<<r.grid[PH], CH_THREADS, 0, st>>>(r.a, reversed(r.a, g), r.b, d.it,
                                                           r.h.plane + PL_LQ * r.h.fsz, r.h.plane + PL_MU * r.h.fsz);
    k_adj_mom_rest<COMP><<<sweep_blocks(g), AC_BLOCK * 32, 0, st>>>(r.a, d, g, r.h);
}
inline void launch_adj_pressure(const RevChains &r, const AdjArgs &d, const SweepGeom &g, cudaStream_t st) {
    if (g.ni <= 0 || g.nj <= 0) return;
    const int rows = std::max(1, 256 / r.a.ks);
    k_adj_press_terms<<<(r.a.ncols + rows - 1) / rows, dim3(r.a.ks, rows), 0, st>>>(r.a, d, r.h);
    k_adj_press_chain<<<r.grid[PH_PRESSURE], CH_THREADS, 0, st>>>(r.a, reversed(r.a, g), r.b, d.it, d.lam[L_DIV]);
}
