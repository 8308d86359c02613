// Fused shifted BiCGStab iteration with on-device scalars and seed switching.
//
// One iteration is five launches, each reading the device-resident scalars, so
// an iteration (or a CUDA graph of many) needs no host round trip:
//   K1 seed_s     s = (A + sigma_s I) p_s, (r^,s) fused
//   K2 seed_q     alpha; q = r_{k-1} - alpha s
//   K3 seed_y     y = (A + sigma_s I) q, (q,q), (q,y) fused
//   K4 seed_upd   omega; r_k = q - omega y ; (r,r), (r^,r); beside it every
//                 shift's recurrence and coefficients
//   K5 shifts     beta, the convergence test and the decision to switch; x_s,
//                 p_s and every unconverged shift's x_j, p_j in one pass
//                 (incremental mode) or the update of every system's
//                 coefficients in the Krylov basis (deferred mode); r_k
//                 rescaled on a switch
// After a switch in the deferred mode the new seed's p is formed from the
// basis by a launch of its own.
// Reference: src/solver_dynamic.c:147-381 (seed step :156-210, shift loop
// :239-256, convergence test :278-303, seed switch :312-359).
#include <vector>

#include "hbk_device.cuh"

using namespace hbk;

namespace {

// Scalar arithmetic of the recurrences is written with explicit round-to-nearest
// operations so no multiply-add is contracted: the recurrences then round
// exactly as the reference's C does for the same inputs.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }

struct Ctx {
    hbk_matrix A;
    hbk_vectors v;
    hbk_shifts sh;
    // partial sums that each step leaves behind (K1, K3, K4; the blocks of K5)
    unsigned np_s, np_y, np_r, np_p;
};

__device__ __forceinline__ size_t ldn(unsigned n) { return ((size_t)n + 31) / 32 * 32; }

// sets of partial sums: (r^,s); (q,q), (q,y); (r,r), (r^,r); (r^, rescaled r) after a switch
enum { P_RS, P_QQ, P_QY, P_RR, P_RRH, P_RRS };
__device__ __forceinline__ double *parts(const Ctx &c, int set) { return c.sh.partials + (size_t)set * HBK_MAX_GRID; }

__device__ __forceinline__ const double *seed_p(const Ctx &c, int seed) {
    return c.v.deferred ? c.v.ps : c.v.P + (size_t)seed * ldn(c.v.n);
}
__device__ __forceinline__ double *vec_r_old(const Ctx &c, const hbk_cur &u) {
    return c.v.deferred ? c.v.V + (size_t)u.slot_r_old * ldn(c.v.n) : c.v.rbuf[(u.k - 1) & 1];
}
__device__ __forceinline__ double *vec_r_new(const Ctx &c, const hbk_cur &u) {
    return c.v.deferred ? c.v.V + (size_t)(u.slots + 1) * ldn(c.v.n) : c.v.rbuf[u.k & 1];
}
__device__ __forceinline__ double *vec_q(const Ctx &c, const hbk_cur &u) {
    return c.v.deferred ? c.v.V + (size_t)u.slots * ldn(c.v.n) : c.v.q;
}
// (an L2 load: in a persistent launch another CTA wrote it in an earlier step)
__device__ __forceinline__ hbk_cur load_cur(const hbk_scalars *sc) {
    const int4 a = __ldcg(reinterpret_cast<const int4 *>(&sc->cur));
    const int4 b = __ldcg(reinterpret_cast<const int4 *>(&sc->cur) + 1);
    hbk_cur u;
    u.k = a.x, u.seed = a.y, u.slots = a.z, u.slot_r_old = a.w;
    u.active = b.x, u.rr_pend = b.y, u.n_done = b.z, u.max_sigma = b.w;
    return u;
}

// ---------------------------------------------------------------------------
// Scalars between the steps.
//
// A kernel boundary inside a graph costs 0.5..1.3 us on GB300; a fence, a
// ticket and a last block that sums and divides cost 4..8 us at the end of
// every step, and the whole scalar stage of an iteration in one last block
// 20 us.  (A grid barrier inside one persistent kernel costs 1..1.7 us too.)
// So no step has a last block.  A step's blocks leave one partial sum each,
// and every block of the next step sums them again in the same fixed order
// (so all blocks get the same bits) while its first loads are in flight.  The
// shifts' recurrences need alpha and omega only: one extra block of K4
// computes them beside the vector work.  The decisions that need (r, r) and
// beta (convergence, the switch) are made by every block of K5 for itself;
// one extra block of K5 records them, replays the histories after a switch
// and advances the iteration.  Measured, whole solves, with the slice pipeline
// of SellRows and early launches: n = 512, 6 shifts 1788 -> 974 us; 32^3, 16
// shifts 5.61 -> 3.22 ms; 97 k rows, 24 shifts 26.4 -> 18.2 ms; 128^3, 32
// shifts 72.9 -> 61.1 ms; 256^3, 64 shifts 805 -> 711 ms (with the changes made
// elsewhere since: 0.79, 2.78, 15.8, 56.2 and 651 ms).
//
// The order of a dot product's sum is part of a solve's outcome: it moves what
// is left of every residual below the tolerance at which the solve stops, and
// results that cancel (the shift gradient -w lambda . x: digits lost by the
// cosine of the two) show that in their ninth digit.  So the order follows from
// n and the number of SMs alone, not from the blocks a kernel is launched in:
// NT threads to a set of rows, at most 6 sets per SM for the products of SELL-32
// matrices (TILE 6, MERGE 4, HYB its lists' grid) and DOT_VEC for K4; a thread
// adds its rows in ascending order, a tree adds the NT, and NT threads and the
// same tree add the sets.  Blocks fewer or larger than a set carry several: K1
// and K3 (3 blocks per SM) two, their NT-row steps in turn, K4 up to four.
// (After a switch (r^, r) is summed once over K5's blocks.)

// The vector kernels (K2, K4, K5) run one block per SM, of as many threads as
// that takes (blockDim.x, 128..1024; K4: set_grid): the sums at a block's start
// then cost an SM one pass, not one per resident block.
constexpr int DOT_VEC = 4, DOT_ROWS = 512;  // K4: sets per SM at most, rows per set while there are fewer

constexpr int MAXW = 32;  // warps of the largest block

// Sum of np partials per set over the block, in a fixed order: the totals are
// valid in warp 0 (every lane).  NA = 2: both sets at once.  FP64 adds cost 64
// clocks per warp and SM quarter whatever the active lanes, so warps without
// partials take no part.  load() issues the loads with the kernel's others;
// total() needs 2 MAXW doubles and has one barrier.
template <int NA>
struct PartSum {
    double x, y;
    unsigned nw;
    __device__ __forceinline__ void load(const double *p0, const double *p1, unsigned np) {
        const unsigned t = threadIdx.x;
        nw = min(min(blockDim.x >> 5, (unsigned)NW), (np + 31) >> 5);
        x = y = 0.0;
        if (t < nw * 32 && t < np) {
            x = __ldcg(p0 + t);
            if (NA == 2) y = __ldcg(p1 + t);
            for (unsigned i = t + nw * 32; i < np; i += nw * 32) {
                x += __ldcg(p0 + i);
                if (NA == 2) y += __ldcg(p1 + i);
            }
        }
    }
    __device__ __forceinline__ double2 total(double *sh) {
        const unsigned w = threadIdx.x >> 5, l = threadIdx.x & 31;
        if (w < nw) {
            x = NA == 2 ? warp_sum_pair(x, y) : warp_sum(x);
            if (NA == 2 ? (l & 15) == 0 : l == 0) sh[(l >> 4) * MAXW + w] = x;
        }
        __syncthreads();
        double2 r = make_double2(0.0, 0.0);
        if (w == 0) {
            double v = 0.0;
            if ((l & 15) < nw && (NA == 2 || l < 16)) v = sh[(l >> 4) * MAXW + (l & 15)];
#pragma unroll
            for (unsigned k = 8; k; k >>= 1)
                if (k < nw) v += __shfl_xor_sync(0xffffffffu, v, k);
            r.x = __shfl_sync(0xffffffffu, v, 0);
            if (NA == 2) r.y = __shfl_sync(0xffffffffu, v, 16);
        }
        return r;
    }
};

// This block's share of one or two dot products into its partial-sum slot.
__device__ __forceinline__ void store_part(double v, double *sh, double *out) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned nw = blockDim.x >> 5;
        double t = threadIdx.x < nw ? sh[threadIdx.x] : 0.0;
#pragma unroll
        for (unsigned k = 16; k; k >>= 1)
            if (k < nw) t += __shfl_xor_sync(0xffffffffu, t, k);
        if (threadIdx.x == 0) *out = t;
    }
}
// Two sums of every 256 threads (NW warps) of the block, where `here`; sh: 2 MAXW
__device__ __forceinline__ void store_part2(double2 v, double *sh, double *out_x, double *out_y, bool here = true) {
    const unsigned w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const double x = warp_sum_pair(v.x, v.y);
    if ((l & 15) == 0) sh[(l >> 4) * MAXW + w] = x;
    __syncthreads();
    if (w % NW == 0) {
        double t = (l & 15) < NW ? sh[(l >> 4) * MAXW + w + (l & 15)] : 0.0;
#pragma unroll
        for (unsigned k = NW / 2; k; k >>= 1) t += __shfl_xor_sync(0xffffffffu, t, k);
        if (here && l == 0) *out_x = t;
        if (here && l == 16) *out_y = t;
    }
}
// and two sums each of two sets (v0, v1) of a block of 256 threads, v1's
// `after` entries behind v0's; sh: 4 MAXW
__device__ __forceinline__ void store_part4(double2 v0, double2 v1, double *sh, double *out_x, double *out_y,
                                            unsigned after) {
    const unsigned w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const double x = warp_sum_pair(v0.x, v0.y), y = warp_sum_pair(v1.x, v1.y);
    if ((l & 15) == 0) {
        sh[(l >> 4) * MAXW + w] = x;
        sh[(2 + (l >> 4)) * MAXW + w] = y;
    }
    __syncthreads();
    if (w < 2) {
        double t = (l & 15) < NW ? sh[(2 * w + (l >> 4)) * MAXW + (l & 15)] : 0.0;
#pragma unroll
        for (unsigned k = NW / 2; k; k >>= 1) t += __shfl_xor_sync(0xffffffffu, t, k);
        if (l == 0) out_x[w * after] = t;
        if (l == 16) out_y[w * after] = t;
    }
}
// shared memory of a body is used again by the next virtual block of the CTA
template <class G>
__device__ __forceinline__ void body_begin() {
    if constexpr (!G::hw) __syncthreads();
    else let_next_start();
}
// nothing that an earlier kernel of the iteration writes is read before this
template <class G>
__device__ __forceinline__ void body_ready() {
    if constexpr (G::hw) wait_previous();
}

// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(NT) k_init(Ctx c, int seed, double tol, int switching, int inline_ps) {
    hbk_scalars *sc = c.sh.sc;
    const int m = c.sh.m, kcap = c.sh.kcap;
    for (int j = threadIdx.x; j < m; j += NT) {
        double *pij = c.sh.pi + (size_t)j * kcap;
        pij[0] = 1.0;
        if (kcap > 1) pij[1] = 1.0;
        c.sh.eta[j] = 0.0;
        c.sh.zeta[j] = 1.0;
        c.sh.done[j] = 0;
        c.sh.conv_k[j] = 0;
    }
    for (int i = threadIdx.x; i < 8; i += NT) c.sh.counters[i] = 0;
    if (threadIdx.x == 0) {
        c.sh.a_hist[0] = 1.0;
        c.sh.b_hist[0] = 0.0;
        c.sh.w_hist[0] = 0.0;
        const double bb = sc->bb;  // written by the (b,b) reduction launched just before
        sc->rr_hat = bb;
        sc->rr_hat_old = bb;
        sc->rr = bb;
        sc->alpha = sc->omega = sc->beta = 0.0;
        sc->tol = tol;
        sc->k = 1;
        sc->seed = seed;
        sc->n_done = 0;
        sc->status = 0;
        sc->n_sw = 0;
        sc->loops = 0;
        sc->flush_rows = 0.0;
        sc->max_sigma = seed;
        sc->m = m;
        sc->kcap = kcap;
        sc->slots = 1;
        sc->slot_r_old = 0;
        sc->slot_cap = c.v.slot_cap;
        sc->need_ps = 0;
        sc->rr_pend = 0;
        sc->switching = switching;
        sc->inline_ps = inline_ps;
        sc->finished = (m <= 0 || kcap <= 1) ? 1 : 0;
        if (bb == 0.0) {  // b = 0: x = 0 solves every system exactly
            sc->finished = 1;
            sc->n_done = m;
        }
        sc->cur.active = 0;
    }
}

// deferred mode: X = 0, Xc = 0, Pc[j][0] = 1 (p_j = b = basis slot 0), own = (0, 0)
__global__ void __launch_bounds__(NT) k_init_coef(Ctx c) {
    const int m = c.sh.m, cap = c.v.slot_cap;
    const size_t tot = (size_t)m * cap;
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < tot; i += (size_t)gridDim.x * NT) {
        c.v.Xc[i] = 0.0;
        c.v.Pc[i] = (i % cap == 0) ? 1.0 : 0.0;
    }
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < (size_t)m; i += (size_t)gridDim.x * NT) {
        c.v.own[2 * i] = 0.0;
        c.v.own[2 * i + 1] = 0.0;
        c.sh.lslot[i] = 1;
    }
}

// ---------------------------------------------------------------------------
// K1: s = (A + sigma_s I) p_s and (r^, s).  Block 0 copies the scalars that
// the iteration's other kernels read (hbk_cur).
// SELL-32: block b carries the sets b and b + (blocks), its NT-row steps in turn.
template <int FMT, class G>
__device__ __forceinline__ void seed_s_body(const Ctx &c, const G &g) {
    __shared__ double red[2 * MAXW];
    hbk_scalars *sc = c.sh.sc;
    body_begin<G>();
    SpmvRows<FMT, G> rows(c.A, g);
    rows.start();
    body_ready<G>();
    const int fin_flag = __ldcg(&sc->finished), seed = __ldcg(&sc->seed);
    if (g.b() == 0 && threadIdx.x == 0) {
        hbk_cur u;
        u.k = __ldcg(&sc->k), u.seed = seed, u.slots = __ldcg(&sc->slots), u.slot_r_old = __ldcg(&sc->slot_r_old);
        u.active = fin_flag == 0, u.rr_pend = __ldcg(&sc->rr_pend);
        u.n_done = __ldcg(&sc->n_done), u.max_sigma = __ldcg(&sc->max_sigma);
        sc->cur = u;
    }
    if (fin_flag) return;
    const double sig = c.sh.sigma[seed];
    const double *__restrict__ ps = seed_p(c, seed);
    const double *__restrict__ rh = c.v.r_hat;
    double *__restrict__ s = c.v.s;
    const bool folded = c.v.sval_shift != nullptr;  // the product already holds sigma p
    double acc = 0.0, alt = 0.0;
    bool odd = false;
    auto pre = [&](unsigned r) { return HBK_LD(G, rh, r); };
    auto epi = [&](unsigned r, double ax, double hr) {
        const double sv = folded ? ax : fma(sig, HBK_LD(G, ps, r), ax);
        s[r] = sv;
        acc = fma(hr, sv, acc);
    };
    auto turn = [&] {
        const double t = acc;
        acc = alt, alt = t, odd = !odd;
    };
    rows.run(ps, pre, epi, turn);
    double *out = parts(c, P_RS) + g.b();
    if constexpr (decltype(rows)::turns) {
        if (odd) turn();
        store_part2(make_double2(acc, alt), red, out, out + g.nb());
    } else {
        store_part(acc, red, out);
    }
}
template <int FMT>
__global__ void __launch_bounds__(NT) k_seed_s(Ctx c) { seed_s_body<FMT>(c, HwGrid()); }
template <>
__global__ void __launch_bounds__(NT, HBK_SELL_MINB) k_seed_s<HBK_FMT_SELL>(Ctx c) {
    seed_s_body<HBK_FMT_SELL>(c, HwGrid());
}
template <>
__global__ void __launch_bounds__(NT, HBK_SELL_MINB) k_seed_s<HBK_FMT_SELLN>(Ctx c) {
    seed_s_body<HBK_FMT_SELLN>(c, HwGrid());
}
template <>
__global__ void __launch_bounds__(NT, HBK_HYBW_MINB) k_seed_s<HBK_FMT_HYBW>(Ctx c) {
    seed_s_body<HBK_FMT_HYBW>(c, HwGrid());
}
template <>
__global__ void __launch_bounds__(NT, HBK_HYB_MINB) k_seed_s<HBK_FMT_HYB>(Ctx c) {
    seed_s_body<HBK_FMT_HYB>(c, HwGrid());
}

// K2: alpha = (r^,r) / (r^,s); q = r_{k-1} - alpha s (deferred mode: q is a
// basis slot; its max |q| is kept for the flush)
template <class G>
__device__ __forceinline__ void seed_q_body(const Ctx &c, const G &g) {
    __shared__ double red[2 * MAXW], s_a;
    __shared__ unsigned long long smx[MAXW];
    hbk_scalars *sc = c.sh.sc;
    body_begin<G>();
    const unsigned n = c.v.n;
    const double *__restrict__ s = c.v.s;
    size_t i = g.b() * (size_t)blockDim.x + threadIdx.x;
    body_ready<G>();
    const hbk_cur u = load_cur(sc);
    PartSum<1> rs;
    rs.load(parts(c, P_RS), nullptr, c.np_s);
    const double rr_hat = __ldcg(&sc->rr_hat);
    double si = i < n ? HBK_LD(G, s, i) : 0.0;
    if (!u.active) return;
    const double *__restrict__ ro = vec_r_old(c, u);
    double *__restrict__ q = vec_q(c, u);
    double ri = i < n ? HBK_LD(G, ro, i) : 0.0;
    double2 t = rs.total(red);
    t.y = rr_hat;
    if (u.rr_pend) {
        __syncthreads();
        PartSum<1> rr;
        rr.load(parts(c, P_RRS), nullptr, c.np_p);
        t.y = rr.total(red).x;
    }
    if (threadIdx.x < 32) {
        const double a = dvd(t.y, t.x);
        if (threadIdx.x == 0) {
            s_a = a;
            if (g.b() == 0) {
                sc->rs = t.x;
                sc->rr_hat_old = t.y;
                c.sh.a_hist[u.k] = a;
                sc->alpha = a;
                if (!fin(a)) {
                    sc->status = __ldcg(&sc->status) | HBK_ST_BREAKDOWN;
                    sc->finished = 1;
                }
            }
        }
    } else if (threadIdx.x == 32 && g.b() == 0) {  // for the recurrences in K4
        sc->ba = dvd(__ldcg(c.sh.b_hist + u.k - 1), __ldcg(c.sh.a_hist + u.k - 1));
    }
    __syncthreads();
    const double a = s_a;
    if (!fin(a)) return;
    unsigned long long mx = 0;
    const size_t step = (size_t)g.nb() * blockDim.x;
    while (i < n) {
        const size_t in = i + step;  // the next element's loads go before this one's store
        const double sn = in < n ? HBK_LD(G, s, in) : 0.0, rnx = in < n ? HBK_LD(G, ro, in) : 0.0;
        const double qi = fma(-a, si, ri);
        q[i] = qi;
        const unsigned long long b = abs_bits(qi);
        mx = b > mx ? b : mx;
        si = sn, ri = rnx, i = in;
    }
    if (c.v.slot_max) block_max_to(mx, smx, c.v.slot_max + (size_t)u.slots * HBK_SLOT_SPREAD);
}
__global__ void __launch_bounds__(1024) k_seed_q(Ctx c) { seed_q_body(c, HwGrid()); }

// K3: y = (A + sigma_s I) q, (q,q) and (q,y).  SELL-32: the sums of two sets take
// the registers of an eighth entry ahead (256^3: 294 us; with it they spill, 367;
// the other set's in shared memory 321, with seven ahead 340).
template <int FMT, class G>
__device__ __forceinline__ void seed_y_body(const Ctx &c, const G &g) {
    __shared__ double red[4 * MAXW];
    body_begin<G>();
    SpmvRows<FMT, G, 7> rows(c.A, g);
    rows.start();
    body_ready<G>();
    const hbk_cur u = load_cur(c.sh.sc);
    if (!u.active || !fin(__ldcg(&c.sh.sc->alpha))) return;
    const double sig = c.sh.sigma[u.seed];
    const double *__restrict__ q = vec_q(c, u);
    double *__restrict__ y = c.v.y;
    const bool folded = c.v.sval_shift != nullptr;  // the product already holds sigma q
    constexpr bool turns = decltype(rows)::turns;
    double2 acc = make_double2(0.0, 0.0), alt = acc;
    bool odd = false;
    // (as HBK_LD: 327 us at 256^3)
    const double *const own = G::hw ? settle(q) : q;
    auto pre = [&](unsigned r) { return G::hw ? ld_settled(own + r) : __ldcg(q + r); };
    auto epi = [&](unsigned r, double ax, double qr) {
        const double yv = folded ? ax : fma(sig, qr, ax);
        y[r] = yv;
        acc.x = fma(qr, qr, acc.x);
        acc.y = fma(qr, yv, acc.y);
    };
    auto turn = [&] {
        const double2 t = alt;
        alt = acc;
        acc = t, odd = !odd;
    };
    rows.run(q, pre, epi, turn);
    double *qq = parts(c, P_QQ) + g.b(), *qy = parts(c, P_QY) + g.b();
    if (turns && odd) turn();
    if (turns && c.np_y > g.nb()) store_part4(acc, alt, red, qq, qy, g.nb());
    else store_part2(acc, red, qq, qy);
}
template <int FMT>
__global__ void __launch_bounds__(NT) k_seed_y(Ctx c) { seed_y_body<FMT>(c, HwGrid()); }
template <>
__global__ void __launch_bounds__(NT, HBK_SELL_MINB) k_seed_y<HBK_FMT_SELL>(Ctx c) {
    seed_y_body<HBK_FMT_SELL>(c, HwGrid());
}
template <>
__global__ void __launch_bounds__(NT, HBK_SELL_MINB) k_seed_y<HBK_FMT_SELLN>(Ctx c) {
    seed_y_body<HBK_FMT_SELLN>(c, HwGrid());
}
template <>
__global__ void __launch_bounds__(NT, HBK_HYBW_MINB) k_seed_y<HBK_FMT_HYBW>(Ctx c) {
    seed_y_body<HBK_FMT_HYBW>(c, HwGrid());
}
template <>
__global__ void __launch_bounds__(NT, HBK_HYB_MINB) k_seed_y<HBK_FMT_HYB>(Ctx c) {
    seed_y_body<HBK_FMT_HYB>(c, HwGrid());
}

// ---------------------------------------------------------------------------
// One extra block of K4: every shift's recurrence (src/solver_dynamic.c:243-253)
// and this iteration's vector coefficients but for the factor beta, which K5
// multiplies in.  Four lanes per shift: FP64 division takes 573 clocks of a
// warp, so a shift's independent quotients go side by side, in two rounds.
struct ShiftState {  // of this thread's shift: read before omega is known
    double pik1, z, e0, sj;
    bool run;
    __device__ __forceinline__ void load(const Ctx &c, const hbk_cur &u, int j0) {
        const hbk_shifts &S = c.sh;
        const int j = j0 + (int)(threadIdx.x / 4);
        pik1 = z = 1.0;
        e0 = sj = 0.0;
        run = false;
        if (j < S.m) {
            run = j == u.seed || !__ldcg(S.done + j);
            sj = S.sigma[j];
            if (j != u.seed) {
                pik1 = __ldcg(S.pi + (size_t)j * S.kcap + u.k - 1);
                z = __ldcg(S.zeta + j);
                e0 = __ldcg(S.eta + j);
            }
        }
    }
};
__device__ void shift_recurrences(const Ctx &c, const hbk_cur &u, double ak, double wk, ShiftState &st) {
    hbk_scalars *sc = c.sh.sc;
    const hbk_shifts &S = c.sh;
    const int k = u.k, seed = u.seed, m = S.m, kcap = S.kcap;
    const double c_prev = mul(__ldcg(&sc->ba), ak);
    const double sig_s = S.sigma[seed];
    const unsigned l = threadIdx.x & 31, quad = l & ~3u, part = threadIdx.x & 3;
    // (whole warps leave together: the shuffles below need all lanes)
    for (int j0 = 0; j0 + (int)(threadIdx.x & ~31u) / 4 < m; j0 += (int)blockDim.x / 4) {
        const int j = j0 + (int)(threadIdx.x / 4);
        if (j0) st.load(c, u, j0);
        const bool here = j < m;
        const bool is_seed = j == seed;
        const bool run = st.run;
        const double pik1 = st.pik1, z = st.z, e0 = st.e0, sj = here ? st.sj : sig_s;
        const double d = sub(sig_s, sj);
        const double eta = sub(mul(c_prev, e0), mul(mul(d, ak), pik1));
        const double pik = add(eta, pik1);
        const double den = sub(1.0, mul(wk, d));
        const double zn = mul(den, z);
        // round 1: pi_{k-1} / pi_k, omega_j, 1 / (pi_k zeta_k); the seed as a
        // system of its own (deferred mode): omega / alpha, alpha / omega
        double num, by;
        if (is_seed) num = part == 0 ? wk : ak, by = part == 0 ? ak : wk;
        else if (part == 0) num = pik1, by = pik;
        else if (part == 1) num = wk, by = den;
        else num = 1.0, by = mul(pik, zn);
        const double q1 = dvd(num, by);
        const double rp = __shfl_sync(0xffffffffu, q1, quad), wj = __shfl_sync(0xffffffffu, q1, quad + 1);
        const double c5 = __shfl_sync(0xffffffffu, q1, quad + 2);
        const double aj = mul(rp, ak);
        // round 2: omega_j / (pi_k zeta_{k-1}), omega_j / (alpha_j zeta pi_k), -omega_j / (alpha_j zeta pi_{k-1})
        const double azj = mul(aj, z);
        const double q2 = dvd(part == 2 ? -wj : wj, part == 0 ? mul(pik, z) : mul(azj, part == 1 ? pik : pik1));
        const double c0 = __shfl_sync(0xffffffffu, q2, quad), c2 = __shfl_sync(0xffffffffu, q2, quad + 1);
        const double c3 = __shfl_sync(0xffffffffu, q2, quad + 2);
        if (!here || part) continue;
        double *co = S.coef + (size_t)j * HBK_NCOEF;
        if (is_seed) {
            // pi = zeta = 1, shift 0.  Its x is not carried in coefficient
            // form: K5 adds alpha p_s + omega q to its row of X directly, with
            // the materialised p_s, as the reference's seed step does
            // (src/solver_dynamic.c:156-210).  In coefficient form p_s would
            // enter through s = (r_{k-1} - q) / alpha, which cancels when a
            // step makes little progress; its p coefficients stay (needed
            // after a switch).
            co[0] = co[1] = 0.0;
            co[2] = rp;  // omega / alpha
            co[3] = -rp;
            co[4] = co[5] = 1.0;
            sc->aw = wj;  // alpha / omega
            S.live[j] = __ldcg(S.done + j) ? 0 : 1;
            continue;
        }
        if (!run) {
            S.live[j] = 0;
            continue;
        }
        const double c4 = mul(rp, rp);
        // Shift breakdown (the reference never tests for it and carries the
        // inf or nan into x_j): pi_k = 0, 1 - omega_k d = 0, or any scalar of
        // the update not finite (K5 tests beta c4).  The shift stops at its
        // last finite iterate, counts as finished so the others run on, and
        // records -k.
        const bool ok = !is_zero(pik) && !is_zero(den) && fin(eta) && fin(zn) && fin(c0) && fin(aj) && fin(c2) && fin(c3) &&
                        fin(c4) && fin(c5);
        S.live[j] = ok ? 1 : 2;
        if (!ok) continue;
        S.pi[(size_t)j * kcap + k] = pik;
        S.eta[j] = eta;
        S.zeta[j] = zn;
        co[0] = c0;
        co[1] = aj;
        co[2] = c2;
        co[3] = c3;
        co[4] = c4;
        co[5] = c5;
    }
}

// K4: omega = (q,q) / (q,y); r_k = q - omega y; (r,r), (r^,r); the extra block:
// the shifts' recurrences
template <class G>
__device__ __forceinline__ void seed_update_body(const Ctx &c, const G &g) {
    __shared__ double sh[2 * MAXW], s_w;
    __shared__ unsigned long long smx[MAXW];
    hbk_scalars *sc = c.sh.sc;
    body_begin<G>();
    const unsigned n = c.v.n;
    const double *__restrict__ y = c.v.y;
    const double *__restrict__ rh = c.v.r_hat;
    const bool extra = g.extra();
    // 256 threads per set of rows
    const unsigned set = g.b() * (blockDim.x / NT) + threadIdx.x / NT, nset = c.np_r;
    const bool here = !extra && set < nset;
    size_t i = here ? set * (size_t)NT + threadIdx.x % NT : (size_t)n;
    double hi = i < n ? HBK_LD(G, rh, i) : 0.0;
    body_ready<G>();
    const hbk_cur u = load_cur(sc);
    const double ak = __ldcg(&sc->alpha);
    PartSum<2> qs;
    qs.load(parts(c, P_QQ), parts(c, P_QY), c.np_y);
    double yi = i < n ? HBK_LD(G, y, i) : 0.0;
    if (!u.active || !fin(ak)) return;
    const double *__restrict__ q = vec_q(c, u);
    double *__restrict__ rn = vec_r_new(c, u);
    double qi = i < n ? HBK_LD(G, q, i) : 0.0;
    ShiftState st;
    if (extra) st.load(c, u, 0);
    const double2 t = qs.total(sh);
    if (threadIdx.x < 32) {
        const double w = dvd(t.x, t.y);
        if (threadIdx.x == 0) {
            s_w = w;
            if (extra) {
                sc->qq = t.x;
                sc->qy = t.y;
                c.sh.w_hist[u.k] = w;
                sc->omega = w;
                if (!fin(w) || is_zero(w)) {
                    sc->status = __ldcg(&sc->status) | HBK_ST_BREAKDOWN;
                    sc->finished = 1;
                }
            }
        }
    }
    __syncthreads();
    const double w = s_w;
    if (!fin(w) || is_zero(w)) return;
    if (extra) {
        shift_recurrences(c, u, ak, w, st);
        return;
    }
    double2 acc = make_double2(0.0, 0.0);
    unsigned long long mx = 0;
    const size_t step = (size_t)nset * NT;
    while (i < n) {
        const size_t in = i + step;  // the next element's loads go before this one's store
        const double yn = in < n ? HBK_LD(G, y, in) : 0.0, hn = in < n ? HBK_LD(G, rh, in) : 0.0;
        const double qn = in < n ? HBK_LD(G, q, in) : 0.0;
        const double r = fma(-w, yi, qi);
        rn[i] = r;
        acc.x = fma(r, r, acc.x);
        acc.y = fma(hi, r, acc.y);
        const unsigned long long b = abs_bits(r);
        mx = b > mx ? b : mx;
        yi = yn, hi = hn, qi = qn, i = in;
    }
    if (c.v.slot_max) block_max_to(mx, smx, c.v.slot_max + (size_t)(u.slots + 1) * HBK_SLOT_SPREAD);  // r_k
    store_part2(acc, sh, parts(c, P_RR) + set, parts(c, P_RRH) + set, here);
}
template <int PER_SM>
__global__ void __launch_bounds__(PER_SM == 1 ? DOT_VEC * NT : 2 * NT, PER_SM) k_seed_update(Ctx c) {
    seed_update_body(c, HwGridX{1});
}

// ---------------------------------------------------------------------------
// Argmax of |1/(zeta_j pi_j)| over the systems still running after this
// iteration's test, strict '>' from 1.0, lowest index on an exact tie (the
// reference's order, src/solver_dynamic.c:278-303); run by warp 0, result in
// every lane; -1: none.
__device__ int running_argmax(const hbk_shifts &S, int seed, double bk, double rr, double thr) {
    double best = 1.0;
    int bidx = -1;
    for (int j = threadIdx.x; j < S.m; j += 32) {
        if (j == seed || __ldcg(S.live + j) != 1) continue;
        const double *co = S.coef + (size_t)j * HBK_NCOEF;
        if (!fin(mul(__ldcg(co + 4), bk))) continue;
        const double a = fabs(__ldcg(co + 5));
        if (mul(mul(a, a), rr) > thr && a > best) {
            best = a;
            bidx = j;
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
        if (oi >= 0 && (bidx < 0 || ob > best || (ob == best && oi < bidx))) {
            best = ob;
            bidx = oi;
        }
    }
    return bidx;
}

// What an iteration's end decides, the same in every block of K5.
struct StepEnd {
    double bk, bw, rr, rrh, thr, rsc;  // bw = -beta omega
    int ok;      // beta is finite
    int n_done;  // finished systems, this iteration's included
    int sw, t;   // seed switch to system t; rsc = 1 / (zeta_t pi_t)
};

// What step_end reads, loaded with the kernel's other first loads.
struct StepLoads {
    PartSum<2> rs;
    double aw, rho, tol, bb, c4, c5;
    int live, switching;
    __device__ __forceinline__ void load(const Ctx &c) {
        const hbk_scalars *sc = c.sh.sc;
        rs.load(parts(c, P_RR), parts(c, P_RRH), c.np_r);
        aw = __ldcg(&sc->aw), rho = __ldcg(&sc->rr_hat_old), tol = __ldcg(&sc->tol), bb = __ldcg(&sc->bb);
        switching = __ldcg(&sc->switching);
        live = 0;
        c4 = c5 = 1.0;
        if ((int)threadIdx.x < c.sh.m) {
            live = __ldcg(c.sh.live + threadIdx.x);
            const double2 cc =
                __ldcg(reinterpret_cast<const double2 *>(c.sh.coef + (size_t)threadIdx.x * HBK_NCOEF + 4));
            c4 = cc.x;
            c5 = cc.y;
        }
    }
};

// beta from K4's partial sums, the convergence test on the recursive residual
// (src/solver_dynamic.c:278-303) and the decision to switch (:312-326).
// Every thread returns the same.
__device__ __forceinline__ StepEnd step_end(const Ctx &c, const hbk_cur &u, double wk, StepLoads &ld, double *sh) {
    __shared__ double s_bk, s_bw, s_rr, s_rrh, s_thr, s_rsc;
    __shared__ int s_t;
    const hbk_shifts &S = c.sh;
    const int m = S.m;
    int live = ld.live;
    double c4 = ld.c4, c5 = ld.c5;
    const double aw = ld.aw, rho = ld.rho, tol = ld.tol, bb = ld.bb;
    const int switching = ld.switching;
    PartSum<2> &rs = ld.rs;
    const double2 t = rs.total(sh);
    if (threadIdx.x < 32) {
        const double bk = mul(aw, dvd(t.y, rho));
        if (threadIdx.x == 0) s_bk = bk, s_bw = -mul(bk, wk), s_rr = t.x, s_rrh = t.y;
    } else if (threadIdx.x < 64) {  // (one warp: every other would pay for the two operations too)
        const double thr = mul(mul(tol, tol), bb);
        if (threadIdx.x == 32) s_thr = thr;
    }
    __syncthreads();
    StepEnd e;
    e.bk = s_bk;
    e.rr = s_rr;
    e.rrh = s_rrh;
    e.ok = fin(e.bk);
    e.sw = 0;
    e.t = u.max_sigma;
    e.rsc = 1.0;
    e.n_done = u.n_done;
    e.thr = s_thr;
    e.bw = s_bw;
    if (!e.ok) return e;
    int seed_done = 0;
    for (int j0 = 0; j0 < m; j0 += (int)blockDim.x) {
        const int j = j0 + (int)threadIdx.x;
        if (j0 && j < m) {
            live = __ldcg(S.live + j);
            c4 = __ldcg(S.coef + (size_t)j * HBK_NCOEF + 4);
            c5 = __ldcg(S.coef + (size_t)j * HBK_NCOEF + 5);
        }
        int now = 0;
        if (j < m && live) {
            if (j == u.seed) now = e.rr <= e.thr;
            else now = live == 2 || !fin(mul(c4, e.bk)) || mul(mul(c5, c5), e.rr) <= e.thr;
        }
        seed_done |= j == u.seed && (now || !live);
        e.n_done += __syncthreads_count(now);
    }
    if (!switching) return e;
    if (!__syncthreads_or(seed_done) || e.n_done >= m) return e;
    if (threadIdx.x < 32) {
        const int b = running_argmax(S, u.seed, e.bk, e.rr, e.thr);
        if (threadIdx.x == 0) {
            s_t = b >= 0 ? b : u.max_sigma;
            s_rsc = __ldcg(S.coef + (size_t)s_t * HBK_NCOEF + 5);  // 1 / (zeta_t pi_t)
        }
    }
    __syncthreads();
    e.sw = 1;
    e.t = s_t;
    e.rsc = s_rsc;
    return e;
}

// The extra block of K5: records the iteration, replays the histories after a
// switch (src/solver_dynamic.c:312-359) and advances the iteration.
__device__ void record_step(const Ctx &c, const hbk_cur &u, const StepEnd &e) {
    hbk_scalars *sc = c.sh.sc;
    const hbk_shifts &S = c.sh;
    const int k = u.k, seed = u.seed, m = S.m, kcap = S.kcap;
    int nfail = 0, nact = 0;
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
        const int live = __ldcg(S.live + j);
        if (!live) continue;
        const double *co = S.coef + (size_t)j * HBK_NCOEF;
        const double a = j == seed ? 1.0 : __ldcg(co + 5);
        if (j != seed && (live == 2 || !fin(mul(__ldcg(co + 4), e.bk)))) {
            S.done[j] = 1;
            S.conv_k[j] = -k;
            nfail = 1;
            continue;
        }
        if (j != seed) nact++;
        if (mul(mul(a, a), e.rr) <= e.thr) {
            S.done[j] = 1;
            S.conv_k[j] = k;
        }
    }
    __shared__ int s_nact;
    if (threadIdx.x == 0) s_nact = 0;
    nfail = __syncthreads_or(nfail);
    if (nact) atomicAdd(&s_nact, nact);
    __syncthreads();
    int top = -1;
    if (threadIdx.x < 32) top = running_argmax(S, seed, e.bk, e.rr, e.thr);
    if (threadIdx.x == 0) {
        if (k < kcap) {
            S.rr_hist[k] = e.rr;
            S.act_hist[k] = s_nact;
        }
        S.b_hist[k] = e.bk;
        sc->beta = e.bk;
        sc->rr = e.rr;
        sc->rr_hat = e.rrh;
        sc->rr_pend = e.sw;
        sc->n_done = e.n_done;
        if (top >= 0) sc->max_sigma = top;
        int status = __ldcg(&sc->status);
        if (nfail) status |= HBK_ST_SHIFT_FAIL;
        int finished = e.n_done >= m || k + 1 >= kcap;
        if (e.sw) {
            const int n_sw = __ldcg(&sc->n_sw);
            if (n_sw < m) {
                S.sw_k[n_sw] = k;
                S.sw_seed[n_sw] = e.t;
            }
            sc->n_sw = n_sw + 1;
            sc->seed = e.t;
        }
        if (c.v.deferred) {
            const int slots = u.slots + (e.sw ? 3 : 2);
            sc->slot_r_old = slots - 1;  // r_k (after a switch the rescaled r_k)
            sc->slots = slots;
            if (e.sw) {
                sc->need_ps = 1;
                if (!__ldcg(&sc->inline_ps)) {
                    status |= HBK_ST_NEED_PS;
                    finished = 1;  // the host has the new seed's p formed and resumes
                }
            }
            if (!(e.n_done >= m || k + 1 >= kcap) && slots + 3 > __ldcg(&sc->slot_cap)) {
                status |= HBK_ST_BASIS_FULL;
                finished = 1;  // the host flushes the basis and resumes
            }
        }
        sc->status = status;
        sc->k = k + 1;
        sc->finished = finished;
    }
    if (!e.sw) return;
    // rescale the seed history, replay eta/pi/zeta of every running shift
    // relative to sigma_t
    __syncthreads();
    const int t = e.t;
    const double sig_s = S.sigma[seed], sig_t = S.sigma[t];
    const double *pit = S.pi + (size_t)t * kcap;
    const double dst = sub(sig_s, sig_t);
    for (int i = 1 + threadIdx.x; i <= k; i += blockDim.x) {
        const double rp = dvd(__ldcg(pit + i - 1), __ldcg(pit + i));
        S.a_hist[i] = mul(rp, __ldcg(S.a_hist + i));
        S.b_hist[i] = mul(mul(rp, rp), i == k ? e.bk : __ldcg(S.b_hist + i));
        const double wi = __ldcg(S.w_hist + i);
        S.w_hist[i] = dvd(wi, sub(1.0, mul(wi, dst)));
    }
    __syncthreads();
    for (int i = 1 + threadIdx.x; i <= k; i += blockDim.x) S.ratio[i] = mul(dvd(S.b_hist[i - 1], S.a_hist[i - 1]), S.a_hist[i]);
    __syncthreads();
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
        if (S.done[j] || j == t) {
            S.eta[j] = 0.0;
            S.zeta[j] = 1.0;
            continue;
        }
        double *pij = S.pi + (size_t)j * kcap;
        const double d = sub(sig_t, S.sigma[j]);
        double eta = 0.0, z = 1.0, pprev = __ldcg(pij);
        for (int i = 1; i <= k; i++) {
            eta = sub(mul(S.ratio[i], eta), mul(mul(d, S.a_hist[i]), pprev));
            const double pc = add(eta, pprev);
            pij[i] = pc;
            z = mul(sub(1.0, mul(S.w_hist[i], d)), z);
            pprev = pc;
        }
        S.eta[j] = eta;
        S.zeta[j] = z;
    }
}

// beta not finite: the solve stops after the seed's x of this iteration
template <class G>
__device__ __forceinline__ void seed_x_only(const Ctx &c, const hbk_cur &u, const G &g) {
    hbk_scalars *sc = c.sh.sc;
    if (g.extra()) {
        if (threadIdx.x == 0) {
            sc->status = __ldcg(&sc->status) | HBK_ST_BREAKDOWN;
            sc->finished = 1;
        }
        return;
    }
    const double a = __ldcg(&sc->alpha), w = __ldcg(&sc->omega);
    const unsigned n = c.v.n;
    const double *ps = seed_p(c, u.seed), *q = vec_q(c, u);
    for (size_t i = g.b() * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)g.nb() * blockDim.x) {
        double *xi = c.v.deferred ? c.v.Xp + panel_idx(u.seed, (unsigned)i, c.v.pm)
                                  : c.v.X + (size_t)u.seed * ldn(n) + i;
        *xi = fma(w, HBK_LD(G, q, i), fma(a, HBK_LD(G, ps, i), HBK_LD(G, xi, 0)));
    }
}

// K5 (incremental): the seed's x_s and p_s, then every running shift's x_j and
// p_j in one pass over q, r_{k-1}, r_k (src/solver_dynamic.c:200-210, :248-255);
// r_k rescaled on a switch.  The first element's vectors and, up to MAXS
// shifts, the coefficients are loaded before the iteration's end is decided,
// and each shift's x_j, p_j before the shift ahead of it is stored.
template <int MAXS, class G>
__device__ __forceinline__ void shift_update_body(const Ctx &c, const G &g) {
    __shared__ double s_co[MAXS * 6];
    __shared__ int s_j[MAXS], s_cnt, s_next;
    __shared__ unsigned s_act[MAXS / 32];
    __shared__ double sh[2 * MAXW];
    hbk_scalars *sc = c.sh.sc;
    body_begin<G>();
    body_ready<G>();
    const hbk_cur u = load_cur(sc);
    const double ak = __ldcg(&sc->alpha), wk = __ldcg(&sc->omega);
    StepLoads sl;
    sl.load(c);
    const int m = c.sh.m;
    const unsigned t = threadIdx.x;
    const bool once = m <= MAXS;
    int live = 0;
    double co[6];
    if (once && t < MAXS) {
        const double2 *p = reinterpret_cast<const double2 *>(c.sh.coef + (size_t)t * HBK_NCOEF);
        if ((int)t < m) {
            live = __ldcg(c.sh.live + t);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double2 v = __ldcg(p + k);
                co[2 * k] = v.x, co[2 * k + 1] = v.y;
            }
        }
    }
    if (!u.active || !fin(ak) || !fin(wk) || is_zero(wk)) return;
    const int seed = u.seed, k = u.k;
    const unsigned n = c.v.n;
    const size_t ld = ldn(n), step = (size_t)g.nb() * blockDim.x;
    double *__restrict__ xs = c.v.X + (size_t)seed * ld;
    double *__restrict__ ps = c.v.P + (size_t)seed * ld;
    const double *__restrict__ q = c.v.q;
    const double *__restrict__ s = c.v.s;
    const double *__restrict__ ro = c.v.rbuf[(k - 1) & 1];
    double *__restrict__ rn = c.v.rbuf[k & 1];
    const double *__restrict__ rh = c.v.r_hat;
    size_t i = g.extra() ? (size_t)n : g.b() * (size_t)blockDim.x + t;
    double qi = 0.0, oi = 0.0, ri = 0.0, pi = 0.0, xi = 0.0, si = 0.0;
    if (i < n) {
        qi = HBK_LD(G, q, i), oi = HBK_LD(G, ro, i), ri = HBK_LD(G, rn, i);
        pi = HBK_LD(G, ps, i), xi = HBK_LD(G, xs, i), si = HBK_LD(G, s, i);
    }
    const StepEnd e = step_end(c, u, wk, sl, sh);
    if (!e.ok) {
        seed_x_only(c, u, g);
        return;
    }
    if (g.extra()) {
        record_step(c, u, e);
        return;
    }
    const double bk = e.bk, bw = e.bw;
    double acc = 0.0;
    for (int next = 0, first = 1;; first = 0) {
        // up to MAXS running shifts in index order
        int cnt;
        if (once) {
            bool act = false;
            if (t < MAXS) {
                if ((int)t < m && live == 1 && (int)t != seed) {
                    co[4] = mul(co[4], bk);
                    act = fin(co[4]);
                }
                const unsigned b = __ballot_sync(0xffffffffu, act);
                if ((t & 31) == 0) s_act[t / 32] = b;
            }
            __syncthreads();
            cnt = 0;
            unsigned at = 0;
#pragma unroll
            for (int w = 0; w < MAXS / 32; ++w) {
                if ((unsigned)w == t / 32) at = cnt + __popc(s_act[w] & ((1u << (t & 31)) - 1u));
                cnt += __popc(s_act[w]);
            }
            if (act) {
                s_j[at] = (int)t;
#pragma unroll
                for (int v = 0; v < 6; ++v) s_co[at * 6 + v] = co[v];
            }
            next = m;
        } else {
            if (t < 32) {
                int found = 0, j0 = next;
                for (; j0 < m && found + 32 <= MAXS; j0 += 32) {
                    const int j = j0 + (int)t;
                    const bool act = j < m && j != seed && __ldcg(c.sh.live + j) == 1 &&
                                     fin(mul(__ldcg(c.sh.coef + (size_t)j * HBK_NCOEF + 4), bk));
                    const unsigned b = __ballot_sync(0xffffffffu, act);
                    if (act) s_j[found + __popc(b & ((1u << t) - 1u))] = j;
                    found += __popc(b);
                }
                if (t == 0) s_cnt = found, s_next = j0;
            }
            __syncthreads();
            cnt = s_cnt;
            next = s_next;
            for (int a = (int)t; a < cnt * 6; a += (int)blockDim.x) {
                const double v = __ldcg(c.sh.coef + (size_t)s_j[a / 6] * HBK_NCOEF + a % 6);
                s_co[a] = a % 6 == 4 ? mul(v, bk) : v;
            }
            if (!first) {
                i = g.b() * (size_t)blockDim.x + t;
                if (i < n) qi = HBK_LD(G, q, i), oi = HBK_LD(G, ro, i), ri = HBK_LD(G, rn, i);
            }
        }
        __syncthreads();
        while (i < n) {
            double xn = 0.0, pn = 0.0;
            if (cnt) {
                xn = HBK_LD(G, c.v.X + (size_t)s_j[0] * ld, i);
                pn = HBK_LD(G, c.v.P + (size_t)s_j[0] * ld, i);
            }
            if (first) {
                xs[i] = fma(wk, qi, fma(ak, pi, xi));
                ps[i] = fma(bw, si, fma(bk, pi, ri));
            }
            for (int a = 0; a < cnt; a++) {
                const double *cf = s_co + a * 6;
                double x = xn, p = pn;
                if (a + 1 < cnt) {
                    xn = HBK_LD(G, c.v.X + (size_t)s_j[a + 1] * ld, i);
                    pn = HBK_LD(G, c.v.P + (size_t)s_j[a + 1] * ld, i);
                }
                x = fma(cf[0], qi, x);
                x = fma(cf[1], p, x);
                p = fma(cf[2], qi, p);
                p = fma(cf[3], oi, p);
                p = cf[4] * p;
                p = fma(cf[5], ri, p);
                c.v.X[(size_t)s_j[a] * ld + i] = x;
                c.v.P[(size_t)s_j[a] * ld + i] = p;
            }
            if (e.sw && next >= m) {
                const double rs = ri * e.rsc;
                rn[i] = rs;
                acc = fma(HBK_LD(G, rh, i), rs, acc);
            }
            i += step;
            if (i < n) {
                qi = HBK_LD(G, q, i), oi = HBK_LD(G, ro, i), ri = HBK_LD(G, rn, i);
                if (first) pi = HBK_LD(G, ps, i), xi = HBK_LD(G, xs, i), si = HBK_LD(G, s, i);
            }
        }
        if (next >= m) break;
        __syncthreads();
    }
    if (e.sw) {
        __syncthreads();
        store_part(acc, sh, parts(c, P_RRS) + g.b());
    }
}
template <int MAXS>
__global__ void __launch_bounds__(1024) k_shift_update(Ctx c) { shift_update_body<MAXS>(c, HwGridX{1}); }

// Deferred mode: coefficient update of every running system over the basis
// slots in use, items it0, it0 + step, ... of m x L.  Per coefficient the
// operations follow the vector update's order (x += c0 q; x += c1 p;
// p += c2 q; p += c3 r_{k-1}; p *= beta_j; p += c5 r_k).
template <class G>
__device__ __forceinline__ void coef_update(const Ctx &c, const hbk_cur &u, double bk, unsigned it0, unsigned step) {
    const int sq = u.slots, sr = u.slots + 1, so = u.slot_r_old;
    const unsigned L = (unsigned)u.slots + 2;
    const int cap = c.v.slot_cap;
    const unsigned tot = (unsigned)c.sh.m * L;
    for (unsigned it = it0; it < tot; it += step) {
        const int j = (int)(it / L), i = (int)(it - (unsigned)j * L);
        const double *co = c.sh.coef + (size_t)j * HBK_NCOEF;
        double *xc = c.v.Xc + (size_t)j * cap + i;
        double *pc = c.v.Pc + (size_t)j * cap + i;
        const int live = __ldcg(c.sh.live + j);
        const double c1 = __ldcg(co + 1), c4 = mul(__ldcg(co + 4), bk);
        double x = HBK_LD(G, xc, 0), p = HBK_LD(G, pc, 0);
        if (j != u.seed && (live != 1 || !fin(c4))) continue;
        if (i == sq) x = x + __ldcg(co);
        x = fma(c1, p, x);
        if (i == sq) p = p + __ldcg(co + 2);
        if (i == so) p = p + __ldcg(co + 3);
        p = c4 * p;
        if (i == sr) p = p + __ldcg(co + 5);
        *xc = x;
        *pc = p;
        if (i == 0) {
            double *ow = c.v.own + 2 * (size_t)j;
            const double o1 = HBK_LD(G, ow, 1);
            ow[0] = fma(c1, o1, HBK_LD(G, ow, 0));
            ow[1] = c4 * o1;
            c.sh.lslot[j] = (int)L;
        }
    }
}

// K5 (deferred): x_s and p_s, the coefficient update (in a one-family launch
// by g.ncb() extra blocks, else by every block), on a switch the rescaled
// r_k in a new slot
template <class G>
__device__ __forceinline__ void seed_p_deferred_body(const Ctx &c, const G &g) {
    __shared__ double sh[2 * MAXW];
    __shared__ unsigned long long smx[MAXW];
    hbk_scalars *sc = c.sh.sc;
    body_begin<G>();
    body_ready<G>();
    const hbk_cur u = load_cur(sc);
    const double ak = __ldcg(&sc->alpha), wk = __ldcg(&sc->omega);
    StepLoads sl;
    sl.load(c);
    if (!u.active || !fin(ak) || !fin(wk) || is_zero(wk)) return;
    const unsigned n = c.v.n;
    const size_t ld = ldn(n), step = (size_t)g.nb() * blockDim.x;
    double *__restrict__ ps = c.v.ps;
    const double *__restrict__ s = c.v.s;
    const double *__restrict__ q = vec_q(c, u);
    const double *__restrict__ rn = c.v.V + (size_t)(u.slots + 1) * ld;
    double *__restrict__ rsl = c.v.V + (size_t)(u.slots + 2) * ld;
    double *__restrict__ xp = c.v.Xp;
    const double *__restrict__ rh = c.v.r_hat;
    const int pm = c.v.pm, seed = u.seed;
    size_t i = g.extra() || g.coef_only() ? (size_t)n : g.b() * (size_t)blockDim.x + threadIdx.x;
    double ri = 0.0, pi = 0.0, si = 0.0, qi = 0.0, xi = 0.0;
    if (i < n) {
        ri = HBK_LD(G, rn, i), pi = HBK_LD(G, ps, i), si = HBK_LD(G, s, i), qi = HBK_LD(G, q, i);
        xi = HBK_LD(G, xp, panel_idx(seed, (unsigned)i, pm));
    }
    const StepEnd e = step_end(c, u, wk, sl, sh);
    if (!e.ok) {
        if (!g.coef_only()) seed_x_only(c, u, g);
        return;
    }
    if (g.extra()) {
        record_step(c, u, e);
        return;
    }
    if (g.does_coef()) coef_update<G>(c, u, e.bk, g.cb() * blockDim.x + threadIdx.x, g.ncb() * blockDim.x);
    if (g.coef_only()) return;
    const double bk = e.bk, bw = e.bw;
    double acc = 0.0;
    unsigned long long mx = 0;
    while (i < n) {
        const size_t in = i + step;  // the next element's loads go before this one's stores
        double r2 = 0.0, p2 = 0.0, s2 = 0.0, q2 = 0.0, x2 = 0.0;
        if (in < n) {
            r2 = HBK_LD(G, rn, in), p2 = HBK_LD(G, ps, in), s2 = HBK_LD(G, s, in), q2 = HBK_LD(G, q, in);
            x2 = HBK_LD(G, xp, panel_idx(seed, (unsigned)in, pm));
        }
        xp[panel_idx(seed, (unsigned)i, pm)] = fma(wk, qi, fma(ak, pi, xi));
        ps[i] = fma(bw, si, fma(bk, pi, ri));
        if (e.sw) {
            const double rs = ri * e.rsc;
            rsl[i] = rs;
            acc = fma(HBK_LD(G, rh, i), rs, acc);
            const unsigned long long b = abs_bits(rs);
            mx = b > mx ? b : mx;
        }
        ri = r2, pi = p2, si = s2, qi = q2, xi = x2, i = in;
    }
    if (!e.sw) return;  // uniform: the reduction is needed only after a switch
    if (c.v.slot_max) block_max_to(mx, smx, c.v.slot_max + (size_t)(u.slots + 2) * HBK_SLOT_SPREAD);  // rescaled r_k
    __syncthreads();
    store_part(acc, sh, parts(c, P_RRS) + g.b());
}
__global__ void __launch_bounds__(1024) k_seed_p_deferred(Ctx c, unsigned ncoef) {
    seed_p_deferred_body(c, HwGridX{1 + ncoef});
}

// Deferred mode, after a switch: the new seed's p = own term + Pc[t] . V, and
// its shift on the diagonal of the seed kernels' products
template <class G>
__device__ __forceinline__ void materialize_ps_body(const Ctx &c, const G &g) {
    __shared__ double s_c[1024];
    hbk_scalars *sc = c.sh.sc;
    if (!__ldcg(&sc->need_ps)) return;
    const int t = __ldcg(&sc->seed);
    const int L = HBK_LD(G, c.sh.lslot, t);
    const unsigned n = c.v.n;
    const size_t ld = ldn(n);
    const double *pc = c.v.Pc + (size_t)t * c.v.slot_cap;
    const double rho = HBK_LD(G, c.v.own, 2 * (size_t)t + 1);
    const double *pmat = c.v.Pmat;  // panel-major
    for (size_t i0 = (size_t)g.b() * NT; i0 < n; i0 += (size_t)g.nb() * NT) {
        const size_t i = i0 + threadIdx.x;
        double acc = (pmat && i < n) ? rho * pmat[panel_idx(t, (unsigned)i, c.v.pm)] : 0.0;
        for (int l0 = 0; l0 < L; l0 += 1024) {
            const int cnt = min(1024, L - l0);
            __syncthreads();
            for (int l = threadIdx.x; l < cnt; l += NT) s_c[l] = HBK_LD(G, pc, l0 + l);
            __syncthreads();
            if (i < n)
                for (int l = 0; l < cnt; l++) acc = fma(s_c[l], HBK_LD(G, c.v.V, (size_t)(l0 + l) * ld + i), acc);
        }
        if (i < n) c.v.ps[i] = acc;
    }
    if (c.v.sval_shift) {
        const double sg = c.sh.sigma[t];
        for (size_t r = g.b() * (size_t)NT + threadIdx.x; r < n; r += (size_t)g.nb() * NT) {
            const unsigned long long d = c.v.sdiag[r];
            c.v.sval_shift[d] = c.v.sval_orig[d] + sg;
        }
    }
    if (take_ticket(c.sh.counters + 5, g.nb())) {
        if (threadIdx.x == 0) {
            sc->need_ps = 0;
            c.sh.counters[5] = 0;
            const int status = __ldcg(&sc->status);
            if (status & HBK_ST_NEED_PS) {  // paused for this: run on, unless the basis is full or the solve over
                sc->status = status & ~HBK_ST_NEED_PS;
                if (!(status & (HBK_ST_BASIS_FULL | HBK_ST_BREAKDOWN)) && sc->n_done < sc->m && sc->k < sc->kcap)
                    sc->finished = 0;
            }
        }
    }
}
__global__ void __launch_bounds__(NT) k_materialize_ps(Ctx c) { materialize_ps_body(c, HwGrid()); }

// Flush: X_j += xi_j Pmat_j + Xc_j . V ; when keep_p, Pmat_j = rho_j Pmat_j + Pc_j . V.
// Each thread owns one row and GROUP systems; coefficients are staged in
// shared memory per chunk of slots.  FP64 FMA-bound by design: it is the
// only place the per-shift solutions are formed.
constexpr int GROUP = 16;
constexpr int LCH = 64;
__global__ void __launch_bounds__(NT) k_flush(Ctx c, int keep_p, int which) {
    __shared__ double s_c[GROUP * LCH];
    const unsigned n = c.v.n;
    const size_t ld = ldn(n);
    const int m = c.sh.m, cap = c.v.slot_cap;
    const int j0 = blockIdx.y * GROUP;
    const int g = min(GROUP, m - j0);
    int L = 0;
    for (int t = 0; t < g; t++) L = max(L, c.sh.lslot[j0 + t]);
    const double *coef = which == 0 ? c.v.Xc : c.v.Pc;
    double *out = which == 0 ? c.v.Xp : c.v.Pmat;  // panel-major
    const int pm = c.v.pm;
    for (size_t i0 = (size_t)blockIdx.x * NT; i0 < n; i0 += (size_t)gridDim.x * NT) {
        const size_t i = i0 + threadIdx.x;
        double acc[GROUP];
#pragma unroll
        for (int t = 0; t < GROUP; t++) {
            acc[t] = 0.0;
            if (t < g && i < n) {
                const int j = j0 + t;
                const size_t pi = panel_idx(j, (unsigned)i, pm);
                const double *pmat = c.v.Pmat;
                if (which == 0) {
                    acc[t] = c.v.Xp[pi];
                    if (pmat) acc[t] = fma(c.v.own[2 * (size_t)j], pmat[pi], acc[t]);
                } else if (pmat) {
                    acc[t] = c.v.own[2 * (size_t)j + 1] * pmat[pi];
                }
            }
        }
        for (int l0 = 0; l0 < L; l0 += LCH) {
            const int cnt = min(LCH, L - l0);
            __syncthreads();
            for (int e = threadIdx.x; e < GROUP * LCH; e += NT) {
                const int t = e / LCH, l = e % LCH;
                s_c[e] = (t < g && l < cnt) ? coef[(size_t)(j0 + t) * cap + l0 + l] : 0.0;
            }
            __syncthreads();
            if (i < n) {
                for (int l = 0; l < cnt; l++) {
                    const double v = c.v.V[(size_t)(l0 + l) * ld + i];
#pragma unroll
                    for (int t = 0; t < GROUP; t++) acc[t] = fma(s_c[t * LCH + l], v, acc[t]);
                }
            }
        }
        if (i < n) {
#pragma unroll
            for (int t = 0; t < GROUP; t++)
                if (t < g) out[panel_idx(j0 + t, (unsigned)i, pm)] = acc[t];
        }
    }
    (void)keep_p;
}

// after a flush: reset the coefficients, own = (0, 1), slot 0 = r_{k-1}
__global__ void __launch_bounds__(NT) k_flush_reset(Ctx c, int keep_p, const int *__restrict__ live) {
    hbk_scalars *sc = c.sh.sc;
    const int m = c.sh.m, cap = c.v.slot_cap;
    const unsigned n = c.v.n;
    const size_t ld = ldn(n);
    const int so = sc->slot_r_old;
    const size_t tot = (size_t)m * cap;
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < tot; i += (size_t)gridDim.x * NT) {
        c.v.Xc[i] = 0.0;
        c.v.Pc[i] = 0.0;
    }
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < (size_t)m; i += (size_t)gridDim.x * NT) {
        c.v.own[2 * i] = 0.0;
        c.v.own[2 * i + 1] = keep_p ? 1.0 : 0.0;
        c.sh.lslot[i] = 1;
    }
    if (so != 0)
        for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < n; i += (size_t)gridDim.x * NT)
            c.v.V[i] = c.v.V[(size_t)so * ld + i];
    if (c.v.slot_max) {
        // slot 0 takes the copied slot's maximum (one thread: no other thread
        // touches slots 0 and so); the others start empty
        const size_t tot_e = (size_t)cap * HBK_SLOT_SPREAD;
        for (size_t e = blockIdx.x * (size_t)NT + threadIdx.x; e < tot_e; e += (size_t)gridDim.x * NT) {
            const size_t l = e / HBK_SLOT_SPREAD;
            if (l != 0 && l != (size_t)so) c.v.slot_max[e] = 0;
        }
        if (blockIdx.x == 0 && threadIdx.x < HBK_SLOT_SPREAD && so != 0) {
            const size_t e0 = threadIdx.x, es = (size_t)so * HBK_SLOT_SPREAD + threadIdx.x;
            c.v.slot_max[e0] = c.v.slot_max[es];
            c.v.slot_max[es] = 0;
        }
    }
    if (take_ticket(c.sh.counters + 6)) {
        if (threadIdx.x == 0) {
            if (live) sc->flush_rows += (keep_p ? 4.0 : 3.0) * *live;
            sc->slots = 1;
            sc->slot_r_old = 0;
            sc->status &= ~HBK_ST_BASIS_FULL;
            if (sc->n_done < sc->m && sc->k < sc->kcap && !(sc->status & HBK_ST_BREAKDOWN)) sc->finished = 0;
            c.sh.counters[6] = 0;
        }
    }
}

// first vectors of a solve, all equal to b: incremental mode r_0 and every
// p_j; deferred mode basis slot 0 (with its maximum) and the seed's p.  The
// shadow residual is the caller's copy of b itself when the two are one array.
__global__ void __launch_bounds__(NT) k_init_vectors(Ctx c, const double *b) {
    __shared__ unsigned long long smx[NW];
    const unsigned n = c.v.n;
    const size_t ld = ldn(n);
    unsigned long long mx = 0;
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < n; i += (size_t)gridDim.x * NT) {
        const double bi = b[i];
        if (c.v.r_hat != b) c.v.r_hat[i] = bi;
        if (c.v.deferred) {
            c.v.V[i] = bi;
            c.v.ps[i] = bi;
            const unsigned long long a = abs_bits(bi);
            mx = a > mx ? a : mx;
        } else {
            c.v.rbuf[0][i] = bi;
            for (int j = 0; j < c.sh.m; ++j) c.v.P[(size_t)j * ld + i] = bi;
        }
    }
    if (c.v.deferred && c.v.slot_max) block_max_to(mx, smx, c.v.slot_max);
}

// hbk_pack's block (hbk.h)
__global__ void __launch_bounds__(NT) k_pack(hbk_shifts S, int nk, const double *__restrict__ res,
                                             const int *__restrict__ err, double *__restrict__ out) {
    const int m = S.m;
    int *w = reinterpret_cast<int *>(out + 1 + m + 4 * (size_t)nk);
    for (int i = blockIdx.x * NT + threadIdx.x; i < nk || i < m; i += gridDim.x * NT) {
        if (i < m) {
            out[1 + i] = res[i];
            w[i] = S.conv_k[i];
            w[m + i] = S.sw_k[i];
            w[2 * m + i] = S.sw_seed[i];
        }
        if (i < nk) {
            double *h = out + 1 + m;
            h[i] = S.a_hist[i];
            h[(size_t)nk + i] = S.b_hist[i];
            h[2 * (size_t)nk + i] = S.w_hist[i];
            h[3 * (size_t)nk + i] = S.rr_hist[i];
            w[3 * m + 1 + i] = S.act_hist[i];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        out[0] = S.sc->flush_rows;
        w[3 * m] = err ? *err : 0;
    }
}

// End of a while-loop body in a CUDA graph: run again while the solve goes on
// (not finished: converged, at max_iter, broken down or waiting for a basis
// flush), and never more than loop_cap bodies per solve.
__global__ void k_loop_condition(hbk_scalars *sc, cudaGraphConditionalHandle cond, int loop_cap) {
    const int loops = ++sc->loops;
    cudaGraphSetConditional(cond, (!sc->finished && loops < loop_cap) ? 1u : 0u);
}

// x[i] = element i of system j of the panel-major Xp (runs of HBK_PANEL)
__global__ void __launch_bounds__(NT) k_panel_row(const double *__restrict__ Xp, int m, unsigned n, int j,
                                                  double *__restrict__ x) {
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < n; i += (size_t)gridDim.x * NT)
        x[i] = Xp[panel_idx(j, (unsigned)i, m)];
}

// X[j][i] = element i of system j of the panel-major Xp: one block per panel
// (m * HBK_PANEL values read contiguously, written as runs of HBK_PANEL);
// nothing where *err says that a flush failed
__global__ void __launch_bounds__(NT) k_panel_to_rows(const double *__restrict__ Xp, int m, unsigned n,
                                                      double *__restrict__ X, size_t ld,
                                                      const int *__restrict__ err) {
    if (err && *err) return;
    const unsigned per = (unsigned)m * HBK_PANEL;
    const size_t np = ((size_t)n + HBK_PANEL - 1) / HBK_PANEL;
    for (size_t p = blockIdx.x; p < np; p += gridDim.x) {
        const double *src = Xp + p * per;
        const size_t i0 = p * HBK_PANEL;
        for (unsigned r = threadIdx.x; r < per; r += NT) {
            const unsigned j = r / HBK_PANEL, c = r - j * HBK_PANEL;
            if (i0 + c < n) X[(size_t)j * ld + i0 + c] = src[r];
        }
    }
}

// ---------------------------------------------------------------------------
// Many families in one persistent launch (SELL-32, either shift mode).
//
// Each family's rows are cut into virtual blocks of HBK_GROUP_ROWS rows; the
// CTAs of one cooperative launch take the virtual blocks of all families in
// turn (virtual block v goes to CTA v mod grid, so a family's rows stay on
// the same CTAs from step to step) and run, for every family at once, the
// same steps as the one-family kernels (K1..K5, and the forming of a new
// seed's p in the deferred mode, with a virtual block in place of the launch's
// block: same partial sums and, per family, one more entry for the extra block
// of K4 and K5).  A grid-wide barrier separates the steps.  Families stop one by one
// (converged, max_iter, breakdown) or pause with a full basis; their virtual
// blocks then return at once, and the launch ends when every family has
// stopped or paused (the host flushes the paused ones and launches again).
struct GroupFam {
    Ctx c;
    unsigned vb0, nvb;  // entry vb0: the extra block of K4 and K5; then its nvb virtual blocks
};

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned atom_add_acq_rel_u32(unsigned *p, unsigned v) {
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Barrier over every CTA of a cooperative launch: bar[0] counts arrivals,
// bar[1] is the generation (the last CTA to arrive resets the count and bumps
// it, with release order; the others wait for it with acquire loads).  A wait
// longer than HBK_GROUP_WAIT_NS sets *err; every CTA that sees *err leaves the
// wait, so the launch ends (with the error) instead of hanging.  Returns
// false in every thread of the CTA when the launch must stop.  withhold:
// this CTA waits without arriving (the bounded-wait test: every CTA then
// waits out the bound, and the launch ends with HBK_GROUP_ERR_WAIT).
__device__ bool grid_barrier(unsigned *bar, int *err, bool withhold = false) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned gen = ld_acquire_u32(bar + 1);
        const unsigned arrived = withhold ? 0u : atom_add_acq_rel_u32(bar, 1u) + 1u;
        if (arrived == gridDim.x) {
            atomicExch(bar, 0u);
            st_release_u32(bar + 1, gen + 1u);
        } else {
            const unsigned long long t0 = global_ns();
            while (ld_acquire_u32(bar + 1) == gen) {
                if (*(volatile int *)err) {
                    ok = 0;
                    break;
                }
                if (global_ns() - t0 > HBK_GROUP_WAIT_NS) {
                    atomicExch(err, HBK_GROUP_ERR_WAIT);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
            __threadfence();
        }
        s_ok = ok && *(volatile int *)err == 0;
    }
    __syncthreads();
    return s_ok != 0;
}

// step 5: the shift update (incremental) or the seed's p update (deferred)
template <int MAXS>
__device__ __forceinline__ void step5_body(const Ctx &c, const VGrid &g) {
    if (c.v.deferred) seed_p_deferred_body(c, g);
    else shift_update_body<MAXS>(c, g);
}
__device__ __forceinline__ void materialize_if_deferred(const Ctx &c, const VGrid &g) {
    if (c.v.deferred) materialize_ps_body(c, g);
}

// (3 CTAs per SM: the register cap costs a few spills in the scalar stage)
template <int MAXS>
__global__ void __launch_bounds__(NT, 3) k_group(const GroupFam *__restrict__ fams, int nf,
                                                 const unsigned *__restrict__ vb_fam, unsigned nvb, unsigned *bar,
                                                 int *err, int iter_cap, int any_deferred, int withhold) {
#define HBK_GROUP_STEP(body, with_extra)                                           \
    for (unsigned vb = blockIdx.x; vb < nvb; vb += gridDim.x) {                    \
        const GroupFam &F = fams[vb_fam[vb]];                                      \
        const bool extra = vb == F.vb0; /* a family's first entry */               \
        if (extra && !(with_extra)) continue;                                      \
        body(F.c, VGrid{vb - F.vb0 - 1u, F.nvb, extra});                           \
    }                                                                              \
    if (!grid_barrier(bar, err)) return;
    for (int it = 0; it <= iter_cap; ++it) {
        // any family still running?  (read between two barriers: no step
        // writes a family's stop flag meanwhile, so every CTA sees the same)
        int alive = 0;
        for (int f = threadIdx.x; f < nf; f += NT) alive |= __ldcg(&fams[f].c.sh.sc->finished) == 0;
        alive = __syncthreads_or(alive);
        if (!grid_barrier(bar, err, withhold && it == 0 && blockIdx.x == 0) || !alive) return;
        HBK_GROUP_STEP(seed_s_body<HBK_FMT_SELL>, false)
        HBK_GROUP_STEP(seed_q_body, false)
        HBK_GROUP_STEP(seed_y_body<HBK_FMT_SELL>, false)
        HBK_GROUP_STEP(seed_update_body, true)
        HBK_GROUP_STEP(step5_body<MAXS>, true)
        if (any_deferred) {
            HBK_GROUP_STEP(materialize_if_deferred, false)
        }
    }
#undef HBK_GROUP_STEP
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(err, HBK_GROUP_ERR_CAP);
}

}  // namespace

extern "C" {

int hbk_panel_row(const double *Xp, int m, unsigned n, int j, double *x, cudaStream_t st) {
    if (n == 0 || j < 0 || j >= m) return 0;
    k_panel_row<<<grid_for(n, 4), NT, 0, st>>>(Xp, m, n, j, x);
    return (int)cudaGetLastError();
}

int hbk_panel_to_rows(const double *Xp, int m, unsigned n, double *X, size_t ld, const int *err, cudaStream_t st) {
    if (m <= 0 || n == 0) return 0;
    const size_t np = ((size_t)n + HBK_PANEL - 1) / HBK_PANEL;
    k_panel_to_rows<<<(unsigned)(np < 4864 ? np : 4864), NT, 0, st>>>(Xp, m, n, X, ld, err);
    return (int)cudaGetLastError();
}

static Ctx make_ctx(const hbk_matrix *A, const hbk_vectors *v, const hbk_shifts *sh) {
    Ctx c;
    c.np_s = c.np_y = c.np_r = c.np_p = 0;
    c.A = *A;
    c.v = *v;
    c.sh = *sh;
    // the seed shift sits on the diagonal of a private copy of the SELL-32
    // values: only while the matrix is in that form and the copy was made from it
    if (c.v.sval_shift && c.A.fmt == HBK_FMT_SELL && c.v.deferred && c.A.sval == c.v.sval_orig)
        c.A.sval = c.v.sval_shift;
    else
        c.v.sval_shift = nullptr;
    return c;
}

int hbk_fused_init(const hbk_matrix *A, const hbk_vectors *v, const hbk_shifts *sh, const double *b, int seed,
                   double tol, int switching, int inline_ps, cudaStream_t st) {
    Ctx c = make_ctx(A, v, sh);
    const unsigned n = v->n;
    const size_t ld = ((size_t)n + 31) / 32 * 32;
    int e;
    if ((e = hbk_dot(n, b, b, sh->partials, sh->counters + 7, &sh->sc->bb, st))) return e;
    if (v->deferred) {
        if (v->sval_shift && A->fmt == HBK_FMT_SELL && A->sval == v->sval_orig &&
            (e = hbk_fold_diag(n, A->sval, A->sell_len, v->sdiag, sh->sigma + seed, v->sval_shift, st)))
            return e;
        if (v->slot_max && (e = (int)cudaMemsetAsync(v->slot_max, 0,
                                                     sizeof(unsigned long long) * (size_t)v->slot_cap * HBK_SLOT_SPREAD,
                                                     st)))
            return e;
        k_init_coef<<<grid_for((unsigned)((size_t)sh->m * v->slot_cap), 1), NT, 0, st>>>(c);
    }
    k_init_vectors<<<grid_for(n ? n : 1, 2), NT, 0, st>>>(c, b);
    if ((e = (int)cudaGetLastError())) return e;
    if (v->deferred) {
        if ((e = (int)cudaMemsetAsync(v->Xp, 0, sizeof(double) * hbk_panel_elems(n, v->pm), st))) return e;
    } else if ((e = (int)cudaMemsetAsync(v->X, 0, sizeof(double) * ld * (size_t)sh->m, st))) {
        return e;
    }
    k_init<<<1, NT, 0, st>>>(c, seed, tol, switching, inline_ps);
    return (int)cudaGetLastError();
}

int hbk_hyb_wave_fused(int wide) {
    const int a = wide ? wave_grid<k_seed_s<HBK_FMT_HYBW>>(HBK_MAX_GRID) : wave_grid<k_seed_s<HBK_FMT_HYB>>(HBK_MAX_GRID);
    const int b = wide ? wave_grid<k_seed_y<HBK_FMT_HYBW>>(HBK_MAX_GRID) : wave_grid<k_seed_y<HBK_FMT_HYB>>(HBK_MAX_GRID);
    return a < b ? a : b;
}

}  // extern "C"

// Blocks of a vector kernel beside `extra` others: one per SM at most, of
// n / SMs rows rounded up to two warps (128..1024 threads; longer vectors in a
// grid-stride loop).  Above 512 threads an SM holds one block, so the extra
// ones take SMs of their own.
struct VecGrid {
    int blocks, threads;
};
static VecGrid vec_grid(unsigned n, int extra, unsigned least = 128) {
    const int sms = sm_count();
    const unsigned per = (n / (unsigned)sms + 64) / 64 * 64;
    const unsigned t = per < least ? least : (per > 1024 ? 1024 : per);
    const int most = t <= 512 ? sms : (sms > 2 * extra ? sms - extra : 1);
    const unsigned need = n ? (n + t - 1) / t : 1;
    return {need < (unsigned)most ? (int)need : most, (int)t};
}
// K4's: all its sets of rows resident at once beside the extra block, in one block
// per SM and 64 registers where that leaves the extra one an SM; else (the most
// sets, DOT_VEC per SM) two blocks per SM and 40 registers, so that a third fits
// (their spills are the scalars' in the extra block, which need not be fast then;
// n = 512 would take 8.5 instead of 6.3 us).
static int vec_sets(unsigned n) {
    const int most = DOT_VEC * sm_count();
    const unsigned want = n ? (n + DOT_ROWS - 1) / DOT_ROWS : 1;
    return want < (unsigned)most ? (int)want : most;
}
struct SetGrid {
    int blocks, threads;
    bool one;    // one block per SM
    bool early;  // may start early
};
// Early only where blocks cannot crowd onto the SMs that the kernel before
// leaves first: blocks that fill an SM's registers, or few small ones.  Measured, an
// iteration, early / not: 256^3, 2 shifts 1010 / 950 us, 128^3 172 / 163, 80 k power-law
// rows 47.9 / 46.4, 42^3 34.1 / 31.9; blocks of 1024: 64^3 61.6 / 63.0; 36^3 26.5 both.
static SetGrid set_grid(int sets) {
    const int sms = sm_count();
    if (sets <= sms) return {sets, NT, true, sets <= sms * 4 / 5};
    for (int per = 2; per <= DOT_VEC; ++per)
        if (sets <= per * (sms - 1)) return {(sets + per - 1) / per, per * NT, true, per == DOT_VEC};
    return {(sets + 1) / 2, 2 * NT, false, false};
}

// kernel<<<...>>>, allowed to start before the stream's previous kernel ends
// (the kernel waits for it before it reads anything the iteration writes)
template <class... P, class... Arg>
static void launch(void (*kernel)(P...), int blocks, int threads, bool early, cudaStream_t st, Arg... arg) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, P(arg)...);
}

template <int FMT>
static void launch_iteration(Ctx &c, const hbk_matrix *A, int early, cudaStream_t st) {
    // the products are grid-stride loops: at most one wave of them, and of the
    // forms whose blocks are the sets, a number that registers do not move
    const int most = FMT == HBK_FMT_MERGE ? 4 * sm_count() : FMT == HBK_FMT_TILE ? 6 * sm_count() : HBK_MAX_GRID;
    const int want = A->grid < most ? A->grid : most;
    const int gs = wave_grid<k_seed_s<FMT>>(want), gy = wave_grid<k_seed_y<FMT>>(want);
    constexpr bool sell = FMT == HBK_FMT_SELL || FMT == HBK_FMT_SELLN;
    // (K2 adds K1's sums with NT threads, or fewer where there are no more sums
    // than these, as a few rows leave of SELL-32 only)
    const VecGrid q = vec_grid(c.v.n, 0, sell ? 128 : NT);
    const SetGrid r = set_grid(vec_sets(c.v.n));
    const unsigned ncoef = !c.v.deferred ? 0 : ((unsigned)(c.sh.m < 256 ? c.sh.m : 256) * 64u + q.threads - 1) / q.threads;
    const VecGrid p = vec_grid(c.v.n, 1 + (int)ncoef);
    // (SELL-32: a set for every NT rows up to two per block)
    const auto sets = [&](int blocks) { return (unsigned)(sell && A->grid < 2 * blocks ? A->grid : sell ? 2 * blocks : blocks); };
    c.np_s = sets(gs), c.np_y = sets(gy);
    c.np_r = (unsigned)vec_sets(c.v.n), c.np_p = (unsigned)p.blocks;
    // Early starts: measured on whole solves, SELL-32, n = 512: 1163 -> 1061 us;
    // 97 k rows: 20.1 -> 18.5 ms; 128^3: 64.2 -> 63.0 ms.  Not where blocks
    // that start early would crowd onto the SMs the kernel before leaves free
    // and then run long: the incremental update (FP64-bound; 32^3: 3.4 -> 4.7
    // ms), the products of the other forms (HYB, an iteration with 16 shifts, 20 k
    // rows 34.6 -> 34.0 us, but 60 k 49.1 -> 56.8, 1 M 294 -> 303), K4 by set_grid.
    const bool e = early > 0, es = e && sell;
    launch(k_seed_s<FMT>, gs, NT, es && early > 1, st, c);
    launch(k_seed_q, q.blocks, q.threads, e, st, c);
    launch(k_seed_y<FMT>, gy, NT, es, st, c);
    launch(r.one ? k_seed_update<1> : k_seed_update<3>, r.blocks + 1, r.threads, e && r.early, st, c);
    if (!c.v.deferred) launch(k_shift_update<64>, p.blocks + 1, p.threads, false, st, c);
    else launch(k_seed_p_deferred, p.blocks + 1 + (int)ncoef, p.threads, e, st, c, ncoef);
}

extern "C" {

int hbk_fused_iteration(const hbk_matrix *A, const hbk_vectors *v, const hbk_shifts *sh, int early, cudaStream_t st) {
    Ctx c = make_ctx(A, v, sh);
    if (sell_narrow(*A)) launch_iteration<HBK_FMT_SELLN>(c, A, early, st);
    else if (A->fmt == HBK_FMT_SELL) launch_iteration<HBK_FMT_SELL>(c, A, early, st);
    else if (A->fmt == HBK_FMT_MERGE) launch_iteration<HBK_FMT_MERGE>(c, A, early, st);
    else if (A->fmt == HBK_FMT_HYB && A->nwide) launch_iteration<HBK_FMT_HYBW>(c, A, early, st);
    else if (A->fmt == HBK_FMT_HYB) launch_iteration<HBK_FMT_HYB>(c, A, early, st);
    else launch_iteration<HBK_FMT_TILE>(c, A, early, st);
    return (int)cudaGetLastError();
}

size_t hbk_pack_bytes(int m, int nk) {
    return sizeof(double) * (1 + (size_t)(m > 0 ? m : 0) + 4 * (size_t)nk) +
           sizeof(int) * (3 * (size_t)(m > 0 ? m : 0) + 2 + (size_t)nk);
}

int hbk_pack(const hbk_shifts *sh, int nk, const double *res, const int *err, void *out, cudaStream_t st) {
    const int most = nk > sh->m ? nk : sh->m;
    const int blocks = most / NT + 1;
    k_pack<<<blocks < 32 ? blocks : 32, NT, 0, st>>>(*sh, nk, res, err, (double *)out);
    return (int)cudaGetLastError();
}

int hbk_materialize_ps(const hbk_matrix *A, const hbk_vectors *v, const hbk_shifts *sh, cudaStream_t st) {
    Ctx c = make_ctx(A, v, sh);
    k_materialize_ps<<<wave_grid<k_materialize_ps>(grid_for(v->n, 2)), NT, 0, st>>>(c);
    return (int)cudaGetLastError();
}

// the next shared launch's CTA 0 withholds its first barrier arrival (one
// shot; for the test of the bounded wait)
static int g_group_withhold = 0;
void hbk_group_test_withhold(int on) { g_group_withhold = on ? 1 : 0; }

static unsigned group_vblocks(unsigned n, unsigned rows) {
    if (rows == 0) rows = HBK_GROUP_ROWS;
    const unsigned v = (n + rows - 1) / rows;
    return v < 1 ? 1 : (v > HBK_MAX_GRID ? HBK_MAX_GRID : v);
}

static const size_t kGroupHead = 256;  // barrier words and the error flag

static size_t group_bytes(int nf, size_t nvb) {
    return kGroupHead + ((sizeof(GroupFam) * (size_t)nf + 255) / 256) * 256 + sizeof(unsigned) * nvb;
}

size_t hbk_group_ws_bytes(int nf, const hbk_vectors *v, unsigned rows_per_vb) {
    size_t nvb = 0;
    for (int f = 0; f < nf; ++f) nvb += 1 + group_vblocks(v[f].n, rows_per_vb);
    return group_bytes(nf, nvb);
}

int hbk_group_ctas(int max_ctas) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_group<64>, NT, 0) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    const int one_wave = per_sm * sm_count();
    return max_ctas > 0 && max_ctas < one_wave ? max_ctas : one_wave;
}

int hbk_group_run(int nf, const hbk_matrix *A, const hbk_vectors *v, const hbk_shifts *sh, int iter_cap, int max_ctas,
                  unsigned rows_per_vb, void *ws, size_t ws_bytes, int *err_out, cudaStream_t st) {
    *err_out = 0;
    if (nf <= 0) return 0;
    int dev = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return (int)cudaErrorNotSupported;
    std::vector<GroupFam> tab((size_t)nf);
    std::vector<unsigned> map;
    int any_deferred = 0;
    for (int f = 0; f < nf; ++f) {
        if (A[f].fmt != HBK_FMT_SELL) return (int)cudaErrorInvalidValue;
        any_deferred |= v[f].deferred != 0;
        tab[f].c = make_ctx(&A[f], &v[f], &sh[f]);
        tab[f].vb0 = (unsigned)map.size();
        tab[f].nvb = group_vblocks(v[f].n, rows_per_vb);
        tab[f].c.np_s = tab[f].c.np_y = tab[f].c.np_r = tab[f].c.np_p = tab[f].nvb;
        map.insert(map.end(), 1 + tab[f].nvb, (unsigned)f);
    }
    const unsigned nvb = (unsigned)map.size();
    if (ws_bytes < group_bytes(nf, nvb)) return (int)cudaErrorInvalidValue;
    char *base = (char *)ws;
    unsigned *bar = (unsigned *)base;
    int *err = (int *)(base + 64);
    GroupFam *dtab = (GroupFam *)(base + kGroupHead);
    unsigned *dmap = (unsigned *)(base + kGroupHead + ((sizeof(GroupFam) * (size_t)nf + 255) / 256) * 256);
    int e;
    if ((e = (int)cudaMemsetAsync(base, 0, kGroupHead, st))) return e;
    if ((e = (int)cudaMemcpyAsync(dtab, tab.data(), sizeof(GroupFam) * (size_t)nf, cudaMemcpyHostToDevice, st)))
        return e;
    if ((e = (int)cudaMemcpyAsync(dmap, map.data(), sizeof(unsigned) * (size_t)nvb, cudaMemcpyHostToDevice, st)))
        return e;
    int ctas = hbk_group_ctas(max_ctas);
    if ((unsigned)ctas > nvb) ctas = (int)nvb; /* a CTA without a virtual block would only wait at barriers */
    int withhold = g_group_withhold;
    g_group_withhold = 0;
    const GroupFam *a0 = dtab;
    const unsigned *a2 = dmap;
    void *args[] = {(void *)&a0,  (void *)&nf,  (void *)&a2,       (void *)&nvb,
                    (void *)&bar, (void *)&err, (void *)&iter_cap, (void *)&any_deferred, (void *)&withhold};
    if ((e = (int)cudaLaunchCooperativeKernel((const void *)k_group<64>, dim3(ctas), dim3(NT), args, 0, st))) return e;
    /* pageable destination: returns once the launch has finished */
    return (int)cudaMemcpyAsync(err_out, err, sizeof(int), cudaMemcpyDeviceToHost, st);
}

int hbk_loop_condition(const hbk_shifts *sh, cudaGraphConditionalHandle cond, int loop_cap, cudaStream_t st) {
    k_loop_condition<<<1, 1, 0, st>>>(sh->sc, cond, loop_cap);
    return (int)cudaGetLastError();
}

int hbk_deferred_flush(const hbk_vectors *v, const hbk_shifts *sh, int keep_p, cudaStream_t st) {
    hbk_matrix A0 = {};
    Ctx c = make_ctx(&A0, v, sh);
    const int groups = (sh->m + GROUP - 1) / GROUP;
    dim3 grid(grid_for(v->n, 1), groups);
    // x first: it reads the old Pmat, which the p pass then overwrites
    k_flush<<<grid, NT, 0, st>>>(c, keep_p, 0);
    if (keep_p) k_flush<<<grid, NT, 0, st>>>(c, keep_p, 1);
    k_flush_reset<<<grid_for(v->n, 2), NT, 0, st>>>(c, keep_p, nullptr);
    return (int)cudaGetLastError();
}

int hbk_deferred_reset(const hbk_vectors *v, const hbk_shifts *sh, int keep_p, const int *live, cudaStream_t st) {
    hbk_matrix A0 = {};
    Ctx c = make_ctx(&A0, v, sh);
    k_flush_reset<<<grid_for(v->n, 2), NT, 0, st>>>(c, keep_p, live);
    return (int)cudaGetLastError();
}

}  // extern "C"
