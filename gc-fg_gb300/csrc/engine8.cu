// engine8.cu -- graphs with the 8-neighbourhood (the reference built with
// NEIGHBORHOOD == 8: GraphCut.h:22, the #if NEIGHBORHOOD == 8 blocks of
// GraphCut.cu and GraphCutKernels.cu).
//
// A separate engine from the tiled 4-neighbour solver, so that the latter
// keeps its layout and tuning.  Pixels are row-major; the residual
// capacities are eight planes, cap[d * n + i] from pixel i toward direction
// d (0 left, 1 right, 2 up, 3 down, 4 up-left, 5 up-right, 6 down-left,
// 7 down-right).  One cooperative launch runs the whole solve:
//   * global relabel, exact but for the first (up to nine steps): the distances to the sink-connected pixels
//     (excess < 0) over the residual edges, by rounds over 32x32 tiles with a
//     bit-parallel BFS of each tile (gr8_tile);
//   * count: pixels with excess that can still reach the sink; none left
//     after an exact global relabel means the preflow is maximum (an exact
//     termination test);
//   * tile rounds: every 32x8 tile that is due once per round, each visit a few
//     block-local push/relabel sweeps in shared memory (tile8_visit), the
//     results added back as deltas;
//   * cuts: S_max = pixels at height INF after the last exact global
//     relabel, S_min = the forward closure of the pixels with excess, by
//     rounds over 32x32 tiles like the global relabel (reach8_tile).
// Every spin is bounded; a timeout or an iteration cap sets an error that
// the host reports as GCFG_ERR_NOT_CONVERGED.
#include <cstring>

#include "engine.cuh"

namespace gcfg {
namespace {

constexpr int ND = 8;
__device__ __forceinline__ int dxd(int d) { return d == 0 || d == 4 || d == 6 ? -1 : (d == 1 || d == 5 || d == 7 ? 1 : 0); }
__device__ __forceinline__ int dyd(int d) { return d == 2 || d == 4 || d == 5 ? -1 : (d == 3 || d == 6 || d == 7 ? 1 : 0); }
__device__ __forceinline__ int opp(int d) { return d < 4 ? (d ^ 1) : 11 - d; }

struct Ctl8 {
    unsigned bar_count, bar_gen;
    int err, err_code;
    int round_active[3];  // tiles that had work (or changed a height) in round p, at [p % 3]
    unsigned long long active, pos_excess, interior_dp, ref_init;
    unsigned long long tile_visits;  // push visits of tiles that had work
    int global_relabels, tile_rounds, gr_rounds, reach_rounds;
};

struct G8 {
    int W, H;
    long long n;
    int *cap;  // 8 * n
    int *e, *h, *mark;
    unsigned *tm;  // NPLANE x 32 row masks per 32x32 tile, made by each global relabel
    int *due;      // per 32x8 tile: the last tile round that has to visit it
    Ctl8 *ctl;
};

struct P8 {
    int max_outer;   // global relabels at most
    int rounds;      // tile rounds between global relabels
    int sweeps;      // push/relabel sweeps per tile visit
    int near_h;      // > 0: the first iteration relabels and pushes only this close to the sinks (engine.cuh, near_h)
};

enum { E8_BARRIER = 1, E8_OUTER = 2 };

__device__ __forceinline__ void set_err8(Ctl8 *c, int code) {
    atomicExch(&c->err, 1);
    atomicCAS(&c->err_code, 0, code);
}

// Grid barrier (bounded spin).
__device__ __forceinline__ unsigned atom_add_acq_rel8(unsigned *p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

__device__ __forceinline__ unsigned ld_acquire8(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ bool sync8(Ctl8 *c) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned gen = ld_acquire8(&c->bar_gen);
        if (atom_add_acq_rel8(&c->bar_count, 1u) == gridDim.x - 1) {
            c->bar_count = 0;
            atom_add_acq_rel8(&c->bar_gen, 1u);
        } else {
            unsigned long long it = 0;
            while (ld_acquire8(&c->bar_gen) == gen) {
                if (++it > (1ull << 25)) {
                    set_err8(c, E8_BARRIER);
                    break;
                }
                __nanosleep(32);
            }
        }
    }
    // thread 0's reading of the error word decides for the whole block
    return !__syncthreads_or(threadIdx.x == 0 && *(volatile int *)&c->err != 0);
}

// Graph of the reference's InitGraph / InitGraphVarEdges with NEIGHBORHOOD
// == 8 (GraphCutKernels.cu:112-214): interior pixels only, excess dp - dn,
// caps from the arrays (or the penalty), edges toward the 1-pixel border
// zeroed, diagonals included.
struct Arr8 {
    const int *a[8];  // left, right, up, down, up-left, up-right, down-left, down-right (NULL: penalty)
};

__global__ void k8_build(G8 g, const int *__restrict__ dp, const int *__restrict__ dn, int penalty, Arr8 arr) {
    const long long w32 = (long long)((g.W + 31) / 32) * 32;
    unsigned long long idp = 0, rinit = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < g.n; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % g.W), y = (int)(i / g.W);
        const bool inside = x > 0 && y > 0 && x < g.W - 1 && y < g.H - 1;
        const int vdp = dp[i];
        if ((long long)x + (long long)y * w32 < g.n && vdp > 0) rinit += (unsigned)vdp;
        int e = 0;
        if (inside) {
            e = vdp - dn[i];
            idp += (unsigned)vdp;
            if (vdp < 0 || dn[i] < 0 || vdp > GCFG_MAX_CAP8 || dn[i] > GCFG_MAX_CAP8) set_err8(g.ctl, 9);
        }
        for (int d = 0; d < ND; ++d) {
            int c = 0;
            if (inside) {
                c = arr.a[0] ? arr.a[d][i] : penalty;
                if (c < 0 || c > GCFG_MAX_CAP8) set_err8(g.ctl, 9);
                const int xx = x + dxd(d), yy = y + dyd(d);
                if (xx < 1 || yy < 1 || xx > g.W - 2 || yy > g.H - 2) c = 0;  // toward the border ring
            }
            g.cap[(long long)d * g.n + i] = c;
        }
        g.e[i] = e;
    }
    // one atomic per warp and counter: per-thread atomics on these two
    // addresses serialise in L2 (about 0.4 ms for a 640x480 graph)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        idp += __shfl_down_sync(0xffffffffu, idp, o);
        rinit += __shfl_down_sync(0xffffffffu, rinit, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (idp) atomicAdd(&g.ctl->interior_dp, idp);
        if (rinit) atomicAdd(&g.ctl->ref_init, rinit);
    }
}

// One push visit of a 32x8 tile (one pixel per thread): the tile's
// capacities, excess and heights and a one-pixel ring of heights (corners
// included) are staged in shared memory, up to `sweeps` push/relabel sweeps
// run with block barriers only, and the results go back as additive deltas.
// A visit that ends with a pixel still active makes its tile due in the next
// round, and flow that leaves the tile makes the receiving one due; a round
// visits the tiles that are due.
// Every tile of the image is visited concurrently in a round, so a tile's
// ring heights are a snapshot and its neighbours change its pixels meanwhile;
// that stays safe because every concurrent update is an addition: a pixel's
// own capacity toward a neighbour falls only by its own pushes (never more
// than the value it read, which others can only have raised), excess falls
// only by its owner's pushes, and flow into another tile is added with
// global atomics to the receiver's excess and reverse capacity.  Heights are
// written only by their owner.  Stale ring heights can only make labels
// inexact, never a flow invalid; the exact global relabel and its count
// decide termination.
constexpr int T8W = 32, T8H = 8;
#ifndef GCFG_N8_ROUNDS
#define GCFG_N8_ROUNDS 8    // tile rounds between global relabels
#endif
#ifndef GCFG_N8_SWEEPS
#define GCFG_N8_SWEEPS 8    // sweeps per tile visit
#endif
// More rounds than this between relabels are taken as this many: the setting
// accepts any count, a long solve takes three times as many, and pixels whose
// excess cannot reach a sink keep their tiles due, a few levels higher per
// round, until a relabel finds them cut off.
constexpr int MAX_ROUNDS8 = 1 << 12;

__device__ void tile8_visit(const G8 &g, int t, int tiles_x, int sweeps, int hlim, int round) {
    // excess and capacities have a ring too: flow that leaves the tile collects
    // there (a ring cell's excess, and its capacity back into the tile)
    __shared__ int sh[T8H + 2][T8W + 2];
    __shared__ int se[T8H + 2][T8W + 2];
    __shared__ int sc[ND][T8H + 2][T8W + 2];
    __shared__ int live[3];
    const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
    const int x = (t % tiles_x) * T8W + lx, y = (t / tiles_x) * T8H + ly;
    const bool inb = x < g.W && y < g.H;
    const long long i = (long long)y * g.W + x;
    const int e0 = inb ? __ldcg(g.e + i) : 0;
    int hh = inb ? __ldcg(g.h + i) : INF_H;
    int c0[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) c0[d] = inb ? __ldcg(g.cap + (long long)d * g.n + i) : 0;
    // this thread's ring cell, if it has one: the rows above and below (with
    // the corners), then the sides
    constexpr int RING = 2 * (T8W + 2) + 2 * T8H;
    int rx = -1, ry = 0;
    if (threadIdx.x < 2 * (T8W + 2)) {
        rx = threadIdx.x % (T8W + 2);
        ry = threadIdx.x < T8W + 2 ? 0 : T8H + 1;
    } else if (threadIdx.x < RING) {
        rx = (threadIdx.x - 2 * (T8W + 2)) & 1 ? T8W + 1 : 0;
        ry = 1 + ((threadIdx.x - 2 * (T8W + 2)) >> 1);
    }
    static_assert(RING <= 256, "a ring cell per thread");
    if (rx >= 0) {
        const int xx = x - lx + rx - 1, yy = y - ly + ry - 1;
        const bool in = xx >= 0 && yy >= 0 && xx < g.W && yy < g.H;
        sh[ry][rx] = in ? __ldcg(g.h + (long long)yy * g.W + xx) : INF_H;
        se[ry][rx] = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) sc[d][ry][rx] = 0;
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) sc[d][ly + 1][lx + 1] = c0[d];
    se[ly + 1][lx + 1] = e0;
    if (threadIdx.x < 3) live[threadIdx.x] = 0;
    sh[ly + 1][lx + 1] = hh;
    bool alive = true;
    __syncthreads();
    for (int s = 0; s < sweeps; ++s) {
        // push half: heights fixed.  All loads first, the flows in registers,
        // then fire-and-forget atomics.
        int e = *(volatile int *)&se[ly + 1][lx + 1];
        if (e > 0 && hh <= hlim) {
            int cd[ND], hn[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                cd[d] = sc[d][ly + 1][lx + 1];
                hn[d] = sh[ly + 1 + dyd(d)][lx + 1 + dxd(d)];
            }
            const int e_in = e;
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                // zero or not: an add takes a cycle or two, a branch some twenty (with a
                // test or a predicate per add 640x480 penalty 600 took 950 us, now 808)
                const int f = hn[d] == hh - 1 ? min(e, cd[d]) : 0;
                e -= f;
                const int ny = ly + 1 + dyd(d), nx = lx + 1 + dxd(d);
                atomicAdd(&sc[d][ly + 1][lx + 1], -f);
                atomicAdd(&se[ny][nx], f);
                atomicAdd(&sc[opp(d)][ny][nx], f);
            }
            atomicAdd(&se[ly + 1][lx + 1], e - e_in);
        }
        if (threadIdx.x == 0) live[(s + 1) % 3] = 0;  // last read in sweep s - 2
        __syncthreads();
        // relabel half: capacities and excess fixed
        e = se[ly + 1][lx + 1];
        if (e > 0 && hh <= hlim) {
            int m = INF_H;
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const int hn = sh[ly + 1 + dyd(d)][lx + 1 + dxd(d)];
                m = min(m, sc[d][ly + 1][lx + 1] > 0 ? hn : INF_H);
            }
            if (m >= hh) hh = min(m, INF_H - 1) + 1;
            sh[ly + 1][lx + 1] = hh;
        }
        // still active?  A flag per sweep, three in rotation (set before a
        // barrier, read after it, cleared two sweeps later)
        if (__any_sync(0xffffffffu, e > 0 && hh <= hlim) && lx == 0) live[s % 3] = 1;
        __syncthreads();
        alive = live[s % 3] != 0;
        if (!alive) break;
    }
    if (alive && threadIdx.x == 0) g.due[t] = round + 1;
    if (inb) {
        g.h[i] = hh;
        const int de = se[ly + 1][lx + 1] - e0;
        if (de) atomicAdd(&g.e[i], de);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const int dc = sc[d][ly + 1][lx + 1] - c0[d];
            if (dc) atomicAdd(&g.cap[(long long)d * g.n + i], dc);
        }
    }
    if (rx >= 0 && se[ry][rx]) {  // flow left the tile here (only toward pixels of the image: their heights are finite)
        const int xx = x - lx + rx - 1, yy = y - ly + ry - 1;
        const long long j = (long long)yy * g.W + xx;
        atomicAdd(&g.e[j], se[ry][rx]);
#pragma unroll
        for (int d = 0; d < ND; ++d)
            if (sc[d][ry][rx]) atomicAdd(&g.cap[(long long)d * g.n + j], sc[d][ry][rx]);
        g.due[(yy / T8H) * tiles_x + xx / T8W] = round + 1;  // the tile it reached, in the next round
    }
    __syncthreads();  // the shared arrays are reused by the block's next tile
}

// ---- exact global relabel: a bit-parallel BFS per 32x32 tile ----
// Heights are 1 on the sink-connected pixels (excess < 0) and otherwise
// 1 + the fewest residual edges to one of them (INF when there is none), as a
// frontier BFS from those pixels would give.  First every tile's residual
// edges, sinks and active pixels become row masks (mask8_tile); then rounds
// over the tiles, one warp per tile with lane = row: a BFS of the whole tile
// from its sinks and from its ring's heights, eight directions by shifts and
// shuffles of the masks (bfs8_tile).  In round 0 the ring is the neighbours'
// sinks; in a later round a tile whose ring would lower one of its border
// pixels does its BFS again.  Every height ever written is the length of a
// real path to the sink (or INF), so a neighbour that reads a height
// mid-round reads a valid upper bound; a round in which no tile had a border
// pixel to lower leaves every residual edge with h(u) <= h(v) + 1, which with
// those upper bounds makes every height exact.  A shortest path about as long
// as a tile side crosses few tiles, so a relabel takes a few rounds (grid
// barriers) where a level-synchronous BFS takes one per level.
//
// (The relabel this replaced swept each tile to its fixpoint in shared memory,
// reading 36 KB of capacities per tile and round.)  A round of a 640x480 graph
// takes 8.4 us, of which the grid barrier is 2: the latency of one warp's BFS,
// 40 to 60 levels.
constexpr int G8W = 32, G8H = 32;
constexpr int G8_ROWS = G8H / 8;  // rows per thread (256 threads)
constexpr int NPLANE = 11;        // mask planes of a tile: 8 directions, excess < 0, excess > 0, reached by the BFS
constexpr int PL_NEG = 8, PL_POS = 9, PL_REACH = 10;
constexpr unsigned FULL8 = 0xffffffffu;

__device__ __forceinline__ const unsigned *plane8(const G8 &g, int t, int k) {
    return g.tm + ((size_t)t * NPLANE + k) * 32;
}

// Mask planes of tile t (one block).
__device__ void mask8_tile(const G8 &g, int t, int tiles_x) {
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int x = (t % tiles_x) * G8W + lane, y0 = (t / tiles_x) * G8H;
#pragma unroll
    for (int k = 0; k < G8_ROWS; ++k) {
        const int ly = wy + 8 * k, y = y0 + ly;
        const bool in = x < g.W && y < g.H;
        const long long i = (long long)y * g.W + x;
        int c[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d) c[d] = in ? __ldcg(g.cap + (long long)d * g.n + i) : 0;
        const int e = in ? __ldcg(g.e + i) : 0;
        unsigned w = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const unsigned m = __ballot_sync(FULL8, c[d] > 0);
            if (lane == d) w = m;
        }
        const unsigned neg = __ballot_sync(FULL8, e < 0), pos = __ballot_sync(FULL8, e > 0);
        if (lane == PL_NEG) w = neg;
        if (lane == PL_POS) w = pos;
        if (lane <= PL_POS) g.tm[((size_t)t * NPLANE + lane) * 32 + ly] = w;
    }
}

// Heights around a tile: hl / hr beside the lane's row, ht / hb above and
// below column `lane`, and the four corners (the same in every lane).
struct Ring8 {
    int hl, hr, ht, hb, tl, tr, bl, br;
};

// Smallest ring level above lvl (warp-uniform), INF when there is none.
__device__ __forceinline__ int next_ring8(const Ring8 &q, int lvl) {
    int m = INF_H;
    const int v[8] = {q.hl, q.hr, q.ht, q.hb, q.tl, q.tr, q.bl, q.br};
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (v[k] > lvl) m = min(m, v[k]);
    return __reduce_min_sync(FULL8, m);
}

// Scratch of one warp: the index of the expansion that reached each pixel as
// bit planes per row, and the level of each index.
constexpr int B8_PL = 7, B8_IDX = 1 << B8_PL;
struct Bfs8Scratch {
    unsigned pl[B8_PL][32], reached[32], base[32];
    int lv[B8_IDX];
};

// BFS of the tile with first pixel (x0, y0) on its planes m, the ring q; the
// heights go to g.h.  A pixel's expansion index is kept in bit planes and the
// heights are written row by row afterwards (coalesced); after B8_IDX
// expansions the levels so far are written and the planes start again.
__device__ unsigned bfs8_tile(const G8 &g, int x0, int y0, const unsigned m[9], const Ring8 &q, int hlim,
                              Bfs8Scratch &sc) {
    const int lane = threadIdx.x & 31;
    unsigned S = m[PL_NEG], base = 0u, P[B8_PL];
#pragma unroll
    for (int k = 0; k < B8_PL; ++k) P[k] = 0u;
    if (lane == 0) sc.lv[0] = 1;
    int nidx = 4, lvl = 1;  // index 0: the seeds; expansions in fours from 4 on
    auto expand = [&](unsigned S, int lvl) -> unsigned {
        const unsigned T = __ballot_sync(FULL8, q.ht <= lvl), B = __ballot_sync(FULL8, q.hb <= lvl);
        const unsigned side = (q.hl <= lvl ? 1u : 0u) | (q.hr <= lvl ? 0x80000000u : 0u);  // ring beside this row
        unsigned up = __shfl_up_sync(FULL8, S, 1), dn = __shfl_down_sync(FULL8, S, 1);
        unsigned su = __shfl_up_sync(FULL8, side, 1), sd = __shfl_down_sync(FULL8, side, 1);  // beside the rows above, below
        if (lane == 0) {
            up = T;
            su = (q.tl <= lvl ? 1u : 0u) | (q.tr <= lvl ? 0x80000000u : 0u);
        }
        if (lane == 31) {
            dn = B;
            sd = (q.bl <= lvl ? 1u : 0u) | (q.br <= lvl ? 0x80000000u : 0u);
        }
        const unsigned near = (m[0] & ((S << 1) | (side & 1u))) | (m[1] & ((S >> 1) | (side & 0x80000000u))) |
                              (m[2] & up) | (m[3] & dn);
        const unsigned diag = (m[4] & ((up << 1) | (su & 1u))) | (m[5] & ((up >> 1) | (su & 0x80000000u))) |
                              (m[6] & ((dn << 1) | (sd & 1u))) | (m[7] & ((dn >> 1) | (sd & 0x80000000u)));
        return (near | diag) & ~S;
    };
    auto flush = [&](bool final) {
#pragma unroll
        for (int k = 0; k < B8_PL; ++k) sc.pl[k][lane] = P[k];
        sc.reached[lane] = S;
        sc.base[lane] = base;
        __syncwarp();
        const unsigned bit = 1u << lane;
        const bool col_in = x0 + lane < g.W;
#pragma unroll 4
        for (int r = 0; r < 32; ++r) {
            const unsigned sr = sc.reached[r], br = sc.base[r];
            int idx = 0;
#pragma unroll
            for (int k = 0; k < B8_PL; ++k) idx |= (int)((sc.pl[k][r] >> lane) & 1u) << k;
            const bool fresh = ((sr & ~br) & bit) != 0;
            const int v = fresh ? sc.lv[idx] : INF_H;
            if (col_in && y0 + r < g.H && (fresh || (final && !(sr & bit))))
                g.h[(long long)(y0 + r) * g.W + x0 + lane] = v;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < B8_PL; ++k) P[k] = 0u;
        base = S;
        nidx = 0;
    };
    // four levels per vote; a BFS ends after at most one expansion per pixel
    // and ring level.  The four of a vote share the upper bits of their index.
    for (int it = 0; it < G8W * G8H + 4 * 32 + 8 && lvl < hlim; ++it) {
        const unsigned nw1 = expand(S, lvl);
        const unsigned S1 = S | nw1;
        const unsigned nw2 = expand(S1, lvl + 1);
        const unsigned S2 = S1 | nw2;
        const unsigned nw3 = expand(S2, lvl + 2);
        const unsigned S3 = S2 | nw3;
        const unsigned nw4 = expand(S3, lvl + 3);
        const unsigned all = nw1 | nw2 | nw3 | nw4;
        if (__any_sync(FULL8, all != 0)) {
            if (nidx + 4 > B8_IDX) flush(false);
            P[0] |= nw2 | nw4;
            P[1] |= nw3 | nw4;
#pragma unroll
            for (int k = 2; k < B8_PL; ++k)
                if ((nidx >> k) & 1) P[k] |= all;  // warp-uniform
            if (lane < 4) sc.lv[nidx + lane] = lvl + 1 + lane;
            S = S3 | nw4;
            nidx += 4;
            lvl += 4;
        } else {
            const int nxt = next_ring8(q, lvl + 3);
            if (nxt >= INF_H) break;
            lvl = nxt;
        }
    }
    flush(true);
    return S;
}

// One warp's visit of tile t in a relabel round.  Returns whether it did the
// BFS (round 0: always).
__device__ bool gr8_tile(const G8 &g, int t, int tiles_x, int tiles_y, bool round0, int hlim,
                         Bfs8Scratch &sc) {
    const int lane = threadIdx.x & 31;
    const int tx = t % tiles_x, ty = t / tiles_x;
    const int x0 = tx * G8W, y0 = ty * G8H;
    unsigned m[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) m[k] = __ldcg(plane8(g, t, k) + lane);
    Ring8 q;
    if (round0) {
        const bool L = tx > 0, R = tx < tiles_x - 1, U = ty > 0, D = ty < tiles_y - 1;
        // sinks of the neighbour tile at offset o from t: row `row`, bit x
        auto sink = [&](bool there, int o, int row, int x) {
            return there && ((__ldcg(plane8(g, t + o, PL_NEG) + row) >> x) & 1u) ? 1 : INF_H;
        };
        q.hl = sink(L, -1, lane, 31);
        q.hr = sink(R, 1, lane, 0);
        q.ht = sink(U, -tiles_x, 31, lane);
        q.hb = sink(D, tiles_x, 0, lane);
        q.tl = sink(U && L, -tiles_x - 1, 31, 31);
        q.tr = sink(U && R, -tiles_x + 1, 31, 0);
        q.bl = sink(D && L, tiles_x - 1, 0, 31);
        q.br = sink(D && R, tiles_x + 1, 0, 0);
    } else {
        auto at = [&](int xx, int yy) -> int {
            return xx < 0 || yy < 0 || xx >= g.W || yy >= g.H ? INF_H : *(volatile const int *)&g.h[(long long)yy * g.W + xx];
        };
        q.hl = at(x0 - 1, y0 + lane);
        q.hr = at(x0 + G8W, y0 + lane);
        q.ht = at(x0 + lane, y0 - 1);
        q.hb = at(x0 + lane, y0 + G8H);
        q.tl = at(x0 - 1, y0 - 1);
        q.tr = at(x0 + G8W, y0 - 1);
        q.bl = at(x0 - 1, y0 + G8H);
        q.br = at(x0 + G8W, y0 + G8H);
        // would the ring lower a border pixel?  Each side: the least ring level
        // that a border pixel's residual edges reach, against its own height.
        const int ol = at(x0, y0 + lane), orr = at(x0 + G8W - 1, y0 + lane);
        const int ot = at(x0 + lane, y0), ob = at(x0 + lane, y0 + G8H - 1);
        auto edge = [](unsigned w, int x, int h) { return (w >> x) & 1u ? h : INF_H; };
        // left and right columns (lane = row): straight, and the diagonals to the ring beside rows lane -+ 1
        int lu = __shfl_up_sync(FULL8, q.hl, 1), ld = __shfl_down_sync(FULL8, q.hl, 1);
        int ru = __shfl_up_sync(FULL8, q.hr, 1), rd = __shfl_down_sync(FULL8, q.hr, 1);
        int tl = __shfl_up_sync(FULL8, q.ht, 1), tr = __shfl_down_sync(FULL8, q.ht, 1);
        int bl = __shfl_up_sync(FULL8, q.hb, 1), br = __shfl_down_sync(FULL8, q.hb, 1);
        if (lane == 0) { lu = q.tl; ru = q.tr; tl = q.tl; bl = q.bl; }
        if (lane == 31) { ld = q.bl; rd = q.br; tr = q.tr; br = q.br; }
        const int vl = min(edge(m[0], 0, q.hl), min(edge(m[4], 0, lu), edge(m[6], 0, ld)));
        const int vr = min(edge(m[1], 31, q.hr), min(edge(m[5], 31, ru), edge(m[7], 31, rd)));
        // top and bottom rows (lane = column): the masks of rows 0 and 31
        const int vt = min(edge(__shfl_sync(FULL8, m[2], 0), lane, q.ht),
                           min(edge(__shfl_sync(FULL8, m[4], 0), lane, tl), edge(__shfl_sync(FULL8, m[5], 0), lane, tr)));
        const int vb = min(edge(__shfl_sync(FULL8, m[3], 31), lane, q.hb),
                           min(edge(__shfl_sync(FULL8, m[6], 31), lane, bl), edge(__shfl_sync(FULL8, m[7], 31), lane, br)));
        const bool imp = (vl < hlim && vl + 1 < ol) || (vr < hlim && vr + 1 < orr) || (vt < hlim && vt + 1 < ot) ||
                         (vb < hlim && vb + 1 < ob);
        if (!__any_sync(FULL8, imp)) return false;
    }
    g.tm[((size_t)t * NPLANE + PL_REACH) * 32 + lane] = bfs8_tile(g, x0, y0, m, q, hlim, sc);
    return true;
}

// ---- the source-side closure (S_min) by rounds over 32x32 tiles ----
// Marks start on the pixels with excess > 0; a visit stages the marks of the
// tile and its ring, spreads them along the residual edges of the tile's
// pixels (inside the tile and onto the ring) until nothing changes, and
// writes the new marks back, ring pixels included (their own tile spreads
// them in a later round).  Marks only ever go from 0 to 1, so a round in
// which no visit wrote a mark leaves every residual edge out of a marked
// pixel ending at a marked pixel: the marks are the closure.  Returns
// whether the visit wrote a mark.
__device__ bool reach8_tile(const G8 &g, int t, int tiles_x) {
    __shared__ int gm[G8H + 2][G8W + 2];
    const int lx = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int x0 = (t % tiles_x) * G8W, y0 = (t / tiles_x) * G8H;
    auto outside = [&](int xx, int yy) { return xx < 0 || yy < 0 || xx >= g.W || yy >= g.H; };
    // a cell outside the image counts as marked, so that nothing is written there
    auto mark_at = [&](int xx, int yy) -> int {
        return outside(xx, yy) ? 1 : *(volatile const int *)&g.mark[(long long)yy * g.W + xx];
    };
    unsigned rm[G8_ROWS];
    int m0[G8_ROWS];
#pragma unroll
    for (int k = 0; k < G8_ROWS; ++k) {
        const int ly = wy + 8 * k, x = x0 + lx, y = y0 + ly;
        const int mv = mark_at(x, y);
        unsigned m = 0;
        if (!outside(x, y)) {
            const long long i = (long long)y * g.W + x;
#pragma unroll
            for (int d = 0; d < ND; ++d) m |= (g.cap[(long long)d * g.n + i] > 0 ? 1u : 0u) << d;
        }
        rm[k] = m;
        m0[k] = mv;
        gm[ly + 1][lx + 1] = mv;
    }
    // the ring: warps 0-3 one side each, warp 4 the corners; each keeps what it read
    int rx = 0, ry = 0, r0 = 1;
    if (wy < 4 || (wy == 4 && lx < 4)) {
        if (wy == 0) { rx = lx + 1; ry = 0; }
        else if (wy == 1) { rx = lx + 1; ry = G8H + 1; }
        else if (wy == 2) { rx = 0; ry = lx + 1; }
        else if (wy == 3) { rx = G8W + 1; ry = lx + 1; }
        else { rx = lx & 1 ? G8W + 1 : 0; ry = lx & 2 ? G8H + 1 : 0; }
        r0 = mark_at(x0 - 1 + rx, y0 - 1 + ry);
        gm[ry][rx] = r0;
    }
    __syncthreads();
    // each sweep that changes something marks a new cell of the tile or ring
    for (int s = 0; s <= (G8W + 2) * (G8H + 2); ++s) {
        bool ch = false;
#pragma unroll
        for (int k = 0; k < G8_ROWS; ++k) {
            const int ly = wy + 8 * k;
            if (!rm[k] || !gm[ly + 1][lx + 1]) continue;
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                if (!((rm[k] >> d) & 1u)) continue;
                int *cell = &gm[ly + 1 + dyd(d)][lx + 1 + dxd(d)];
                if (!*cell) {
                    *cell = 1;
                    ch = true;
                }
            }
        }
        if (!__syncthreads_or(ch)) break;
    }
    bool wrote = false;
#pragma unroll
    for (int k = 0; k < G8_ROWS; ++k) {
        const int ly = wy + 8 * k, x = x0 + lx, y = y0 + ly;
        if (!m0[k] && gm[ly + 1][lx + 1]) {  // m0 is 1 outside the image
            g.mark[(long long)y * g.W + x] = 1;
            wrote = true;
        }
    }
    if (!r0 && gm[ry][rx]) {  // r0 is 1 for threads without a ring cell and outside the image
        g.mark[(long long)(y0 - 1 + ry) * g.W + (x0 - 1 + rx)] = 1;
        wrote = true;
    }
    return __syncthreads_or(wrote);  // also: gm is reused by the block's next tile
}

__global__ void __launch_bounds__(256) k8_solve(G8 g, P8 prm) {
    Ctl8 *c = g.ctl;
    const long long gtid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nth = (long long)gridDim.x * blockDim.x;
    bool finished = false;
    int R = 0;  // tile and relabel rounds so far in this solve (grid-uniform)
    const int gtiles_x = (g.W + G8W - 1) / G8W;
    const int gtiles_y = (g.H + G8H - 1) / G8H, gtiles = gtiles_x * gtiles_y;
    __shared__ Bfs8Scratch sc[8];
    __shared__ unsigned s_todo;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int swarp = warp * gridDim.x + blockIdx.x, nwarps = gridDim.x * 8;  // block-interleaved warp rank
    for (int outer = 0; outer < prm.max_outer; ++outer) {
        // ---- exact global relabel (mask8_tile, then gr8_tile rounds); with a
        // height limit one further round after round 0, and heights that may
        // come out too high ----
        // The round counters are the tile rounds' (round_active, R), with the
        // same clearing rule.
        const int hlim = outer == 0 && prm.near_h > 0 ? prm.near_h : INF_H - 1;
        if (gtid == 0) c->active = 0;
        for (int t = blockIdx.x; t < gtiles; t += gridDim.x) mask8_tile(g, t, gtiles_x);
        if (!sync8(c)) return;
        for (int q = 0;; ++q) {
            if (gtid == 0) c->round_active[(R + 1) % 3] = 0;
            int changed = 0;
            for (int t = swarp; t < gtiles; t += nwarps)
                changed += gr8_tile(g, t, gtiles_x, gtiles_y, q == 0, hlim, sc[warp]);
            if (lane == 0 && changed) atomicAdd(&c->round_active[R % 3], changed);
            if (gtid == 0) c->gr_rounds++;
            if (!sync8(c)) return;
            const int more = *(volatile int *)&c->round_active[R % 3];
            ++R;
            if (!more || (hlim < INF_H - 1 && q == 1)) break;
            if (q > g.n) {  // unreachable: a round makes at least one more path segment exact
                if (gtid == 0) set_err8(c, E8_OUTER);
                return;
            }
        }
        if (gtid == 0) c->global_relabels++;
        // ---- count: excess that can still reach the sink (lane = row of a
        // 32x32 tile), and the tiles of the first round ----
        unsigned act = 0;
        const int tiles_x = (g.W + T8W - 1) / T8W, tiles_y = (g.H + T8H - 1) / T8H;
        const int ntiles = tiles_x * tiles_y;
        for (int t = swarp; t < gtiles; t += nwarps) {
            const unsigned w = __ldcg(plane8(g, t, PL_POS) + lane) & __ldcg(plane8(g, t, PL_REACH) + lane);
            act += __popc(w);
            const unsigned rows = __ballot_sync(FULL8, w != 0);
            const int ty8 = (t / gtiles_x) * (G8H / T8H) + lane;  // lanes 0..3: the tile's 32x8 quarters
            if (lane < G8H / T8H && ((rows >> (T8H * lane)) & 0xFFu)) g.due[ty8 * tiles_x + t % gtiles_x] = R;
        }
        act = __reduce_add_sync(0xffffffffu, act);
        if ((threadIdx.x & 31) == 0 && act) atomicAdd(&c->active, (unsigned long long)act);
        if (gtid == 0) c->round_active[(R + 1) % 3] = 0;
        if (!sync8(c)) return;
        if (*(volatile unsigned long long *)&c->active == 0) {
            if (hlim < INF_H - 1) continue;  // none within the limit: the exact relabel next
            finished = true;
            break;
        }
        // ---- tile rounds: the due tiles, block-local sweeps ----
        // A graph that takes a fourth relabel moves its flow far: three times the
        // rounds per relabel from there on (640x480 penalty 600 808 -> 771 us,
        // 1920x1080 3086 -> 2596, 200x150 penalty 100 1303 -> 1109; twice 785,
        // 2631, 1189; graphs of fewer relabels are unchanged).
        const int rounds = outer > 2 ? 3 * prm.rounds : prm.rounds;
        for (int p = 0; p < rounds; ++p) {
            // round_active[R % 3] counts this round's tiles and is read after the
            // round's barrier; the counter of round R + 1 was last read after
            // the barrier of round R - 2, which every block has passed
            if (gtid == 0) c->round_active[(R + 1) % 3] = 0;
            int worked = 0;
            // the block's tiles 32 at a time, their stamps in one load
            for (int tb = blockIdx.x; tb < ntiles; tb += 32 * gridDim.x) {  // block-uniform
                const int mine = tb + lane * gridDim.x;
                unsigned todo = __ballot_sync(FULL8, mine < ntiles && *(volatile int *)(g.due + mine) >= R);
                // (a neighbour may raise a stamp meanwhile: thread 0's reading decides for the block)
                if (threadIdx.x == 0) s_todo = todo;
                __syncthreads();
                todo = s_todo;
                for (; todo; todo &= todo - 1) {
                    tile8_visit(g, tb + (__ffs(todo) - 1) * gridDim.x, tiles_x, prm.sweeps, hlim, R);
                    ++worked;
                }
                __syncthreads();
            }
            if (threadIdx.x == 0 && worked) {
                atomicAdd(&c->round_active[R % 3], worked);
                atomicAdd(&c->tile_visits, (unsigned long long)worked);
            }
            if (gtid == 0) c->tile_rounds++;
            if (!sync8(c)) return;
            const int done_round = *(volatile int *)&c->round_active[R % 3] == 0;
            ++R;
            if (done_round) break;  // nothing left to push: relabel
        }
    }
    if (!finished) {
        if (gtid == 0) set_err8(c, E8_OUTER);
        return;
    }
    // ---- final positive excess and the source-side closure (S_min) ----
    unsigned long long pos = 0;
    for (long long i = gtid; i < g.n; i += nth) {
        const int e = g.e[i];
        if (e > 0) pos += (unsigned)e;
        g.mark[i] = e > 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pos += __shfl_down_sync(0xffffffffu, pos, o);
    if ((threadIdx.x & 31) == 0 && pos) atomicAdd(&c->pos_excess, pos);
    if (!sync8(c)) return;
    if (*(volatile unsigned long long *)&c->pos_excess == 0) return;  // nothing marked: S_min is empty
    for (int q = 0;; ++q) {
        if (gtid == 0) c->round_active[(R + 1) % 3] = 0;
        int changed = 0;
        for (int t = blockIdx.x; t < gtiles; t += gridDim.x) changed += reach8_tile(g, t, gtiles_x);
        if (threadIdx.x == 0 && changed) atomicAdd(&c->round_active[R % 3], changed);
        if (gtid == 0) c->reach_rounds++;
        if (!sync8(c)) return;
        const int more = *(volatile int *)&c->round_active[R % 3];
        ++R;
        if (!more) break;
        if (q > g.n) {  // unreachable: every round but the last marks at least one more pixel
            if (gtid == 0) set_err8(c, E8_OUTER);
            return;
        }
    }
}

__global__ void k8_extract(G8 g, int *label, uint8_t *smin, uint8_t *smax) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < g.n; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % g.W), y = (int)(i / g.W);
        const bool inside = x > 0 && y > 0 && x < g.W - 1 && y < g.H - 1;
        const int s = inside && g.h[i] >= INF_H;
        if (label) label[i] = s;
        if (smax) smax[i] = (uint8_t)s;
        if (smin) smin[i] = (uint8_t)g.mark[i];
    }
}

int grid8(long long n) {
    long long b = (n + 255) / 256;
    return (int)(b < 4096 ? (b > 0 ? b : 1) : 4096);
}

}  // namespace
}  // namespace gcfg

using namespace gcfg;

struct gcfg_graph8 {
    int W = 0, H = 0;
    long long n = 0;
    const int32_t *dp = nullptr, *dn = nullptr;
    const int32_t *arr[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    int32_t penalty = 0;
    bool varying = false, built = false, solved = false;
    int *cap = nullptr, *e = nullptr, *h = nullptr, *mark = nullptr;
    unsigned *tm = nullptr;
    int *due = nullptr;
    int32_t *d_label = nullptr;
    Ctl8 *ctl = nullptr, *h_ctl = nullptr;
    cudaStream_t st = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr;  // solve start, solve end, extract end
    // schedule: 8 sweeps per visit; solve kernel at 12 / 8 / 6 tile rounds per
    // global relabel (the same to the end): 640x480, penalty 600 801 / 808 / 840
    // us, penalty 20 398 / 345 / 321, arrays 175 / 166 / 156, 1920x1080 penalty
    // 600 2682 / 3086 / 3388; with three times as many from the fourth relabel on
    // 8 rounds take 771, 347, 166 and 2596 (12 sweeps 825, 363, 178, 2636; 6 sweeps,
    // twice as many, 802, 331, 163, 2895).  2 blocks per SM: 874, 361, 169, 3278
    int rounds = GCFG_N8_ROUNDS, max_outer = 100000, blocks_per_sm = 3, sweeps = GCFG_N8_SWEEPS;

    G8 g() const {
        G8 x;
        x.W = W;
        x.H = H;
        x.n = n;
        x.cap = cap;
        x.e = e;
        x.h = h;
        x.mark = mark;
        x.tm = tm;
        x.due = due;
        x.ctl = ctl;
        return x;
    }
    void release() {
        cudaFree(cap); cudaFree(e); cudaFree(h); cudaFree(mark);
        cudaFree(d_label); cudaFree(ctl); cudaFree(tm); cudaFree(due);
        if (h_ctl) cudaFreeHost(h_ctl);
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
        if (ev2) cudaEventDestroy(ev2);
    }
};

extern "C" {

gcfg_status gcfg_set_dataterms8(gcfg_graph8 *g, const int32_t *dp, const int32_t *dn) {
    if (!g) return GCFG_ERR_INVALID;
    g->dp = dp;
    g->dn = dn;
    g->built = false;
    return GCFG_OK;
}

gcfg_status gcfg_set_edges8(gcfg_graph8 *g, const int32_t *up, const int32_t *down, const int32_t *left,
                            const int32_t *right, const int32_t *upleft, const int32_t *upright,
                            const int32_t *downleft, const int32_t *downright) {
    if (!g || !up || !down || !left || !right || !upleft || !upright || !downleft || !downright)
        return GCFG_ERR_INVALID;
    const int32_t *a[8] = {left, right, up, down, upleft, upright, downleft, downright};
    memcpy(g->arr, a, sizeof(a));
    g->varying = true;
    g->built = false;
    return GCFG_OK;
}

gcfg_status gcfg_set_penalty8(gcfg_graph8 *g, int32_t penalty) {
    if (!g || penalty < 0 || penalty > GCFG_MAX_CAP8) return GCFG_ERR_INVALID;
    g->penalty = penalty;
    g->varying = false;
    g->built = false;
    return GCFG_OK;
}

gcfg_status gcfg_set_schedule8(gcfg_graph8 *g, int rounds_per_gr, int blocks_per_sm) {
    if (!g || rounds_per_gr < 1 || blocks_per_sm < 0) return GCFG_ERR_INVALID;
    g->rounds = rounds_per_gr;
    g->blocks_per_sm = blocks_per_sm;
    return GCFG_OK;
}

gcfg_status gcfg_set_stream8(gcfg_graph8 *g, void *stream) {
    if (!g) return GCFG_ERR_INVALID;
    g->st = (cudaStream_t)stream;
    return GCFG_OK;
}

gcfg_status gcfg_set_graph8(gcfg_graph8 *g) {
    if (!g || !g->dp || !g->dn) return GCFG_ERR_STATE;
    GCFG_CK(cudaMemsetAsync(g->ctl, 0, sizeof(Ctl8), g->st));
    GCFG_CK(cudaMemsetAsync(g->due, 0xff, (size_t)((g->W + 31) / 32) * ((g->H + 7) / 8) * sizeof(int), g->st));
    Arr8 arr;
    for (int d = 0; d < 8; ++d) arr.a[d] = g->varying ? g->arr[d] : nullptr;
    k8_build<<<grid8(g->n), 256, 0, g->st>>>(g->g(), g->dp, g->dn, g->penalty, arr);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    GCFG_CK(cudaGetLastError());
    GCFG_CK(cudaMemcpyAsync(g->h_ctl, g->ctl, sizeof(Ctl8), cudaMemcpyDeviceToHost, g->st));
    GCFG_CK(cudaStreamSynchronize(g->st));
    if (g->h_ctl->err) return GCFG_ERR_INVALID;  // capacities outside [0, GCFG_MAX_CAP8]
    g->built = true;
    g->solved = false;
    return GCFG_OK;
}

gcfg_status gcfg_init8(int w, int h, const int32_t *dp, const int32_t *dn, int32_t penalty, const int32_t *up,
                       const int32_t *down, const int32_t *left, const int32_t *right, const int32_t *upleft,
                       const int32_t *upright, const int32_t *downleft, const int32_t *downright,
                       gcfg_graph8 **out) {
    if (!out || w <= 0 || h <= 0 || (long long)w * h > (1LL << 31) - 1) return GCFG_ERR_INVALID;
    if (penalty < 0 || penalty > GCFG_MAX_CAP8) return GCFG_ERR_INVALID;
    gcfg_graph8 *g = new gcfg_graph8();
    g->W = w;
    g->H = h;
    g->n = (long long)w * h;
    g->penalty = penalty;
    const size_t n = (size_t)g->n;
    gcfg_status rc = GCFG_OK;
    if (cudaMalloc(&g->cap, 8 * n * sizeof(int)) != cudaSuccess || cudaMalloc(&g->e, n * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&g->h, n * sizeof(int)) != cudaSuccess || cudaMalloc(&g->mark, n * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&g->d_label, n * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&g->tm, (size_t)((w + 31) / 32) * ((h + 31) / 32) * NPLANE * 32 * sizeof(unsigned)) != cudaSuccess ||
        cudaMalloc(&g->due, (size_t)((w + 31) / 32) * ((h + 7) / 8) * sizeof(int)) != cudaSuccess || cudaMalloc(&g->ctl, sizeof(Ctl8)) != cudaSuccess ||
        cudaMallocHost(&g->h_ctl, sizeof(Ctl8)) != cudaSuccess)
        rc = GCFG_ERR_OOM;
    if (rc == GCFG_OK && (cudaEventCreate(&g->ev0) != cudaSuccess || cudaEventCreate(&g->ev1) != cudaSuccess ||
                          cudaEventCreate(&g->ev2) != cudaSuccess))
        rc = GCFG_ERR_CUDA;
    if (rc == GCFG_OK && dp) {
        gcfg_set_dataterms8(g, dp, dn);
        if (up) rc = gcfg_set_edges8(g, up, down, left, right, upleft, upright, downleft, downright);
        if (rc == GCFG_OK) rc = gcfg_set_graph8(g);
    }
    if (rc) {
        g->release();
        delete g;
        return rc;
    }
    *out = g;
    return GCFG_OK;
}

gcfg_status gcfg_optimize8(gcfg_graph8 *g, int32_t *host_label, gcfg_result *res) {
    if (!g) return GCFG_ERR_INVALID;
    if (!g->built) return GCFG_ERR_STATE;
    int per_sm = 0, sms = 0, dev = 0;
    GCFG_CK(cudaGetDevice(&dev));
    GCFG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GCFG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k8_solve, 256, 0));
    long long want = (g->n + 255) / 256;
    if (g->blocks_per_sm > 0 && g->blocks_per_sm < per_sm) per_sm = g->blocks_per_sm;
    long long grid = (long long)(per_sm > 0 ? per_sm : 1) * (sms > 0 ? sms : 1);
    if (want < grid) grid = want > 0 ? want : 1;
    G8 gg = g->g();
    // A height limit for the first iteration pays where edges saturate, as
    // contrast-sensitive ones do (640x480 / 1920x1080, us without -> with: arrays
    // 272 -> 177, 602 -> 393).  A constant penalty leaves most of them open and
    // flow has to travel: penalty 600 770 -> 862, 2473 -> 2662; penalty 100, where
    // some saturate, 1803 -> 1719, 2459 -> 2032 (three graphs each; the penalty
    // given by itself and as arrays).
    P8 prm{g->max_outer, g->rounds < MAX_ROUNDS8 ? g->rounds : MAX_ROUNDS8, g->sweeps, g->varying ? 9 : 0};
    void *args[] = {&gg, &prm};
    GCFG_CK(cudaEventRecord(g->ev0, g->st));
    GCFG_CK(cudaLaunchCooperativeKernel((const void *)k8_solve, dim3((unsigned)grid), dim3(256), args, 0, g->st));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    GCFG_CK(cudaEventRecord(g->ev1, g->st));
    k8_extract<<<grid8(g->n), 256, 0, g->st>>>(gg, g->d_label, nullptr, nullptr);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    GCFG_CK(cudaGetLastError());
    GCFG_CK(cudaEventRecord(g->ev2, g->st));
    if (host_label)
        GCFG_CK(cudaMemcpyAsync(host_label, g->d_label, (size_t)g->n * sizeof(int32_t), cudaMemcpyDeviceToHost, g->st));
    GCFG_CK(cudaMemcpyAsync(g->h_ctl, g->ctl, sizeof(Ctl8), cudaMemcpyDeviceToHost, g->st));
    GCFG_CK(cudaStreamSynchronize(g->st));
    g->built = false;  // the graph is consumed, as in the reference
    const Ctl8 &c = *g->h_ctl;
    const gcfg_status st = c.err ? GCFG_ERR_NOT_CONVERGED : GCFG_OK;
    g->solved = st == GCFG_OK;
    if (res) {
        memset(res, 0, sizeof(*res));
        res->flow = (long long)c.interior_dp - (long long)c.pos_excess;
        res->ref_energy = (int32_t)((uint32_t)c.ref_init - (uint32_t)c.pos_excess);
        res->status = st;
        res->global_relabels = c.global_relabels;
        res->gr_sweeps = c.gr_rounds;
        res->push_rounds = c.tile_rounds;
        res->cut_sweeps = c.reach_rounds;
        res->push_tiles = (int64_t)c.tile_visits;
        res->gr_tiles = (int64_t)c.gr_rounds * (((g->W + G8W - 1) / G8W) * (long long)((g->H + G8H - 1) / G8H));
        float ms = 0.f;
        cudaEventElapsedTime(&ms, g->ev0, g->ev1);
        res->ms = ms;
    }
    return st;
}

gcfg_status gcfg_get_cuts8(gcfg_graph8 *g, uint8_t *d_smin, uint8_t *d_smax) {
    if (!g) return GCFG_ERR_INVALID;
    if (!g->solved) return GCFG_ERR_STATE;
    k8_extract<<<grid8(g->n), 256, 0, g->st>>>(g->g(), nullptr, d_smin, d_smax);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    GCFG_CK(cudaGetLastError());
    GCFG_CK(cudaStreamSynchronize(g->st));
    return GCFG_OK;
}

gcfg_status gcfg_end8(gcfg_graph8 *g) {
    if (!g) return GCFG_ERR_INVALID;
    cudaStreamSynchronize(g->st);
    g->release();
    delete g;
    return GCFG_OK;
}

}  // extern "C"
