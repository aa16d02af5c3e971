// lb_ensemble.cu -- many independent periodic D2Q9 Shan-Chen domains of
// different sizes advanced together (include/lbgb300.h, ensemble API).
//
// All domains live in one packed structure-of-arrays slab (domain d occupies
// nodes [off_d, off_d + W_d*H_d), node x + W_d*y inside it), in two
// population sets that alternate like the single-lattice context.  A step
// walks a host-built work list (a domain's extents and physics, a first row
// and column).  By default one launch advances one or two steps by strips of
// column pairs, or by strips of 32 columns on ensembles of many narrow domains
// (ens_strips_pay); the other forms are tiles, and two persistent launches
// over row groups: the density pass writes psi = psi(rho) of every node, the
// fused pass pulls the populations, adds the Shan-Chen shift from the 3x3 psi
// stencil and relaxes.  In the persistent forms each block walks the list with
// a stride of the grid size, and the grid is a multiple of the SM count, so
// uneven domain sizes do not leave SMs idle.  Batches of steps are replayed
// from a captured CUDA graph.  lb_ensemble_autotune times each form on the
// ensemble itself.
//
// The per-node arithmetic is the single-domain native D2Q9 Shan-Chen step's
// (same device functions, same order: d2q9_moments_native,
// d2q9_sc_shift_native, d2q9_bgk_native), so a domain of the ensemble evolves
// bit for bit like the same domain run alone through the context API.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/lbgb300.h"
#include "lb_pairs.cuh"

using namespace lb;

namespace {

struct EnsDomain {
    int W, H, off;
    float G, tau_inv;
};

// one work item: a group of rows of one domain, with the domain's extents
// and physics copied in, so that a block needs one load (not two dependent
// ones) before it can address its populations
struct EnsItem {
    int off, W, H, y;
    float G, tau_inv;
    int x;  // single-pass tiles: first column of the tile (0 for row groups)
};

struct EnsArgs {
    const float *src[9];
    float *dst[9];
    float *psi;
    float *rho, *ux, *uy;
    const EnsItem *items;
    int nitems;
    int psi_form;
    float w0, w1, w5;
};

// pull of node (x, y) of a periodic domain starting at node `off`
__device__ __forceinline__ void ens_pull(const EnsArgs &a, const EnsItem &dm, int x, int y,
                                         float (&g)[9]) {
    const int xm = x == 0 ? dm.W - 1 : x - 1, xp = x == dm.W - 1 ? 0 : x + 1;
    const int rm = y == 0 ? dm.H - 1 : y - 1, rp = y == dm.H - 1 ? 0 : y + 1;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        // upstream node x - c_k (row offset -cr_k)
        const int ux = d2_cx(k) > 0 ? xm : (d2_cx(k) < 0 ? xp : x);
        const int uy = d2_cr(k) > 0 ? rm : (d2_cr(k) < 0 ? rp : y);
        g[k] = __ldg(a.src[k] + dm.off + ux + dm.W * uy);
    }
}

// Both passes walk the work list with a stride of the grid size and load the
// next item while they work on the current one.
template <int PSI>
__global__ void ens_density_kernel(const EnsArgs a) {
    int it = blockIdx.x;
    if (it >= a.nitems) return;
    EnsItem dm = a.items[it];
    for (; it < a.nitems; it += gridDim.x) {
        const int nit = it + gridDim.x;
        const EnsItem next = nit < a.nitems ? a.items[nit] : dm;
        const int y = dm.y + threadIdx.y;
        if (y < dm.H) {
            for (int x = threadIdx.x; x < dm.W; x += blockDim.x) {
                float g[9];
                ens_pull(a, dm, x, y, g);
                const float rho = d2q9_rho_native(g);
                a.psi[dm.off + x + dm.W * y] = psi_form<PSI>(rho);
            }
        }
        dm = next;
    }
}

template <bool MOM>
__global__ void ens_fused_kernel(const EnsArgs a) {
    int it = blockIdx.x;
    if (it >= a.nitems) return;
    EnsItem next = a.items[it];
    for (; it < a.nitems; it += gridDim.x) {
        const EnsItem dm = next;
        const int nit = it + gridDim.x;
        if (nit < a.nitems) next = a.items[nit];
        const int y = dm.y + threadIdx.y;
        if (y >= dm.H) continue;
        const int rm = y == 0 ? dm.H - 1 : y - 1, rp = y == dm.H - 1 ? 0 : y + 1;
        const float *psi = a.psi + dm.off;
        for (int x = threadIdx.x; x < dm.W; x += blockDim.x) {
            float g[9];
            ens_pull(a, dm, x, y, g);
            float rho, ux, uy;
            d2q9_moments_native(g, rho, ux, uy);
            const int xm = x == 0 ? dm.W - 1 : x - 1, xp = x == dm.W - 1 ? 0 : x + 1;
            const int W = dm.W;
            const float ps[9] = {__ldg(psi + x + W * y),   __ldg(psi + xp + W * y),
                                 __ldg(psi + x + W * rp),  __ldg(psi + xm + W * y),
                                 __ldg(psi + x + W * rm),  __ldg(psi + xp + W * rp),
                                 __ldg(psi + xm + W * rp), __ldg(psi + xm + W * rm),
                                 __ldg(psi + xp + W * rm)};
            float ex = ux, ey = uy;
            d2q9_sc_shift_native(ps, a.w1, a.w5, dm.G, 1.f / (dm.tau_inv * rho), ex, ey);
            d2q9_bgk_native(g, ex, ey, rho, a.w0, a.w1, a.w5, dm.tau_inv);
            const int o = dm.off + x + W * y;
            if (MOM) { a.rho[o] = rho; a.ux[o] = ux; a.uy[o] = uy; }
#pragma unroll
            for (int k = 0; k < 9; k++) a.dst[k][o] = g[k];
        }
    }
}

// ---------------------------------------------------------------------------
// Single-pass step over tiles of 32 x BY nodes.  A
// block pulls its tile nodes (one per thread) and the ring of nodes around
// them (84 for 32 x 8 tiles), forms psi of all of them in shared memory, and then relaxes
// its tile nodes with the Shan-Chen shift from the shared psi tile.  psi never
// goes through DRAM and a step is one launch: 72 B per node update moved
// (populations read and written once; the ring's pulls are L2 hits of the
// neighbouring tiles) instead of the two passes' 116.  The arithmetic is the
// two-pass path's (same pulls, moments, psi, stencil order, BGK).
// ---------------------------------------------------------------------------
constexpr int ET_BX = 32, ET_PX = ET_BX + 2;  // tile width; psi tile width with its ring

// v modulo n for v in [-n, 2n) (fast) or any v (small domains)
__device__ __forceinline__ int ens_wrap(int v, int n, bool small) {
    if (small) {
        v %= n;
        return v < 0 ? v + n : v;
    }
    return v < 0 ? v + n : (v >= n ? v - n : v);
}

// tiles of ET_BX x BY nodes, one thread per tile node; MINB resident blocks
// per SM bound the registers
template <int BY, int MINB, bool MOM, int PSI>
__global__ void __launch_bounds__(ET_BX * BY, MINB) ens_tile_kernel(const EnsArgs a) {
    constexpr int PY = BY + 2, RING = 2 * ET_PX + 2 * BY;
    // two psi tiles used by alternate items: a block passes one barrier per
    // item (a warp writing tile b for item i + 2 has passed the barrier of
    // item i + 1, which every warp reaches only after its reads of item i)
    __shared__ float sp2[2][PY][ET_PX];
    const int tx = threadIdx.x % ET_BX, ty = threadIdx.x / ET_BX;
    // this thread's ring node, as a position in the psi tile
    int rx = 0, ry = 0;
    {
        const int r = threadIdx.x;
        if (r < ET_PX) { rx = r; ry = 0; }
        else if (r < 2 * ET_PX) { rx = r - ET_PX; ry = PY - 1; }
        else if (r < 2 * ET_PX + BY) { rx = 0; ry = 1 + r - 2 * ET_PX; }
        else { rx = ET_PX - 1; ry = 1 + r - 2 * ET_PX - BY; }
    }
    int it = blockIdx.x;
    if (it >= a.nitems) return;
    EnsItem next = a.items[it];
    for (int b = 0; it < a.nitems; it += gridDim.x, b ^= 1) {
        float (*sp)[ET_PX] = sp2[b];
        const EnsItem dm = next;
        const int nit = it + gridDim.x;
        if (nit < a.nitems) next = a.items[nit];
        const bool small = dm.W < ET_PX || dm.H < PY;
        // the tile node (a wrapped copy where the tile overhangs the domain);
        // the ring node's loads are issued before either density is formed
        const int xt = ens_wrap(dm.x + tx, dm.W, small), yt = ens_wrap(dm.y + ty, dm.H, small);
        const bool ring = threadIdx.x < RING;
        float g[9], g2[9];
        ens_pull(a, dm, xt, yt, g);
        if (ring)
            ens_pull(a, dm, ens_wrap(dm.x - 1 + rx, dm.W, small),
                     ens_wrap(dm.y - 1 + ry, dm.H, small), g2);
        float rho, ux, uy;
        d2q9_moments_native(g, rho, ux, uy);
        sp[ty + 1][tx + 1] = psi_form<PSI>(rho);
        if (ring) {
            sp[ry][rx] = psi_form<PSI>(d2q9_rho_native(g2));
        }
        __syncthreads();
        if (dm.x + tx < dm.W && dm.y + ty < dm.H) {
            // psi(x), psi(x+1,y), psi(x,row+1), psi(x-1,y), psi(x,row-1), then
            // the diagonals: the fused pass's order
            const float ps[9] = {sp[ty + 1][tx + 1], sp[ty + 1][tx + 2], sp[ty + 2][tx + 1],
                                 sp[ty + 1][tx],     sp[ty][tx + 1],     sp[ty + 2][tx + 2],
                                 sp[ty + 2][tx],     sp[ty][tx],         sp[ty][tx + 2]};
            float ex = ux, ey = uy;
            d2q9_sc_shift_native(ps, a.w1, a.w5, dm.G, 1.f / (dm.tau_inv * rho), ex, ey);
            d2q9_bgk_native(g, ex, ey, rho, a.w0, a.w1, a.w5, dm.tau_inv);
            const int o = dm.off + xt + dm.W * yt;
            if (MOM) { a.rho[o] = rho; a.ux[o] = ux; a.uy[o] = uy; }
#pragma unroll
            for (int k = 0; k < 9; k++) a.dst[k][o] = g[k];
        }
    }
}

// ---------------------------------------------------------------------------
// Single pass by warps marching down 32-column strips: no block barrier.  A
// work item is a strip of 32 columns and R rows of one domain, and lane l owns
// column x0 + l (a wrapped copy where the strip overhangs the domain).  For
// each row r the warp pulls row r + 1 and forms its psi (lanes 0 and 31 also
// psi of the columns x0 - 1 and x0 + 32), then relaxes row r with the psi
// stencil of rows r - 1, r, r + 1 from its registers and its neighbour lanes.
// Per node update that is 1 + 2/R + 2/32 pulls instead of the tiles' 1.33.
// Same arithmetic and stencil order as the two-pass step.
// ---------------------------------------------------------------------------
constexpr int ENS_MARCH_THREADS = 256;

// one strip item (march of R rows of 32 columns) by one warp, plain loads
template <int R, bool MOM, int PSI>
__device__ __forceinline__ void ens_march_item(const EnsArgs &a, const EnsItem dm, int lane) {
    constexpr unsigned FULL = 0xffffffffu;
    const bool edge = lane == 0 || lane == 31;
    const bool small = dm.W < ET_PX;
    const int x = ens_wrap(dm.x + lane, dm.W, small);
    const int xh = ens_wrap(lane == 0 ? dm.x - 1 : dm.x + ET_BX, dm.W, small);
    const bool own = dm.x + lane < dm.W;
    const int y_end = min(dm.y + R, dm.H);
    float gc[9], rc, uxc, uyc;  // row r: pulled populations and moments at x
    float pm, pc, hm = 0.f, hc = 0.f;  // psi of rows r - 1, r (h: the halo column)
    {
        float g[9];
        const int ym = ens_wrap(dm.y - 1, dm.H, false);
        ens_pull(a, dm, x, ym, g);
        pm = psi_form<PSI>(d2q9_rho_native(g));
        ens_pull(a, dm, x, dm.y, gc);
        d2q9_moments_native(gc, rc, uxc, uyc);
        pc = psi_form<PSI>(rc);
        if (edge) {
            ens_pull(a, dm, xh, ym, g);
            hm = psi_form<PSI>(d2q9_rho_native(g));
            ens_pull(a, dm, xh, dm.y, g);
            hc = psi_form<PSI>(d2q9_rho_native(g));
        }
    }
    for (int r = dm.y; r < y_end; r++) {
        const int yp = ens_wrap(r + 1, dm.H, false);
        float gn[9], rn, uxn, uyn, hn = 0.f;
        ens_pull(a, dm, x, yp, gn);
        if (edge) {
            float g[9];
            ens_pull(a, dm, xh, yp, g);
            hn = psi_form<PSI>(d2q9_rho_native(g));
        }
        d2q9_moments_native(gn, rn, uxn, uyn);
        const float pn = psi_form<PSI>(rn);
        // x - 1 and x + 1 from the neighbour lanes, the halo at the strip ends
        float lm = __shfl_up_sync(FULL, pm, 1), lc = __shfl_up_sync(FULL, pc, 1);
        float ln = __shfl_up_sync(FULL, pn, 1);
        float qm = __shfl_down_sync(FULL, pm, 1), qc = __shfl_down_sync(FULL, pc, 1);
        float qn = __shfl_down_sync(FULL, pn, 1);
        if (lane == 0) { lm = hm; lc = hc; ln = hn; }
        if (lane == 31) { qm = hm; qc = hc; qn = hn; }
        if (own) {
            // the fused pass's order: psi(x), psi(x+1,y), psi(x,row+1),
            // psi(x-1,y), psi(x,row-1), then the diagonals
            const float ps[9] = {pc, qc, pn, lc, pm, qn, ln, lm, qm};
            float ex = uxc, ey = uyc;
            d2q9_sc_shift_native(ps, a.w1, a.w5, dm.G, 1.f / (dm.tau_inv * rc), ex, ey);
            d2q9_bgk_native(gc, ex, ey, rc, a.w0, a.w1, a.w5, dm.tau_inv);
            const int o = dm.off + x + dm.W * r;
            if (MOM) { a.rho[o] = rc; a.ux[o] = uxc; a.uy[o] = uyc; }
#pragma unroll
            for (int k = 0; k < 9; k++) a.dst[k][o] = gc[k];
        }
#pragma unroll
        for (int k = 0; k < 9; k++) gc[k] = gn[k];
        rc = rn; uxc = uxn; uyc = uyn;
        pm = pc; pc = pn; hm = hc; hc = hn;
    }
}

template <int R, int MINB, bool MOM, int PSI>
__global__ void __launch_bounds__(ENS_MARCH_THREADS, MINB) ens_march_kernel(const EnsArgs a) {
    const int lane = threadIdx.x & 31;
    const int warps_per_block = ENS_MARCH_THREADS / 32;
    const int nwarps = gridDim.x * warps_per_block;
    for (int it = blockIdx.x * warps_per_block + (threadIdx.x >> 5); it < a.nitems;
         it += nwarps)
        ens_march_item<R, MOM, PSI>(a, a.items[it], lane);
}

// ---------------------------------------------------------------------------
// Strips of column pairs, one or two steps per launch.  A warp marches down a
// strip of 64 columns, two per lane, both through the paired FP32 instructions
// (lb_pairs.cuh; every lane the scalar operations in the scalar order, so the
// same bits).  Input rows arrive in a ring of four per warp by 16-byte cp.async,
// three rows ahead.  Per step, a lane keeps the populations that the rows below
// will pull, already moved along x (one shuffle per population and row), the
// pulled populations of the row it relaxes next, and psi of that row and the
// one above with its neighbours' values (two shuffles per row): when input row
// i has arrived, row i - 1 is pulled and its psi formed, and row i - 2 relaxed;
// with two steps the relaxed row goes into a second such level at once and row
// i - 4 goes to memory.  A step loses two columns on each side and two rows at
// each end of an item: 56 of 64 columns are stored, and 4 (8) rows read beyond
// an item's own.  Rows that do not start on 16 bytes are copied and stored per
// node.  One warp per block: blocks refill as items end.
//
// Measured (GLUPS; in brackets the strips of 32 columns whose source rows
// came through a per-warp shared-memory ring, one node per lane, which these
// replace): 512 droplet domains of 64..512
// 101 with two steps, 81 with one (72); 64 domains 88, 77 (66); 24 domains of
// 64..128 31, 30 (9: one item per warp of an eight-warp block left most SMs
// empty).  About 180 issue slots per 64 node updates, 347 per 32 for the row
// ring.  Two steps move 40 B per node update and are bound by the latency of
// their arithmetic chain at 12 warps per SM (168 registers, 56 bytes of them
// spilled), one step by memory and the chain at 16 (128 registers).
// ---------------------------------------------------------------------------
constexpr int EP_EDGE = 4, EP_COLS = 64 - 2 * EP_EDGE;
constexpr int EP_RING = 4;
constexpr int EP_ROW = 9 * 32;  // column pairs of a row's nine populations
// resident blocks (warps) per SM by steps per launch
constexpr int ep_blocks(int steps) { return steps == 1 ? 16 : 12; }

struct EnsPairArgs {
    EnsArgs a;
    int rows;  // rows of an item
    PairConst c;
};

template <int BYTES> __device__ __forceinline__ void ep_copy(void *dst, const void *src) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(dst)),
                     "l"(src)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(dst)),
                     "l"(src)
                     : "memory");
}

template <int STEPS, bool MOM>
__global__ void __launch_bounds__(32, ep_blocks(STEPS))
    ens_pair_kernel(const __grid_constant__ EnsPairArgs pa) {
    const EnsArgs &a = pa.a;
    const PairConst &c = pa.c;
    extern __shared__ __align__(16) float2 ep_smem[];
    const int lane = threadIdx.x;
    const EnsItem dm = a.items[blockIdx.x];
    const int W = dm.W, H = dm.H;
    const int nr = min(pa.rows, H - dm.y);
    const bool vec = ((W | dm.off) & 3) == 0;  // rows and tiles start on 16 bytes
    const int ns = (W + EP_COLS - 1) / EP_COLS, tw = ((W + ns - 1) / ns + 3) & ~3;
    const int nw = min(tw, W - dm.x);
    const int xs = dm.x - EP_EDGE + 2 * lane;
    int xa = xs % W;
    xa += xa < 0 ? W : 0;
    const int xb = xa == W - 1 ? 0 : xa + 1;
    const bool own_a = xs >= dm.x && xs < dm.x + nw, own_b = xs + 1 >= dm.x && xs + 1 < dm.x + nw;
    float2 *const ring = ep_smem + lane;
    const int last = nr + 4 * STEPS;
    int y = (dm.y - 2 * STEPS) % H;
    y += y < 0 ? H : 0;
    const float *cs[5];
#pragma unroll
    for (int j = 0; j < 5; j++) {
        const int ch = min(lane + 32 * j, 143), k = ch >> 4;
        cs[j] = a.src[0];
#pragma unroll
        for (int m = 1; m < 9; m++)
            if (k == m) cs[j] = a.src[m];
        int x = (dm.x - EP_EDGE + 4 * (ch & 15)) % W;
        cs[j] += dm.off + (x < 0 ? x + W : x);
    }
    auto copy = [&](int i, int slot) {
        if (i < last) {
            float2 *const d = ring + slot * EP_ROW;
            const uint32_t o = (uint32_t)y * (uint32_t)W;
            if (vec) {
#pragma unroll
                for (int j = 0; j < 5; j++)
                    if (lane + 32 * j < 144) ep_copy<16>(d - lane + 2 * (lane + 32 * j), cs[j] + o);
            } else {
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    ep_copy<4>(&d[k * 32].x, a.src[k] + dm.off + (o + xa));
                    ep_copy<4>(&d[k * 32].y, a.src[k] + dm.off + (o + xb));
                }
            }
            y = y == H - 1 ? 0 : y + 1;
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    PairD2 d;
    d.n0 = both(-a.w0); d.n1 = both(-a.w1); d.n5 = both(-a.w5);
    d.mt = both(-dm.tau_inv);
    const float2 tau = both(dm.tau_inv), mG = both(-dm.G), w1 = both(a.w1), w5 = both(a.w5);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
    for (int j = 0; j < EP_RING - 1; j++) copy(j, j);
    // per level: populations 4, 7, 8 of the last row (p) and the one before it
    // (q) and 0, 1, 3 of the last row (b), moved along x; the pulled populations
    // and moments of the row that is relaxed next; psi (left, centre, right) of
    // that row (s0) and of the one above it (sm)
    float2 p[STEPS][3], q[STEPS][3], b[STEPS][3], G[STEPS][9], rho[STEPS], ux[STEPS], uy[STEPS];
    float2 s0[STEPS][3], sm[STEPS][3];
#pragma unroll
    for (int t = 0; t < STEPS; t++) {
#pragma unroll
        for (int j = 0; j < 3; j++)
            p[t][j] = q[t][j] = b[t][j] = s0[t][j] = sm[t][j] = both(1.f);
#pragma unroll
        for (int k = 0; k < 9; k++) G[t][k] = both(1.f);
        rho[t] = ux[t] = uy[t] = both(1.f);
    }
    int slot = 0, next = EP_RING - 1;
#pragma unroll 1
    for (int i = 0; i < last; i++) {
        __syncwarp();
        copy(i + EP_RING - 1, next);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(EP_RING - 1) : "memory");
        __syncwarp();
        const float2 *const row = ring + slot * EP_ROW;
        float2 n[9];
#pragma unroll
        for (int k = 0; k < 9; k++) n[k] = row[k * 32];
        next = slot;
        slot = slot == EP_RING - 1 ? 0 : slot + 1;
#pragma unroll
        for (int t = 0; t < STEPS; t++) {
            // n: row j of the level below; pull row j - 1, relax row j - 2
            float2 g[9];
            g[0] = b[t][0]; g[1] = b[t][1]; g[3] = b[t][2];
            g[4] = q[t][0]; g[7] = q[t][1]; g[8] = q[t][2];
            g[2] = n[2];
            g[5] = row_shift(n[5], d2_cx(5));
            g[6] = row_shift(n[6], d2_cx(6));
            b[t][0] = n[0];
            b[t][1] = row_shift(n[1], d2_cx(1));
            b[t][2] = row_shift(n[3], d2_cx(3));
#pragma unroll
            for (int j = 0; j < 3; j++) q[t][j] = p[t][j];
            p[t][0] = n[4];
            p[t][1] = row_shift(n[7], d2_cx(7));
            p[t][2] = row_shift(n[8], d2_cx(8));
            float2 r1, u1, v1;
            d2q9_moments_pairs(c, g, r1, u1, v1);
            const float2 ps = a.psi_form == 0 ? make_float2(psi_ref(r1.x), psi_ref(r1.y))
                                              : pair_psi_exp1(c, r1);
            const float2 sp[3] = {row_shift(ps, 1), ps, row_shift(ps, -1)};
            // relax row j - 2: psi of the row above sm, its own s0, below sp
            const float2 irt = pair_rcp(c, __fmul2_rn(tau, rho[t]));
            const float2 ix = __ffma2_rn(
                w1, pair_sub(c, s0[t][2], s0[t][0]),
                __fmul2_rn(w5, pair_sub(c, pair_add(sp[2], sm[t][2]), pair_add(sp[0], sm[t][0]))));
            const float2 iy = __ffma2_rn(
                w1, pair_sub(c, sm[t][1], sp[1]),
                __fmul2_rn(w5, pair_sub(c, pair_add(sm[t][0], sm[t][2]), pair_add(sp[2], sp[0]))));
            const float2 cc = __fmul2_rn(__fmul2_rn(mG, s0[t][1]), irt);
            const float2 ex = __ffma2_rn(cc, ix, ux[t]), ey = __ffma2_rn(cc, iy, uy[t]);
            d2q9_bgk_pairs(c, d, G[t], ex, ey, rho[t]);
            if (t < STEPS - 1) {
#pragma unroll
                for (int k = 0; k < 9; k++) n[k] = G[t][k];
            } else if (i >= 4 * STEPS) {
                const uint32_t o = (uint32_t)dm.off + (uint32_t)(dm.y + i - 4 * STEPS) * (uint32_t)W;
                if (MOM) {
                    if (own_a) { a.rho[o + xa] = rho[t].x; a.ux[o + xa] = ux[t].x; a.uy[o + xa] = uy[t].x; }
                    if (own_b) { a.rho[o + xb] = rho[t].y; a.ux[o + xb] = ux[t].y; a.uy[o + xb] = uy[t].y; }
                }
                if (vec && own_a && own_b) {
#pragma unroll
                    for (int k = 0; k < 9; k++)
                        *reinterpret_cast<float2 *>(a.dst[k] + (o + xa)) = G[t][k];
                } else {
                    if (own_a) {
#pragma unroll
                        for (int k = 0; k < 9; k++) a.dst[k][o + xa] = G[t][k].x;
                    }
                    if (own_b) {
#pragma unroll
                        for (int k = 0; k < 9; k++) a.dst[k][o + xb] = G[t][k].y;
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 9; k++) G[t][k] = g[k];
            rho[t] = r1; ux[t] = u1; uy[t] = v1;
#pragma unroll
            for (int j = 0; j < 3; j++) { sm[t][j] = s0[t][j]; s0[t][j] = sp[j]; }
        }
    }
}

// march shapes: rows per item and the register bound (resident blocks per SM)
#define LB_ENS_MARCH(X) \
    X(6, 32, 3)         \
    X(7, 32, 4)         \
    X(8, 64, 3)         \
    X(9, 16, 3)

int ens_march_rows(int shape) {
    switch (shape) {
#define LB_ENS_MROWS(S, R, MINB) \
    case S: return R;
        LB_ENS_MARCH(LB_ENS_MROWS)
#undef LB_ENS_MROWS
        default: return 0;
    }
}

// tile shapes: rows per tile and the register bound (resident blocks per SM)
#define LB_ENS_TILES(X) \
    X(1, 8, 5)          \
    X(2, 8, 6)          \
    X(3, 16, 2)         \
    X(4, 16, 3)         \
    X(5, 32, 1)

int ens_tile_rows(int shape) {
    switch (shape) {
#define LB_ENS_ROWS(S, BY, MINB) \
    case S: return BY;
        LB_ENS_TILES(LB_ENS_ROWS)
#undef LB_ENS_ROWS
        default: return 0;
    }
}

struct LaunchShape {
    int bx, ry, bps;  // threads along x, rows per work item (= blockDim.y), blocks per SM;
                      // bx = 0: the single-pass form ry
};

// forms 10 to 12: the column-pair strips, by rows of an item (0: the library's
// choice, and its choice of one or two steps per launch)
bool ens_pairs(const LaunchShape &s) { return s.bx == 0 && s.ry >= 10 && s.ry <= 12; }
int ens_pair_form_rows(int form) { return form == 11 ? 64 : form == 12 ? 16 : 0; }
int ens_pair_tile(int W) {
    const int ns = (W + EP_COLS - 1) / EP_COLS;
    return ((W + ns - 1) / ns + 3) & ~3;
}

}  // namespace

// Form 10 takes two steps per launch from this many nodes on if most of them lie in
// domains whose rows start on 16 bytes (400 domains of 97, 101 and 130 columns: 39
// GLUPS with two, 52 with one).  Time of two over one on such ensembles: 512 domains
// of 32..512 0.80, 64 of them 0.86, 255 of 64^2 (1.04 M nodes) 1.00; below the line it
// depends on how the items fill the warps: 60 of 128^2 0.92, 10 of 256^2 (0.66 M) 0.79,
// 128 of 64^2 0.99, but 6 of 256^2 (0.39 M) 1.21, 64 of 64^2 1.20, 2048 of 16^2 1.17, 16
// of 128^2 0.97; over 37 ensembles of up to 0.98 M nodes 0.78 .. 1.21.
constexpr long ENS_TWO_STEP_MIN_NODES = 1L << 20;

struct lb_ensemble {
    int nd = 0;
    std::vector<EnsDomain> dom;
    long NT = 0, stride = 0;
    float *pop[2] = {nullptr, nullptr};
    float *psi = nullptr, *mom = nullptr;
    EnsItem *items_d = nullptr;
    int nitems = 0, items_cap = 0;
    bool two_steps = false;  // form 10 advances two steps per launch
    int pair_rows = 0;       // column-pair strips: rows of an item
    int cur = 0, psi_form = LB_PSI_EXP1, sms = 1, graph_steps = 32;
    LaunchShape shape{0, 10, 12};  // strips of column pairs (or form 6: ens_strips_pay)
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaGraphExec_t graph[2] = {nullptr, nullptr};
    int64_t launches = 0;
    std::string err;
};

namespace {

int efail(lb_ensemble *e, int code, const std::string &m) {
    if (e) e->err = m;
    return code;
}
#define LB_ETRY(e, where, call)                                                      \
    do {                                                                             \
        cudaError_t c_ = (call);                                                     \
        if (c_ != cudaSuccess)                                                       \
            return efail(e, LB_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(c_)); \
    } while (0)

const float W2F[3] = {(float)(4.0 / 9.0), (float)(1.0 / 9.0), (float)(1.0 / 36.0)};

float *pk(lb_ensemble *e, int set, int k) { return e->pop[set] + (long)k * e->stride; }

EnsArgs args_for(lb_ensemble *e, int from) {
    EnsArgs a{};
    for (int k = 0; k < 9; k++) {
        a.src[k] = pk(e, from, k);
        a.dst[k] = pk(e, 1 - from, k);
    }
    a.psi = e->psi;
    a.rho = e->mom; a.ux = e->mom + e->stride; a.uy = e->mom + 2 * e->stride;
    a.items = e->items_d;
    a.nitems = e->nitems;
    a.psi_form = e->psi_form;
    a.w0 = W2F[0]; a.w1 = W2F[1]; a.w5 = W2F[2];
    return a;
}

int launches_per_step(const lb_ensemble *e) {
    if (e->shape.bx != 0) return 2;
    return 1;
}

// column-pair strips: `steps` (1 or 2) steps in one launch, a programmatic
// dependent of the launch before it
cudaError_t ens_pair_launch(lb_ensemble *e, int from, int steps, bool mom) {
    EnsPairArgs pa{};
    pa.a = args_for(e, from);
    pa.rows = e->pair_rows;
    pa.c = pair_constants();
    e->launches += 1;
    const auto kernel = steps == 1 ? (mom ? ens_pair_kernel<1, true> : ens_pair_kernel<1, false>)
                                   : (mom ? ens_pair_kernel<2, true> : ens_pair_kernel<2, false>);
    return launch_dependent_smem(kernel, dim3(e->nitems), dim3(32),
                                 EP_RING * EP_ROW * sizeof(float2), e->stream, pa);
}

// one step (any form)
cudaError_t ens_step(lb_ensemble *e, int from, bool mom) {
    if (ens_pairs(e->shape)) return ens_pair_launch(e, from, 1, mom);
    const EnsArgs a = args_for(e, from);
    const bool ref = e->psi_form == LB_PSI_REF;
    const unsigned grid = (unsigned)std::max(1, std::min(e->nitems, e->sms * e->shape.bps));
    if (e->shape.bx == 0) {
        switch (e->shape.ry) {
#define LB_ENS_LAUNCH(S, BY, MINB)                                                             \
    case S:                                                                                    \
        (ref ? mom ? ens_tile_kernel<BY, MINB, true, LB_PSI_REF>                               \
                   : ens_tile_kernel<BY, MINB, false, LB_PSI_REF>                              \
             : mom ? ens_tile_kernel<BY, MINB, true, LB_PSI_EXP1>                              \
                   : ens_tile_kernel<BY, MINB, false, LB_PSI_EXP1>)                            \
            <<<grid, ET_BX * BY, 0, e->stream>>>(a);                                           \
        break;
            LB_ENS_TILES(LB_ENS_LAUNCH)
#undef LB_ENS_LAUNCH
#define LB_ENS_MLAUNCH(S, R, MINB)                                                             \
    case S:                                                                                    \
        (ref ? mom ? ens_march_kernel<R, MINB, true, LB_PSI_REF>                               \
                   : ens_march_kernel<R, MINB, false, LB_PSI_REF>                              \
             : mom ? ens_march_kernel<R, MINB, true, LB_PSI_EXP1>                              \
                   : ens_march_kernel<R, MINB, false, LB_PSI_EXP1>)                            \
            <<<grid, ENS_MARCH_THREADS, 0, e->stream>>>(a);                                    \
        break;
            LB_ENS_MARCH(LB_ENS_MLAUNCH)
#undef LB_ENS_MLAUNCH
            default: return cudaErrorInvalidValue;
        }
        e->launches += 1;
        return cudaGetLastError();
    }
    const dim3 block(e->shape.bx, e->shape.ry);
    if (ref) ens_density_kernel<LB_PSI_REF><<<grid, block, 0, e->stream>>>(a);
    else ens_density_kernel<LB_PSI_EXP1><<<grid, block, 0, e->stream>>>(a);
    cudaError_t c = cudaGetLastError();
    if (c != cudaSuccess) return c;
    if (mom) ens_fused_kernel<true><<<grid, block, 0, e->stream>>>(a);
    else ens_fused_kernel<false><<<grid, block, 0, e->stream>>>(a);
    e->launches += 2;
    return cudaGetLastError();
}

void drop_graphs(lb_ensemble *e) {
    for (int i = 0; i < 2; i++)
        if (e->graph[i]) {
            cudaGraphExecDestroy(e->graph[i]);
            e->graph[i] = nullptr;
        }
}

// steps per launch of the current form, and such a launch
int ens_steps_per_launch(const lb_ensemble *e) {
    return e->shape.bx == 0 && e->shape.ry == 10 && e->two_steps ? 2 : 1;
}
cudaError_t ens_launch(lb_ensemble *e, int from, bool mom) {
    const int s = ens_steps_per_launch(e);
    return s > 1 ? ens_pair_launch(e, from, s, mom) : ens_step(e, from, mom);
}

// Column-pair strips: rows per item.  Fewer rows fill the GPU's warps, more rows
// pay less for the 4 (8) rows an item reads beyond its own.  A pass takes an
// item's march times a function of the rounds of items w that was fitted to 64
// domains and two steps (us per step): 16 rows 89.7, 24 89.0, 32 88.3, 48 87.0,
// 64 103 (w = 1.13: a nearly empty second round), 96 94.9 (w = 0.75).
int ens_pick_rows(const lb_ensemble *e) {
    const int steps = ens_steps_per_launch(e);
    const double warps = (double)e->sms * ep_blocks(steps);
    int pick = 8;
    double best = 0;
    for (int r : {8, 12, 16, 24, 32, 48, 64, 96, 128}) {
        long items = 0;
        for (const EnsDomain &m : e->dom) {
            const int tw = ens_pair_tile(m.W);
            items += (long)((m.W + tw - 1) / tw) * ((m.H + r - 1) / r);
        }
        const double w = items / warps;
        const double cost = (r + 4. * steps) * (w <= 1. ? 0.65 + 0.35 * w : std::max(1.42, 0.32 + 0.82 * w));
        if (best == 0 || cost < best) {
            best = cost;
            pick = r;
        }
    }
    return pick;
}

// Whether the strips of 32 columns (form 6) are the default: on many narrow domains
// most of a 64-column strip lies idle, and rows that do not start on 16 bytes are
// copied node by node.  us per step, column pairs / strips: 65 625 domains of 8^2 352 /
// 249, 16 384 of 16^2 140 / 126, 42 000 of 10^2 393 / 194, 5 242 of 10^2 55 / 30, 12 962
// of 18^2 157 / 114; but 512 of 16^2 9.5 / 15, 5 357 of 28^2 76 / 91, 1 310 of 20^2 both
// 25.  The two times are estimated as an item's march times us per row (a warp's row
// of pairs; dearer where it is copied by node) times a function of the rounds of items
// w; over 98 ensembles of 2^2 .. 56^2 domains (4 000 .. 4.2 M nodes) the estimates'
// choice lost at most 9 % to the other form, but for one of 24 %.
struct EnsEstimate {
    double items = 0, sum = 0;  // items; their marches in us
    void add(int count, int rows, double us_per_row) {
        items += count;
        sum += count * (double)rows * us_per_row;
    }
};
bool ens_strips_pay(const lb_ensemble *e) {
    const int steps = e->two_steps ? 2 : 1, r = ens_pick_rows(e), R = ens_march_rows(6);
    EnsEstimate pairs, strips;
    for (const EnsDomain &m : e->dom) {
        const int tw = ens_pair_tile(m.W), k = (m.H + r - 1) / r, n = (m.H + R - 1) / R;
        const double row = ((m.W | m.off) & 3) == 0 ? (steps == 1 ? 1.2 : 1.5)
                                                    : (1.1 + 8. / std::min(m.W, tw)) *
                                                          (steps == 1 ? 1. : 1.25);
        pairs.add((m.W + tw - 1) / tw * k, (m.H + k - 1) / k + 4 * steps, row);
        strips.add((m.W + ET_BX - 1) / ET_BX * n, (m.H + n - 1) / n + 2, 1.7);
    }
    const double wp = pairs.items / ((double)e->sms * ep_blocks(steps));
    const double ws = strips.items / (e->sms * 3. * (ENS_MARCH_THREADS / 32));
    const double fp = wp <= 1. ? std::min(1., 0.2 + 1.1 * wp) : std::max(1.42, 0.32 + 0.82 * wp);
    const double fs = ws <= 1. ? 0.5 + 0.5 * ws : 0.32 + 0.82 * ws;
    return strips.sum / strips.items * fs < 0.95 * pairs.sum / pairs.items * fp / steps;
}

// work list of row groups for the current shape
int build_items(lb_ensemble *e) {
    std::vector<EnsItem> items;
    const bool pairs = ens_pairs(e->shape);
    if (pairs) {
        const int r = ens_pair_form_rows(e->shape.ry);
        e->pair_rows = r ? r : ens_pick_rows(e);
    }
    for (int d = 0; d < e->nd; d++) {
        const EnsDomain &m = e->dom[d];
        if (pairs) {
            const int tw = ens_pair_tile(m.W);
            for (int y = 0; y < m.H; y += e->pair_rows)
                for (int x = 0; x < m.W; x += tw)
                    items.push_back(EnsItem{m.off, m.W, m.H, y, m.G, m.tau_inv, x});
        } else if (e->shape.bx == 0) {  // tiles or strips, row by row
            const int rows = ens_tile_rows(e->shape.ry) + ens_march_rows(e->shape.ry);
            for (int y = 0; y < m.H; y += rows)
                for (int x = 0; x < m.W; x += ET_BX)
                    items.push_back(EnsItem{m.off, m.W, m.H, y, m.G, m.tau_inv, x});
        } else {  // groups of ry rows
            for (int y = 0; y < m.H; y += e->shape.ry)
                items.push_back(EnsItem{m.off, m.W, m.H, y, m.G, m.tau_inv, 0});
        }
    }
    if ((int)items.size() > e->items_cap) {
        if (e->items_d) cudaFree(e->items_d);
        e->items_d = nullptr;
        LB_ETRY(e, "work list", cudaMalloc(&e->items_d, sizeof(EnsItem) * items.size()));
        e->items_cap = (int)items.size();
    }
    // in the steps' stream: a plain copy from pageable memory may return before its
    // last bytes have arrived, and a stream that does not block would not wait for them
    LB_ETRY(e, "work list", cudaMemcpyAsync(e->items_d, items.data(), sizeof(EnsItem) * items.size(),
                                            cudaMemcpyHostToDevice, e->stream));
    LB_ETRY(e, "work list", cudaStreamSynchronize(e->stream));
    e->nitems = (int)items.size();
    drop_graphs(e);
    return LB_OK;
}

int egraph(lb_ensemble *e, int from, cudaGraphExec_t *out) {
    if (e->graph[from]) { *out = e->graph[from]; return LB_OK; }
    const int64_t before = e->launches;
    LB_ETRY(e, "capture", cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t c = cudaSuccess;
    int set = from;
    const int launches = e->graph_steps / ens_steps_per_launch(e);  // even: back to `from`
    for (int i = 0; i < launches && c == cudaSuccess; i++) {
        c = ens_launch(e, set, false);
        set = 1 - set;
    }
    cudaGraph_t g;
    cudaError_t c2 = cudaStreamEndCapture(e->stream, &g);
    e->launches = before;
    LB_ETRY(e, "capture", c);
    LB_ETRY(e, "capture", c2);
    c = cudaGraphInstantiate(&e->graph[from], g, 0);
    cudaGraphDestroy(g);
    LB_ETRY(e, "cudaGraphInstantiate", c);
    *out = e->graph[from];
    return LB_OK;
}

}  // namespace

extern "C" {

int lb_ensemble_create(int nd, const int *nx, const int *ny, const float *G, const float *tau_inv,
                       int psi_form, lb_ensemble **out) {
    if (!out || nd < 1 || !nx || !ny || !G || !tau_inv) return LB_ERR_ARG;
    *out = nullptr;
    if (psi_form != LB_PSI_REF && psi_form != LB_PSI_EXP1) return LB_ERR_ARG;
    lb_ensemble *e = new lb_ensemble;
    e->nd = nd;
    e->psi_form = psi_form;
    long off = 0;
    for (int d = 0; d < nd; d++) {
        if (nx[d] < 1 || ny[d] < 1) { delete e; return LB_ERR_ARG; }
        e->dom.push_back(EnsDomain{nx[d], ny[d], (int)off, G[d], tau_inv[d]});
        off += (long)nx[d] * ny[d];
        if (off > (1L << 31) - 256) { delete e; return LB_ERR_ARG; }
    }
    e->NT = off;
    e->stride = (off + 127) / 128 * 128;
    long aligned = 0;
    for (const EnsDomain &m : e->dom)
        if (((m.W | m.off) & 3) == 0) aligned += (long)m.W * m.H;
    e->two_steps = off >= ENS_TWO_STEP_MIN_NODES && 2 * aligned >= off;
    int dev = 0;
    cudaError_t c = cudaGetDevice(&dev);
    if (c == cudaSuccess) c = cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, dev);
    if (c == cudaSuccess) c = cudaMalloc(&e->pop[0], sizeof(float) * 9 * e->stride);
    if (c == cudaSuccess) c = cudaMalloc(&e->pop[1], sizeof(float) * 9 * e->stride);
    if (c == cudaSuccess) c = cudaMalloc(&e->psi, sizeof(float) * e->stride);
    if (c == cudaSuccess) c = cudaMalloc(&e->mom, sizeof(float) * 3 * e->stride);
    if (c == cudaSuccess) c = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking);
    if (c == cudaSuccess) c = cudaMemsetAsync(e->mom, 0, sizeof(float) * 3 * e->stride, e->stream);
    if (c == cudaSuccess) c = cudaEventCreate(&e->ev0);
    if (c == cudaSuccess) c = cudaEventCreate(&e->ev1);
    if (c != cudaSuccess) {
        lb_ensemble_destroy(e);
        return c == cudaErrorMemoryAllocation ? LB_ERR_NOMEM : LB_ERR_CUDA;
    }
    if (ens_strips_pay(e)) e->shape = LaunchShape{0, 6, 6};
    if (build_items(e) != LB_OK) {
        lb_ensemble_destroy(e);
        return LB_ERR_CUDA;
    }
    // at rest at density 1 until the caller sets a state: the autotuner, which
    // runs before that, would otherwise time the steps on whatever the memory
    // holds (divisions by zero, not numbers)
    Pop<9> p;
    for (int k = 0; k < 9; k++) p.f[k] = pk(e, e->cur, k);
    c = launch_d2q9_equilibrium(p, nullptr, nullptr, nullptr, (int)e->NT, W2F[0], W2F[1], W2F[2],
                                e->stream);
    if (c == cudaSuccess) c = cudaStreamSynchronize(e->stream);
    if (c != cudaSuccess) {
        lb_ensemble_destroy(e);
        return LB_ERR_CUDA;
    }
    *out = e;
    return LB_OK;
}

int lb_ensemble_destroy(lb_ensemble *e) {
    if (!e) return LB_ERR_ARG;
    if (e->stream) cudaStreamSynchronize(e->stream);
    drop_graphs(e);
    for (int i = 0; i < 2; i++)
        if (e->pop[i]) cudaFree(e->pop[i]);
    if (e->psi) cudaFree(e->psi);
    if (e->mom) cudaFree(e->mom);
    if (e->items_d) cudaFree(e->items_d);
    if (e->ev0) cudaEventDestroy(e->ev0);
    if (e->ev1) cudaEventDestroy(e->ev1);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
    return LB_OK;
}

const char *lb_ensemble_error(const lb_ensemble *e) { return e ? e->err.c_str() : "null ensemble"; }
long lb_ensemble_nodes(const lb_ensemble *e) { return e ? e->NT : -1; }
long lb_ensemble_offset(const lb_ensemble *e, int d) {
    return (e && d >= 0 && d < e->nd) ? e->dom[d].off : -1;
}
int64_t lb_ensemble_launch_count(const lb_ensemble *e) { return e ? e->launches : -1; }

int lb_ensemble_set_populations(lb_ensemble *e, const float *f) {
    if (!e || !f) return LB_ERR_ARG;
    for (int k = 0; k < 9; k++)
        LB_ETRY(e, "lb_ensemble_set_populations",
                cudaMemcpyAsync(pk(e, e->cur, k), f + (long)k * e->NT, sizeof(float) * e->NT,
                                cudaMemcpyHostToDevice, e->stream));
    LB_ETRY(e, "lb_ensemble_set_populations", cudaStreamSynchronize(e->stream));
    return LB_OK;
}

int lb_ensemble_get_populations(lb_ensemble *e, float *f) {
    if (!e || !f) return LB_ERR_ARG;
    for (int k = 0; k < 9; k++)
        LB_ETRY(e, "lb_ensemble_get_populations",
                cudaMemcpyAsync(f + (long)k * e->NT, pk(e, e->cur, k), sizeof(float) * e->NT,
                                cudaMemcpyDeviceToHost, e->stream));
    LB_ETRY(e, "lb_ensemble_get_populations", cudaStreamSynchronize(e->stream));
    return LB_OK;
}

int lb_ensemble_init_equilibrium(lb_ensemble *e, const float *rho) {
    if (!e || !rho) return LB_ERR_ARG;
    LB_ETRY(e, "lb_ensemble_init_equilibrium",
            cudaMemcpyAsync(e->mom, rho, sizeof(float) * e->NT, cudaMemcpyHostToDevice, e->stream));
    Pop<9> p;
    for (int k = 0; k < 9; k++) p.f[k] = pk(e, e->cur, k);
    LB_ETRY(e, "lb_ensemble_init_equilibrium",
            launch_d2q9_equilibrium(p, e->mom, nullptr, nullptr, (int)e->NT, W2F[0], W2F[1],
                                    W2F[2], e->stream));
    e->launches += 1;
    LB_ETRY(e, "lb_ensemble_init_equilibrium", cudaStreamSynchronize(e->stream));
    return LB_OK;
}

int lb_ensemble_step(lb_ensemble *e, int nsteps) {
    if (!e || nsteps < 0) return LB_ERR_ARG;
    if (nsteps == 0) return LB_OK;
    const int per = ens_steps_per_launch(e);
    int rest = nsteps;
    for (; rest % per; rest--) {  // single steps first: the last launch writes the moments
        LB_ETRY(e, "lb_ensemble_step", ens_step(e, e->cur, rest == 1));
        e->cur = 1 - e->cur;
    }
    while (rest > e->graph_steps) {
        cudaGraphExec_t g;
        const int rc = egraph(e, e->cur, &g);
        if (rc != LB_OK) return rc;
        LB_ETRY(e, "cudaGraphLaunch", cudaGraphLaunch(g, e->stream));
        e->launches += (int64_t)launches_per_step(e) * (e->graph_steps / per);
        rest -= e->graph_steps;
    }
    for (; rest > 0; rest -= per) {
        LB_ETRY(e, "lb_ensemble_step", ens_launch(e, e->cur, rest == per));
        e->cur = 1 - e->cur;
    }
    return LB_OK;
}

int lb_ensemble_time_steps(lb_ensemble *e, int nsteps, float *ms) {
    if (!e || !ms) return LB_ERR_ARG;
    LB_ETRY(e, "lb_ensemble_time_steps", cudaEventRecord(e->ev0, e->stream));
    const int rc = lb_ensemble_step(e, nsteps);
    if (rc != LB_OK) return rc;
    LB_ETRY(e, "lb_ensemble_time_steps", cudaEventRecord(e->ev1, e->stream));
    LB_ETRY(e, "lb_ensemble_time_steps", cudaEventSynchronize(e->ev1));
    LB_ETRY(e, "lb_ensemble_time_steps", cudaEventElapsedTime(ms, e->ev0, e->ev1));
    return LB_OK;
}

int lb_ensemble_get_moments(lb_ensemble *e, float *rho, float *ux, float *uy) {
    if (!e) return LB_ERR_ARG;
    float *dst[3] = {rho, ux, uy};
    for (int i = 0; i < 3; i++)
        if (dst[i])
            LB_ETRY(e, "lb_ensemble_get_moments",
                    cudaMemcpyAsync(dst[i], e->mom + (long)i * e->stride, sizeof(float) * e->NT,
                                    cudaMemcpyDeviceToHost, e->stream));
    LB_ETRY(e, "lb_ensemble_get_moments", cudaStreamSynchronize(e->stream));
    return LB_OK;
}

int lb_ensemble_set_launch(lb_ensemble *e, int threads_x, int rows, int blocks_per_sm) {
    const bool tiles = threads_x == 0;
    if (!e || blocks_per_sm < 1 || blocks_per_sm > 32 ||
        (tiles && ens_tile_rows(rows) + ens_march_rows(rows) == 0 &&
         !ens_pairs(LaunchShape{0, rows, 1})) ||
        (!tiles && (threads_x < 32 || threads_x % 32 || rows < 1 || threads_x * rows > 1024)))
        return LB_ERR_ARG;
    LB_ETRY(e, "lb_ensemble_set_launch", cudaStreamSynchronize(e->stream));
    e->shape = LaunchShape{threads_x, rows, blocks_per_sm};
    return build_items(e);
}

int lb_ensemble_get_launch(const lb_ensemble *e, int out[3]) {
    if (!e || !out) return LB_ERR_ARG;
    out[0] = e->shape.bx; out[1] = e->shape.ry; out[2] = e->shape.bps;
    return LB_OK;
}

// Times every candidate shape for trial_steps steps (after one untimed step)
// on the ensemble's current state and keeps the fastest.  The state advances by
// (trial_steps + 1) steps per candidate, by up to two more where a launch is two
// steps: tune before setting the initial state.
int lb_ensemble_autotune(lb_ensemble *e, int trial_steps, int out[3]) {
    if (!e || trial_steps < 1) return LB_ERR_ARG;
    // the single-pass tiles, then the two-pass row groups {64, 128, 256
    // threads} x {1, 2, 4 rows} x {2, 4, 8 blocks}
    static const int BX[3] = {64, 128, 256}, RY[3] = {1, 2, 4}, BPS[3] = {2, 4, 8};
    // (tile or strip shape, blocks per SM): each shape at its register-bound
    // residency and at twice it
    static const int TILES[][2] = {{1, 5}, {1, 10}, {2, 6}, {2, 12}, {3, 2}, {3, 4}, {4, 3},
                                   {5, 1}, {6, 3}, {6, 6}, {7, 4}, {7, 8}, {8, 3}, {9, 3},
                                   {10, 12}, {11, 12}, {12, 12}};
    std::vector<LaunchShape> cand;
    for (const auto &t : TILES) cand.push_back(LaunchShape{0, t[0], t[1]});
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++)
            for (int k = 0; k < 3; k++)
                if (BX[i] * RY[j] <= 512) cand.push_back(LaunchShape{BX[i], RY[j], BPS[k]});
    float best = 1e30f;
    LaunchShape pick = e->shape;
    for (const LaunchShape &c : cand) {
        int rc = lb_ensemble_set_launch(e, c.bx, c.ry, c.bps);
        if (rc != LB_OK) return rc;
        LB_ETRY(e, "autotune", ens_launch(e, e->cur, false));  // one untimed launch
        e->cur = 1 - e->cur;
        const int per = ens_steps_per_launch(e), trials = (trial_steps + per - 1) / per;
        LB_ETRY(e, "autotune", cudaEventRecord(e->ev0, e->stream));
        for (int s = 0; s < trials; s++) {
            LB_ETRY(e, "autotune", ens_launch(e, e->cur, false));
            e->cur = 1 - e->cur;
        }
        LB_ETRY(e, "autotune", cudaEventRecord(e->ev1, e->stream));
        LB_ETRY(e, "autotune", cudaEventSynchronize(e->ev1));
        float ms = 0.f;
        LB_ETRY(e, "autotune", cudaEventElapsedTime(&ms, e->ev0, e->ev1));
        ms /= trials * per;  // a step
        if (ms < best) {
            best = ms;
            pick = e->shape;
        }
    }
    const int rc = lb_ensemble_set_launch(e, pick.bx, pick.ry, pick.bps);
    if (rc != LB_OK) return rc;
    if (out) lb_ensemble_get_launch(e, out);
    return LB_OK;
}

}  // extern "C"
