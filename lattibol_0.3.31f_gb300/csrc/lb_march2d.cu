// lb_march2d.cu -- three native D2Q9 steps in one pass over memory.
//
// One step per launch moves 73 B per node and step, so a lattice beyond L2 runs
// at 82-85 GLUPS whatever its kernel does (6 TB/s).  Here a warp marches down a
// strip of 64 columns (a column pair per lane) with the time levels in between
// in registers: when input row i has arrived, level 1 relaxes row i - 1, level 2
// row i - 2 and level 3 row i - 3, which goes to memory.  Per level a lane keeps
// what the rows below will pull -- populations 4, 7, 8 of two rows, 0, 1, 3 of
// one -- already moved along x (the columns' neighbours by one shuffle per
// population and row); there is no barrier and no shared state between warps.
// Each level loses a column on each side and a row at each end of the item, so
// a strip stores 56 of its 64 columns and an item reads 2 T rows more than it
// stores.  Input rows arrive in a ring of four per warp by 16-byte cp.async,
// three rows ahead of their use.
//
// Both nodes of a pair go through the paired FP32 instructions (lb_pairs.cuh),
// every lane the scalar operations in the scalar order: the bits of three
// d2q9_fused_kernel launches, half-way bounce-back and moving walls included.
//
// Measured (GLUPS, one lattice / three side by side; one launch per step in
// brackets): 1568 x 1024 157 / 181 (81 / 82), 2048^2 191 / 215 (80 / 84),
// 4096 x 2048 203 / 230 (82 / 85), 1567 x 1024 (odd rows: 4-byte copies) 140 /
// 163 (83 / 81).  It is bound by the latency of its arithmetic chain at 12 warps
// per SM (152-168 registers; ncu: 48 % issue) and, on large lattices, by memory
// (4.9 TB/s).  What was tried: rows copied 8 bytes per lane through L1 160
// (4096 x 2048; 16-byte copies by way of L2 only: 181 at the same shape), input
// rows prefetched into registers 125, four warps per block instead of one 125
// (a wave of equal warps runs one after another, small blocks refill), the
// march unrolled by four 145 (instruction fetch), levels' rows in shared memory
// instead of registers 139 (nine warps per SM), four steps per pass 212 against
// 203 at 4096 x 2048 but 154 against 157 at 1568 x 1024.
#include <algorithm>

#include "lb_pairs.cuh"

namespace lb {

namespace {

constexpr int T = 3;               // steps per pass
constexpr int MD_BLOCKS = 12;      // one-warp blocks per SM
// tile columns of a strip of 64: each step loses one on each side, rounded up so
// that tiles start on 16 bytes
constexpr int MD_EDGE = 4, MD_COLS = 64 - 2 * MD_EDGE;
constexpr int MD_IN = 4;           // input rows in a warp's ring
constexpr int MD_ROW = 9 * 32 + 16;     // column pairs: nine populations, the masks
constexpr uint32_t MD_NEAR = 0x00ff00ffu;  // wall bits of a mask pair

struct MarchArgs {
    D2Args a;
    const uint16_t *mask;
    int tw, rows, strips, items;  // MarchPlan
    PairConst c;
    PairD2 d;
};

// 16 bytes by way of L2 only, 8 or 4 through L1
template <int BYTES> __device__ __forceinline__ void md_copy(void *dst, const void *src) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(dst)),
                     "l"(src)
                     : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(BYTES == 16 ? 8 : BYTES)
                 : "memory");
}

__device__ __forceinline__ int md_wrap(int v, int n) {
    v %= n;
    return v < 0 ? v + n : v;
}

// own populations of both nodes chosen where the mask says that the upstream
// node is a wall: half-way bounce-back, minus the moving-wall term
template <int K>
__device__ __forceinline__ void md_bounce(float2 &v, float2 own, uint32_t m, const float *corr) {
    constexpr int bit = K - 1;
    const float c = corr[d2_opp(K)];
    if (m >> bit & 1) v.x = (m >> (8 + bit) & 1) ? own.x - c : own.x;
    if (m >> (16 + bit) & 1) v.y = (m >> (24 + bit) & 1) ? own.y - c : own.y;
}

}  // namespace

// VEC: columns per copy of an input row, 4 (W a multiple of 4), 2 (W even) or 1
template <bool MOM, bool WALLS, int VEC>
__global__ void __launch_bounds__(32, MD_BLOCKS)
    d2q9_march_kernel(const __grid_constant__ MarchArgs ma) {
    constexpr bool ALIGNED = VEC > 1;  // W even: a column pair is one access, never wrapped
    extern __shared__ __align__(16) float2 md_smem[];
    const D2Args &a = ma.a;
    const int lane = threadIdx.x;
    const int item = a.reverse ? ma.items - 1 - (int)blockIdx.x : (int)blockIdx.x;
    const int W = a.W, H = a.H;
    const int strip = item % ma.strips, x0 = strip * ma.tw, y0 = (item / ma.strips) * ma.rows;
    const int nw = min(ma.tw, W - x0), nr = min(ma.rows, H - y0);
    const int xs = x0 - MD_EDGE + 2 * lane;
    const int xa = md_wrap(xs, W), xb = wrap_inc(xa, W);
    const bool own_a = xs >= x0 && xs < x0 + nw, own_b = xs + 1 >= x0 && xs + 1 < x0 + nw;
    const bool force = a.Fx != 0.f || a.Fy != 0.f;
    const int last = nr + 2 * T;  // input rows y0 - T .. y0 + nr - 1 + T
    float2 *const ring = md_smem + lane;

    int y = md_wrap(y0 - T, H);
    // VEC 4: this lane's 16-byte chunks of a row (16 of each population's 64 columns)
    const float *cs[5];
#pragma unroll
    for (int j = 0; VEC == 4 && j < 5; j++) {
        const int c = min(lane + 32 * j, 143), k = c >> 4;
        cs[j] = a.src.f[0];
#pragma unroll
        for (int m = 1; m < 9; m++)
            if (k == m) cs[j] = a.src.f[m];
        cs[j] += md_wrap(x0 - MD_EDGE + 4 * (c & 15), W);
    }
    // row i into slot `slot` of the ring as one commit group (empty past the end)
    auto copy = [&](int i, int slot) {
        if (i < last) {
            const uint32_t o = (uint32_t)y * (uint32_t)W;
            float2 *const d = ring + slot * MD_ROW;
            if (VEC == 4) {
#pragma unroll
                for (int j = 0; j < 5; j++)
                    if (lane + 32 * j < 144) md_copy<16>(d - lane + 2 * (lane + 32 * j), cs[j] + o);
            }
#pragma unroll
            for (int k = 0; VEC < 4 && k < 9; k++) {
                if (ALIGNED) {
                    md_copy<8>(d + k * 32, a.src.f[k] + (o + xa));
                } else {
                    md_copy<4>(&d[k * 32].x, a.src.f[k] + (o + xa));
                    md_copy<4>(&d[k * 32].y, a.src.f[k] + (o + xb));
                }
            }
            if (WALLS) {
                uint32_t *const m = reinterpret_cast<uint32_t *>(d - lane + 9 * 32) + lane;
                if (ALIGNED) md_copy<4>(m, ma.mask + (o + xa));
                else {
                    const uint32_t lo = ld_stream<true>(ma.mask + (o + xa));
                    *m = lo | (uint32_t)ld_stream<true>(ma.mask + (o + xb)) << 16;
                }
            }
            y = wrap_inc(y, H);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // programmatic dependent of the previous launch: its rows are complete
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
    for (int j = 0; j < MD_IN - 1; j++) copy(j, j);

    // Per level, moved along x already: populations 4, 7, 8 of the last row (p)
    // and the one before it (q), populations 0, 1, 3 of the last row (b)
    float2 p[T][3], q[T][3], b[T][3];
    uint32_t mk[T + 1];     // masks of rows i, i - 1, .., i - T
    uint32_t hist = 0;      // bit j: some node of row i - j has a wall upstream
#pragma unroll
    for (int t = 0; t < T; t++)
#pragma unroll
        for (int j = 0; j < 3; j++) p[t][j] = q[t][j] = b[t][j] = both(1.f);
#pragma unroll
    for (int t = 0; t <= T; t++) mk[t] = 0;
    int slot = 0, next = MD_IN - 1;
#pragma unroll 1
    for (int i = 0; i < last; i++) {
        if (VEC == 4) __syncwarp();  // every lane has read the slot that the copy overwrites
        copy(i + MD_IN - 1, next);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(MD_IN - 1) : "memory");
        if (VEC == 4) __syncwarp();  // and every lane's copies have landed
        const float2 *const row = ring + slot * MD_ROW;
        float2 n[9];
#pragma unroll
        for (int k = 0; k < 9; k++) n[k] = row[k * 32];
        if (WALLS) {
#pragma unroll
            for (int t = T; t > 0; t--) mk[t] = mk[t - 1];
            mk[0] = (reinterpret_cast<const uint32_t *>(row - lane + 9 * 32))[lane];
            hist = hist << 1 | (__any_sync(0xffffffffu, mk[0] & MD_NEAR) ? 1u : 0u);
        }
        next = slot;
        slot = slot == MD_IN - 1 ? 0 : slot + 1;
#pragma unroll
        for (int t = 1; t <= T; t++) {
            // n: row r + 1 = i - t + 1 of level t - 1; the step computes row r = i - t
            float2(&a1)[3] = p[t - 1], (&a2)[3] = q[t - 1], (&bb)[3] = b[t - 1];
            const uint32_t mr = mk[t], mr1 = mk[t - 1];
            float2 s[9];
#pragma unroll
            for (int k = 0; k < 9; k++) s[k] = row_shift(n[k], d2_cx(k));
            float2 g[9];
            g[0] = bb[0]; g[1] = bb[1]; g[3] = bb[2];
            g[4] = a2[0]; g[7] = a2[1]; g[8] = a2[2];
            g[2] = s[2]; g[5] = s[5]; g[6] = s[6];
            if (WALLS && (hist >> (t - 1) & 3)) {
                // row r: what comes up from row r + 1 where that node is a wall
                const float2 f4 = a1[0];
                const float2 f7 = row_shift(a1[1], 1), f8 = row_shift(a1[2], -1);
                md_bounce<2>(g[2], f4, mr, a.corr);
                md_bounce<5>(g[5], f7, mr, a.corr);
                md_bounce<6>(g[6], f8, mr, a.corr);
                // row r + 1: along the row, and what comes down from row r
                md_bounce<1>(s[1], n[3], mr1, a.corr);
                md_bounce<3>(s[3], n[1], mr1, a.corr);
                md_bounce<4>(a1[0], n[2], mr1, a.corr);
                md_bounce<7>(a1[1], n[5], mr1, a.corr);
                md_bounce<8>(a1[2], n[6], mr1, a.corr);
            }
            bb[0] = s[0]; bb[1] = s[1]; bb[2] = s[3];
#pragma unroll
            for (int j = 0; j < 3; j++) a2[j] = a1[j];
            a1[0] = s[4]; a1[1] = s[7]; a1[2] = s[8];
            {
                float2 rho, ux, uy;
                d2q9_collide_pairs(ma.c, ma.d, g, force, rho, ux, uy);
                const bool wall_a = WALLS && (mr & 0xffffu) == 0xff00u;
                const bool wall_b = WALLS && (mr >> 16) == 0xff00u;
                if (a.probe) {
                    const int r = i - t - T;  // row of the item
                    if (r >= 0 && r < nr) {
                        if (own_a && xa + W * (y0 + r) == a.probe_o)
                            *a.probe = wall_a ? make_float4(0.f, 0.f, 0.f, 0.f)
                                              : make_float4(ux.x, uy.x, 0.f, rho.x);
                        if (own_b && xb + W * (y0 + r) == a.probe_o)
                            *a.probe = wall_b ? make_float4(0.f, 0.f, 0.f, 0.f)
                                              : make_float4(ux.y, uy.y, 0.f, rho.y);
                    }
                }
                if (t < T) {
#pragma unroll
                    for (int k = 0; k < 9; k++) n[k] = g[k];
                } else if (i >= 2 * T) {
                    const uint32_t o = (uint32_t)(y0 + i - 2 * T) * (uint32_t)W;
                    if (MOM) {
                        if (wall_a) { rho.x = 0.f; ux.x = 0.f; uy.x = 0.f; }
                        if (wall_b) { rho.y = 0.f; ux.y = 0.f; uy.y = 0.f; }
                        if (own_a) { a.rho[o + xa] = rho.x; a.ux[o + xa] = ux.x; a.uy[o + xa] = uy.x; }
                        if (own_b) { a.rho[o + xb] = rho.y; a.ux[o + xb] = ux.y; a.uy[o + xb] = uy.y; }
                    }
                    const bool sa = own_a && !wall_a, sb = own_b && !wall_b;
                    if (ALIGNED && sa && sb) {
#pragma unroll
                        for (int k = 0; k < 9; k++)
                            *reinterpret_cast<float2 *>(a.dst.f[k] + (o + xa)) = g[k];
                    } else {
                        if (sa) {
#pragma unroll
                            for (int k = 0; k < 9; k++) a.dst.f[k][o + xa] = g[k].x;
                        }
                        if (sb) {
#pragma unroll
                            for (int k = 0; k < 9; k++) a.dst.f[k][o + xb] = g[k].y;
                        }
                    }
                }
            }
        }
    }
}

// a node's mask: bit k - 1 when the node at x - c_k is a wall, bit 7 + k when
// that wall moves; 0xff00 marks a wall node
__global__ void d2q9_wall_mask_kernel(const uint8_t *flags, uint16_t *mask, int W, int H) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W) return;
    uint32_t m = 0;
    if (flags[x + W * y] & CELL_WALL) {
        m = 0xff00u;
    } else {
#pragma unroll
        for (int k = 1; k < 9; k++) {
            const int ux = wrap_add(x, -d2_cx(k), W), uy = wrap_add(y, -d2_cr(k), H);
            const uint8_t f = flags[ux + W * uy];
            if (f & CELL_WALL) m |= 1u << (k - 1) | (f & CELL_MOVING ? 1u << (7 + k) : 0u);
        }
    }
    mask[x + W * y] = (uint16_t)m;
}

cudaError_t launch_d2q9_wall_mask(const uint8_t *flags, uint16_t *mask, int W, int H,
                                  cudaStream_t s) {
    d2q9_wall_mask_kernel<<<dim3((W + 127) / 128, H), 128, 0, s>>>(flags, mask, W, H);
    return cudaGetLastError();
}

namespace {

template <bool MOM, bool WALLS>
cudaError_t md_launch(const MarchArgs &ma, cudaStream_t s) {
    const int W = ma.a.W;
    const auto kernel = W % 4 == 0   ? d2q9_march_kernel<MOM, WALLS, 4>
                        : W % 2 == 0 ? d2q9_march_kernel<MOM, WALLS, 2>
                                     : d2q9_march_kernel<MOM, WALLS, 1>;
    return launch_dependent_smem(kernel, dim3(ma.items), dim3(32),
                                 MD_IN * MD_ROW * sizeof(float2), s, ma);
}

}  // namespace

int march_steps_per_launch() { return T; }

// Rows per item: fewer rows fill the GPU's warps, more rows pay less for the 2 T
// rows that an item reads beyond its own.  A pass takes an item's march times a
// function of the rounds of items w (a partly filled round runs its warps
// faster, a nearly empty second one costs almost as much as a full one;
// measured at 1568 x 1024, us per step: 16 rows, 1792 items for 1824 warps, 10.2;
// 8 rows 12.6, 12 rows 12.7, 24 rows 13.5, 32 rows 12.8, 48 rows 16.9).
MarchPlan march_plan(int W, int H) {
    MarchPlan p{};
    const int ns = (W + MD_COLS - 1) / MD_COLS;
    p.tw = ((W + ns - 1) / ns + 3) & ~3;
    p.strips = (W + p.tw - 1) / p.tw;
    const double warps = 152. * MD_BLOCKS;
    double best = 0;
    for (int c = 1; c <= H; c++) {
        const int r = (H + c - 1) / c;
        const double w = p.strips * (double)((H + r - 1) / r) / warps;
        const double cost =
            (r + 2. * T) * (w <= 1. ? 0.65 + 0.35 * w : std::max(1.42, 0.32 + 0.82 * w));
        if (best == 0 || cost < best) {
            best = cost;
            p.rows = r;
        }
    }
    p.items = p.strips * ((H + p.rows - 1) / p.rows);
    // us per step: the upper end of what lattices of 0.53 .. 2.7 M nodes without walls
    // and of 3 .. 100 rows gave.  Up to one round of items it is one march, whatever w
    // (odd widths 0.43 .. 0.48 per row, others 0.36 .. 0.42); beyond, it follows the cost
    // (0.43 .. 0.50, 0.38 .. 0.46).
    const bool odd = W % 2 != 0;
    p.us = p.items <= warps ? (p.rows + 2 * T) * (odd ? 0.48 : 0.41) : best * (odd ? 0.50 : 0.45);
    return p;
}

// Whether the strips beat one launch per step (beyond 2^19 nodes).  From 32 rows on
// they did on every shape without force or walls (1.02 to 2.5 times; 135 shapes of 0.53
// .. 2.7 M nodes, with rows that start on 4, 8 and 16 bytes).  With a force, 96 shapes,
// time over one launch per step's, one lattice alone: 0.43 .. 1.07 without walls, 0.40 ..
// 1.01 with 5 % of them, 0.55 .. 1.20 in a box, above 1 only under 1.2 M nodes (a strip
// along a wall marches longer, and one lattice is one round of them); three lattices
// side by side, 21 shapes of 0.53 .. 1.2 M nodes: 0.55 .. 0.90, 0.46 .. 0.82 and 0.59 ..
// 1.00 (925 x 622; with a disc between two walls 1.04).  On fewer rows the 2 T rows that
// an item reads beyond its own can outweigh it: us per step, strips / one launch per
// step, 700 001 x 1 17.6 / 6.4, 175 000 x 4 7.8 / 6.6, 53 125 x 16 9.9 / 8.2, but
// 50 001 x 20 7.5 / 9.7 and 525 000 x 4 19.5 / 25.4.  There the plan's time is compared
// with that of a launch per step, 0.3 us and 9.5 ps per thread (blocks of 128 along a
// row), 11.5 beyond 1.6 M threads, where the two population sets leave L2.
bool march_pays(int W, int H) {
    if (H >= 32) return true;
    const double threads = 128. * ((W + 127) / 128) * H;
    return march_plan(W, H).us < 0.3 + threads * (threads > 1.6e6 ? 11.5e-6 : 9.5e-6);
}

cudaError_t launch_d2q9_march(const D2Args &a, const MarchPlan &p, const uint16_t *mask, bool mom,
                              cudaStream_t s) {
    if (a.G != 0.f) return cudaErrorInvalidValue;  // no Shan-Chen here
    MarchArgs ma{};
    ma.a = a;
    ma.tw = p.tw;
    ma.rows = p.rows;
    ma.strips = p.strips;
    ma.items = p.items;
    ma.mask = mask;
    ma.c = pair_constants();
    const auto two = [](float v) { return make_float2(v, v); };
    ma.d = PairD2{two(-a.w0), two(-a.w1), two(-a.w5), two(-a.tau_inv),
                  two(a.tau_inv), two(a.Fx), two(a.Fy)};
    if (mask) return mom ? md_launch<true, true>(ma, s) : md_launch<false, true>(ma, s);
    return mom ? md_launch<true, false>(ma, s) : md_launch<false, false>(ma, s);
}

}  // namespace lb
