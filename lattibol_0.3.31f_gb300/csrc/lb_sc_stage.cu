// lb_sc_stage.cu -- single-pass D3Q19 Shan-Chen step for lattices without
// wall nodes (the periodic spinodal case), fed by asynchronous copies into
// shared memory.
//
// A block owns a column tile (64 x 8 nodes in 16-bit storage, 32 x 8 in FP32
// and where the width is no multiple of 64), two neighbouring nodes of a row
// per thread, and marches through a chunk of z planes.  The populations reach
// shared memory as "stages": stage z holds, for every population k, what the
// pulls of plane z read for the tile and the ring around it -- rows y0-1-c_y ..
// y0+8-c_y of plane z - c_z(k), the columns rounded out to 16 bytes on the
// sides that c_x needs (28.8 KB per stage in both tiles) -- copied in 16-byte
// cp.async chunks (periodic in x, y and z; the wrap in x and y is folded into
// each thread's chunk addresses, formed once per block) that report on the
// slot's mbarrier when they have landed.  Stages are issued two steps ahead of
// their use, so DRAM latency is covered by copies in flight rather than by
// warps waiting on loads.
//
// Step j of the march takes stage z = z0 - 1 + j: every thread pulls its own
// nodes from it (kept in registers for the relaxation one step later), the
// first warps also pull the two rows and two columns of the ring around the
// tile; each forms psi(rho) into a four-plane psi buffer.  One barrier later
// the slot is refilled with the stage two planes ahead and plane z - 1 is
// relaxed from the kept populations and the psi stencil of planes z - 2 .. z.
// Four psi slots make that one barrier per plane enough (a warp writing psi of
// plane z + 1 has passed the barrier of plane z, reached only after every warp
// relaxed plane z - 2, the last reader of that slot).
//
// Arithmetic: the pulls read the same stored values as the two-pass step,
// widened the same way; the two nodes' density, stencil sum and relaxation are
// the operations of StepArith<S> and d3q19_sc_sum_native in the same order, in
// the paired FP32 instructions (lb_pairs.cuh), so the result is bit-identical
// to the density pass + fused step.
//
// Measured at 256^3 (GLUPS FP32 / FP16 / BF16): 36.1 / 54.5 / 56.2; one node per
// thread, 19 TMA boxes per stage for the interior tiles of 16-bit storage and
// chunks of a divisor of the depth: 35.0 / 42.0 / 42.0; at 128^3 31.8 / 45.3
// against 25.8 / 29.1, at 64^3 19.6 / 27.2 against 17.9 / 20.1.  (800 issue slots
// per node bound the 16-bit step then; now 375.)  With two nodes per thread the TMA
// boxes (ten rows of 160 bytes, 48.5) lose to the cp.async chunks, which read
// fewer bytes on the sides.  What bounds the step now: FP32, memory (the same
// copies and stores without any arithmetic between them: 39); 16-bit, the
// latency of a plane's chain (copies landed, pulls, psi, barrier, stencil,
// relaxation) at 16 warps per SM, which their registers allow (the copies and
// stores alone: 77); at that bound, 128, the compiler spills 28 to 48 bytes per
// thread (80 to 188 bytes of loads), in FP32 (159 to 163 registers) none.  Tried
// without gain (54.8 in the same runs): 3 stages ahead (54.6), populations
// kept as 16-bit words (52.9; 37 at 24 warps per SM, whose 80 registers spill),
// momentum formed when pulled (53.3), the barrier split into arrival and wait
// around the moments (54.6), planes and chunks backwards on odd steps (54.7),
// tiles of 32 x 16 (FP32 35.3, FP16 46.6).
//
// Every mbarrier wait is bounded (wait_limit polls for a stage; ST_WAIT in the
// library's launches); a block that gives up raises
// the device error word, waits (bounded by ST_WAIT) for the stages it still
// has in flight, drains its threads' own copies (cp.async.wait_all) and
// returns.  sc_stage_wait_selftest makes the first wait run out (wait_limit
// 0) to exercise that path.
#include <algorithm>
#include <cmath>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "lb_d3q19.cuh"
#include "lb_pairs.cuh"
#include "lb_tc05.cuh"

namespace lb {

namespace {

constexpr int ST_TY = 8;                              // rows of a tile
constexpr int ST_WAIT = 1 << 22;                      // mbarrier polls before giving up

// A tile of TX columns and the layout of its stages.  Population k holds the 10
// rows its pulls read for the tile and its ring (rows y0-1-c_y .. y0+8-c_y of
// plane z - c_z), row after row, over the columns they read: x0-1-c_x ..
// x0+TX-c_x rounded out to 16-byte chunks, TX + 2E columns for c_x = 0 and TX + E
// otherwise, the populations packed one after another.  Column c below counts
// from x0 - E.
template <typename S, int TX_>
struct StageShape {
    static constexpr int TX = TX_;
    static constexpr int THREADS = TX * ST_TY / 2;     // two nodes each
    static constexpr int PX = TX + 4, PY = ST_TY + 2;  // psi plane: columns -2 .. TX + 1, rows -1 .. 8
    static constexpr int E = 16 / (int)sizeof(S);      // elements per 16-byte chunk
    static constexpr int ROWS = ST_TY + 2;             // rows of every population
    // first column (relative to x0) and width of population k
    static constexpr int col0(int k) { return d3_cx(k) < 0 ? 0 : -E; }
    static constexpr int width(int k) { return d3_cx(k) == 0 ? TX + 2 * E : TX + E; }
    static constexpr int chunks(int k) { return ROWS * width(k) / E; }
    static constexpr int first_chunk(int k) {
        int c = 0;
        for (int j = 0; j < k; j++) c += chunks(j);
        return c;
    }
    static constexpr int CHUNKS = first_chunk(19);      // 1800 of FP32; 1040, 1800 of 16 bits
    static constexpr int BYTES = CHUNKS * 16;
    static constexpr int ELEMS = BYTES / (int)sizeof(S);
    static constexpr int SLOTS = 2;
    // resident blocks per SM: 12 warps of FP32 (shared memory), 16 of 16 bits (registers)
    static constexpr int MIN_BLOCKS = sizeof(S) == 4 ? 3 : 512 / THREADS;
    static constexpr int PSI_BYTES = 4 * PY * PX * (int)sizeof(float);
    static constexpr int SMEM = SLOTS * BYTES + PSI_BYTES + SLOTS * 8;
    // element of population k, stage row r, column c (0 = x0 - E)
    static constexpr int elem(int k, int r, int c) {
        return first_chunk(k) * E + r * width(k) + c - E - col0(k);
    }
    static_assert(BYTES % 16 == 0 && PSI_BYTES % 16 == 0, "stage alignment");
};

// the stored value of population k as the step works on it (Store<S>::load_dev:
// f_k in FP32, the deviation d_k in 16-bit storage)
__device__ __forceinline__ float widen(float v) { return v; }
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }

// v in [-n, 2n): its periodic image in [0, n)
__device__ __forceinline__ int wrap1(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

// 16 bytes from global memory into shared memory (L2 only), asynchronously
__device__ __forceinline__ void cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
// one arrival on mbar once every cp.async this thread issued so far has landed
__device__ __forceinline__ void cp_arrive(uint64_t *mbar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(mbar))
                 : "memory");
}

// What chunk c of a stage is, laid out by the compiler (formed by each thread
// from c, it cost a block some 60 instructions per chunk): population k in bits
// 0..4, its z class (0, 1, 2 for c_z = +1, 0, -1) in bits 5 and 6, row - c_y + 1
// in bits 8..15 (row - 1 - c_y relative to y0, plus 2) and the first column
// relative to x0, plus E, in bits 16 and up.
template <typename S, int TX> struct ChunkTable {
    uint32_t v[StageShape<S, TX>::CHUNKS];
    constexpr ChunkTable() : v() {
        using SS = StageShape<S, TX>;
        int c = 0;
        for (int k = 0; k < 19; k++)
            for (int r = 0; r < SS::ROWS; r++)
                for (int q = 0; q < SS::width(k) / SS::E; q++)
                    v[c++] = (uint32_t)(k | (1 - d3_cz(k)) << 5 | (r - d3_cy(k) + 1) << 8 |
                                        (SS::col0(k) + q * SS::E + SS::E) << 16);
    }
};
template <typename S, int TX> __device__ constexpr ChunkTable<S, TX> chunk_table{};

// cp.async copies of a stage.  Thread t copies chunks t, t +
// THREADS, ...; which global row and column each of its chunks reads does not
// change from plane to plane, so the thread forms those offsets once: the
// element offset from population 0's array in plane z - 1 for stage z (the
// populations lie at f[0] + k * stride, and the launch guarantees 19 strides fit
// in 32 bits), and the chunk's z class -- plane z - c_z is read for plane z --
// for the stages whose planes wrap around.
template <typename S, int TX>
struct StageCopy {
    using SS = StageShape<S, TX>;
    static constexpr int E = SS::E;
    static constexpr int CHUNKS = SS::CHUNKS;
    static constexpr int PER_T = (CHUNKS + SS::THREADS - 1) / SS::THREADS;
    uint32_t off[PER_T];
    uint32_t cls_of = 0;

    __device__ __forceinline__ StageCopy(const D3Args &a, int x0, int y0) {
        const long stride = (reinterpret_cast<const char *>(a.src.f[1]) -
                             reinterpret_cast<const char *>(a.src.f[0])) / (long)sizeof(S);
#pragma unroll
        for (int i = 0; i < PER_T; i++) {
            const int c = min((int)threadIdx.x + SS::THREADS * i, CHUNKS - 1);
            const uint32_t e = chunk_table<S, TX>.v[c];
            const int k = e & 31, cls = e >> 5 & 3;
            const int yr = wrap1(y0 - 2 + (int)(e >> 8 & 255), a.H);
            const int xm = wrap1(x0 - E + (int)(e >> 16), a.W);
            off[i] = (uint32_t)(k * stride + (long)yr * a.W + xm + (long)cls * (a.W * a.H));
            cls_of |= (uint32_t)cls << 2 * i;
        }
    }

    // stage of plane zs into slot; one arrival per thread on mbar
    __device__ __forceinline__ void issue(const D3Args &a, S *slot, uint64_t *mbar, int zs) const {
        const int plane = a.W * a.H;
        char *dst = reinterpret_cast<char *>(slot);
        const S *base = reinterpret_cast<const S *>(a.src.f[0]);
        if (zs >= 1 && zs + 1 < a.D) {
            // no chunk wraps in z
            base += (long)(zs - 1) * plane;
#pragma unroll
            for (int i = 0; i < PER_T; i++) {
                const int c = (int)threadIdx.x + SS::THREADS * i;
                if (i == PER_T - 1 && c >= CHUNKS) break;
                cp16(dst + 16 * c, base + off[i]);
            }
        } else {
            const int zw[3] = {wrap1(zs - 1, a.D), wrap1(zs, a.D) - 1, wrap1(zs + 1, a.D) - 2};
#pragma unroll
            for (int i = 0; i < PER_T; i++) {
                const int c = (int)threadIdx.x + SS::THREADS * i;
                if (i == PER_T - 1 && c >= CHUNKS) break;
                const int cls = cls_of >> 2 * i & 3;
                cp16(dst + 16 * c,
                     base + ((long)(cls == 0 ? zw[0] : cls == 1 ? zw[1] : zw[2]) * plane + off[i]));
            }
        }
        cp_arrive(mbar);
    }
};

// the 19 post-stream populations of the ring node (rx, ry) relative to the
// tile origin (rx in -1..TX, ry in -1..8): population k comes from row
// ry - c_y (local row ry + 1 of its rows) and column rx - c_x
template <typename S, int TX>
__device__ __forceinline__ void pull_stage(const S *st, int rx, int ry, float (&g)[19]) {
    using SS = StageShape<S, TX>;
#pragma unroll
    for (int k = 0; k < 19; k++) g[k] = widen(st[SS::elem(k, ry + 1, rx - d3_cx(k) + SS::E)]);
}

// two neighbouring stored values, widened (aligned to the pair)
__device__ __forceinline__ float2 widen2(const float *p) {
    return *reinterpret_cast<const float2 *>(p);
}
__device__ __forceinline__ float2 widen2(const __half *p) {
    return __half22float2(*reinterpret_cast<const __half2 *>(p));
}
__device__ __forceinline__ float2 widen2(const __nv_bfloat16 *p) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(p));
}
// two neighbouring values to storage (aligned to the pair), as Store<S>::store_dev
__device__ __forceinline__ void store2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }
__device__ __forceinline__ void store2(__half *p, float2 v) {
    *reinterpret_cast<__half2 *>(p) = __float22half2_rn(v);
}
__device__ __forceinline__ void store2(__nv_bfloat16 *p, float2 v) {
    *reinterpret_cast<__nv_bfloat162 *>(p) = __float22bfloat162_rn(v);
}
// the 19 post-stream populations of nodes (rx, ry) and (rx + 1, ry), rx even
template <typename S, int TX>
__device__ __forceinline__ void pull_stage2(const S *st, int rx, int ry, float2 (&g)[19]) {
    using SS = StageShape<S, TX>;
#pragma unroll
    for (int k = 0; k < 19; k++) {
        const S *p = st + SS::elem(k, ry + 1, rx - d3_cx(k) + SS::E);
        g[k] = d3_cx(k) == 0 ? widen2(p) : make_float2(widen(p[0]), widen(p[1]));
    }
}

// the relaxation of two nodes in the order of StepArith<S>'s operations;
// constants of the step, each twice
struct PairD3 {
    float2 tau;                       // tau_inv
    float2 w0, w1, w7, mt;            // FP32: -w0, -w1, -w7, -tau_inv
                                      // 16-bit: w0, w1, w7, 1 - tau_inv
    float2 r0, r1, r7, ref;           // 16-bit: -tau_inv w_k rho_ref; rho_ref
};

// density, and the sums of c_x = +1 and -1, as StepArith<S>::rho
template <typename S>
__device__ __forceinline__ float2 pair_rho(const PairD3 &d, const float2 (&g)[19], float2 &px,
                                           float2 &mx) {
    const auto add = [](float2 a, float2 b) { return pair_add(a, b); };
    px = add(add(add(g[1], g[7]), add(g[8], g[9])), g[10]);
    mx = add(add(add(g[2], g[11]), add(g[12], g[13])), g[14]);
    const float2 zx = add(add(add(add(g[0], g[3]), add(g[4], g[5])),
                              add(add(g[6], g[15]), add(g[16], g[17]))), g[18]);
    const float2 rho = add(add(px, mx), zx);
    return sizeof(S) == 2 ? add(d.ref, rho) : rho;
}

template <typename S>
__device__ __forceinline__ void pair_bgk(const PairConst &c, const PairD3 &d, float2 (&g)[19],
                                         float2 ex, float2 ey, float2 ez, float2 rho) {
    const float2 usq = __ffma2_rn(ez, ez, __ffma2_rn(ey, ey, __fmul2_rn(ex, ex)));
    const float2 base = __ffma2_rn(c.m15, usq, c.one);
    float2 a0 = __fmul2_rn(d.w0, rho), a1 = __fmul2_rn(d.w1, rho), a7 = __fmul2_rn(d.w7, rho);
    if (sizeof(S) == 2) {
        a0 = __fmul2_rn(d.tau, a0);
        a1 = __fmul2_rn(d.tau, a1);
        a7 = __fmul2_rn(d.tau, a7);
    }
    // FP32: e = -(f_eq - g) in one rounding, then g - tau_inv e: the scalar form
    // with both signs turned (rounding is symmetric)
    const auto one = [&](int i, float2 a, float2 r, float2 q) {
        g[i] = sizeof(S) == 4 ? __ffma2_rn(d.mt, __ffma2_rn(a, q, g[i]), g[i])
                              : __ffma2_rn(d.mt, g[i], __ffma2_rn(a, q, r));
    };
    const auto pair = [&](int kp, int km, float2 a, float2 r, float2 p) {
        const float2 t = __ffma2_rn(__fmul2_rn(c.c45, p), p, base);
        one(kp, a, r, __ffma2_rn(c.c3, p, t));
        one(km, a, r, __ffma2_rn(c.m3, p, t));
    };
    one(0, a0, d.r0, base);
    pair(1, 2, a1, d.r1, ex);
    pair(3, 4, a1, d.r1, ey);
    pair(5, 6, a1, d.r1, ez);
    pair(7, 12, a7, d.r7, pair_addp(c, ex, ey));
    pair(8, 11, a7, d.r7, pair_sub(c, ex, ey));
    pair(9, 14, a7, d.r7, pair_addp(c, ex, ez));
    pair(10, 13, a7, d.r7, pair_sub(c, ex, ez));
    pair(15, 18, a7, d.r7, pair_addp(c, ey, ez));
    pair(16, 17, a7, d.r7, pair_sub(c, ey, ez));
}

// the pseudo-potential of both nodes
template <int PSI>
__device__ __forceinline__ float2 psi_of(const PairConst &c, float2 rho) {
    return PSI == 0 ? make_float2(psi_ref(rho.x), psi_ref(rho.y)) : pair_psi_exp1(c, rho);
}

}  // namespace

template <typename S, bool MOM, int PSI, int TX>
__global__ void __launch_bounds__((StageShape<S, TX>::THREADS), (StageShape<S, TX>::MIN_BLOCKS))
    d3q19_sc_stage_kernel(const __grid_constant__ D3Args a, int zc, int wait_limit,
                          const __grid_constant__ PairConst c,
                          const __grid_constant__ PairD3 d) {
    using SS = StageShape<S, TX>;
    extern __shared__ __align__(128) unsigned char smem[];
    S *stage = reinterpret_cast<S *>(smem);
    float(*sp)[SS::PY][SS::PX] =
        reinterpret_cast<float(*)[SS::PY][SS::PX]>(smem + SS::SLOTS * SS::BYTES);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + SS::SLOTS * SS::BYTES + SS::PSI_BYTES);

    // this thread's nodes: columns tx, tx + 1 of row ty
    const int tid = threadIdx.x, tx = 2 * (tid % (TX / 2)), ty = tid / (TX / 2);
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * ST_TY, z0 = blockIdx.z * zc;
    const int x = x0 + tx, y = y0 + ty;

    if (tid == 0)
        for (int s = 0; s < SS::SLOTS; s++) mbar_init(&full[s], SS::THREADS);
    __syncthreads();
    const StageCopy<S, TX> cp(a, x0, y0);
    const int nst = min(zc, a.D - z0) + 2;  // stages z0 - 1 .. one beyond the chunk
    auto issue = [&](int slot, int zs) {
        cp.issue(a, stage + slot * SS::ELEMS, &full[slot], zs);
    };
    after_predecessor();  // barriers and chunk offsets are set up while it drains
    for (int j = 0; j < SS::SLOTS && j < nst; j++) issue(j, z0 - 1 + j);

    // step j: psi of plane z0 - 1 + j from its stage (the own nodes' populations
    // into gn), then the relaxation of the plane before it from gs, pulled one
    // step earlier; false when the block gave up waiting for its copies
    auto step = [&](int j, float2(&gs)[19], float2(&gn)[19]) -> bool {
        const int slot = j % SS::SLOTS;
        const int zs = z0 - 1 + j;
        const S *st = stage + slot * SS::ELEMS;
        const bool ok = mbar_wait(&full[slot], (uint32_t)((j / SS::SLOTS) & 1), wait_limit);
        float(*ps)[SS::PX] = sp[(zs + 4) & 3];
        if (ok) {
            float2 px, mx;
            pull_stage2<S, TX>(st, tx, ty, gn);
            *reinterpret_cast<float2 *>(&ps[ty + 1][tx + 2]) =
                psi_of<PSI>(c, pair_rho<S>(d, gn, px, mx));
            // the ring: its two rows in pairs, then its two columns
            if (tid < TX) {
                const int hx = 2 * (tid % (TX / 2)), hy = tid < TX / 2 ? -1 : ST_TY;
                float2 gh[19];
                pull_stage2<S, TX>(st, hx, hy, gh);
                *reinterpret_cast<float2 *>(&ps[hy + 1][hx + 2]) =
                    psi_of<PSI>(c, pair_rho<S>(d, gh, px, mx));
            } else if (tid < TX + 2 * SS::PY) {
                const int i = tid - TX, hx = i < SS::PY ? -1 : TX, hy = i % SS::PY - 1;
                float gh[19];
                pull_stage<S, TX>(st, hx, hy, gh);
                ps[hy + 1][hx + 2] = psi_form<PSI>(StepArith<S>::rho(gh, a));
            }
        }
        if (__syncthreads_or(!ok)) {
            // give up: report, then wait (bounded) for the stages still in flight
            if (tid == 0 && a.err) atomicExch(a.err, 1);
            for (int i = j; i < j + SS::SLOTS && i < nst; i++)
                mbar_wait(&full[i % SS::SLOTS], (uint32_t)((i / SS::SLOTS) & 1), ST_WAIT);
            // then drain this thread's own copies whatever those waits saw, so
            // that none can land in shared memory that the next block resident
            // on this SM reuses (memory copies always complete; no other party
            // has to act for this wait to end)
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            return false;
        }
        if (j + SS::SLOTS < nst) {
            // the barrier above ordered every thread's reads of this slot
            // before the copies that overwrite it
            issue(slot, zs + SS::SLOTS);
        }
        if (j >= 2) {
            const int z = zs - 1;
            const int o = x + a.W * (y + a.H * z);
            const auto add = [](float2 a, float2 b) { return pair_add(a, b); };
            float2 px, mx;
            const float2 rho = pair_rho<S>(d, gs, px, mx);
            const float2 jy = pair_sub(c, add(add(add(gs[3], gs[7]), add(gs[11], gs[15])), gs[16]),
                                       add(add(add(gs[4], gs[8]), add(gs[12], gs[17])), gs[18]));
            const float2 jz = pair_sub(c, add(add(add(gs[5], gs[9]), add(gs[13], gs[15])), gs[17]),
                                       add(add(add(gs[6], gs[10]), add(gs[14], gs[16])), gs[18]));
            float2 inv = rho, inv_rt = __fmul2_rn(rho, d.tau);
            pair_rcp2(c, inv, inv_rt);
            float2 ex = __fmul2_rn(pair_sub(c, px, mx), inv), ey = __fmul2_rn(jy, inv),
                   ez = __fmul2_rn(jz, inv);
            if (MOM) {
                store2(a.ux + o, ex);
                store2(a.uy + o, ey);
                store2(a.uz + o, ez);
                store2(a.rho + o, rho);
            }
            if (a.probe) {
                if (o == a.probe_o) *a.probe = make_float4(ex.x, ey.x, ez.x, rho.x);
                if (o + 1 == a.probe_o) *a.probe = make_float4(ex.y, ey.y, ez.y, rho.y);
            }
            if (a.Fx != 0.f) ex = __ffma2_rn(both(a.Fx), inv_rt, ex);
            if (a.Fy != 0.f) ey = __ffma2_rn(both(a.Fy), inv_rt, ey);
            if (a.Fz != 0.f) ez = __ffma2_rn(both(a.Fz), inv_rt, ez);
            // IF = sum_k w_k psi(x + c_k) c_k in the order of d3q19_sc_sum_native;
            // a row: psi of columns x - 1, (x, x + 1), x + 2
            struct Row {
                float l;
                float2 v;
                float r;
            };
            const auto row = [&](int cy, int cz) {
                const float *p = &sp[(z + cz + 4) & 3][ty + 1 + cy][tx + 2];
                return Row{p[-1], *reinterpret_cast<const float2 *>(p), p[2]};
            };
            const auto mid = [&](int cy, int cz) {
                return *reinterpret_cast<const float2 *>(&sp[(z + cz + 4) & 3][ty + 1 + cy][tx + 2]);
            };
            const Row r0 = row(0, 0), yp = row(1, 0), ym = row(-1, 0), zp = row(0, 1),
                      zm = row(0, -1);
            const float2 pp = mid(1, 1), pm = mid(1, -1), mp = mid(-1, 1), mm = mid(-1, -1);
            // the four diagonals at each of the columns, then their differences along x
            const float2 s_v = add(add(yp.v, ym.v), add(zp.v, zm.v));
            const float s_l = (yp.l + ym.l) + (zp.l + zm.l), s_r = (yp.r + ym.r) + (zp.r + zm.r);
            const auto across = [](const Row &q) { return make_float2(q.v.y + q.l, q.r + q.v.x); };
            const float2 w1 = both(a.w1), w7 = both(a.w7);
            const float2 IFx = __ffma2_rn(w1, make_float2(r0.v.y - r0.l, r0.r - r0.v.x),
                                          __fmul2_rn(w7, make_float2(s_v.y - s_l, s_r - s_v.x)));
            const float2 IFy = __ffma2_rn(
                w1, pair_sub(c, yp.v, ym.v),
                __fmul2_rn(w7, pair_sub(c, add(across(yp), add(pp, pm)),
                                        add(across(ym), add(mp, mm)))));
            const float2 IFz = __ffma2_rn(
                w1, pair_sub(c, zp.v, zm.v),
                __fmul2_rn(w7, pair_sub(c, add(across(zp), add(pp, mp)),
                                        add(across(zm), add(pm, mm)))));
            const float2 cf = __fmul2_rn(__fmul2_rn(both(-a.G), r0.v), inv_rt);
            ex = __ffma2_rn(cf, IFx, ex);
            ey = __ffma2_rn(cf, IFy, ey);
            ez = __ffma2_rn(cf, IFz, ez);
            pair_bgk<S>(c, d, gs, ex, ey, ez, rho);
            S *const *dst = reinterpret_cast<S *const *>(a.dst.f);
#pragma unroll
            for (int k = 0; k < 19; k++) store2(dst[k] + o, gs[k]);
        }
        return true;
    };
    // two steps per iteration with the population arrays swapped, so that no
    // step copies the pulled populations from one array to the other
    float2 ga[19], gb[19];
#pragma unroll
    for (int k = 0; k < 19; k++) ga[k] = gb[k] = both(0.f);
    int j = 0;
    for (; j + 1 < nst; j += 2) {
        if (!step(j, ga, gb)) return;
        if (!step(j + 1, gb, ga)) return;
    }
    if (j < nst && !step(j, ga, gb)) return;
    // every wait has completed and no copy is in flight
    if (tid == 0)
        for (int s = 0; s < SS::SLOTS; s++) mbar_inval(&full[s]);
}

// Lattices that the staged kernel takes: whole tiles.  The chunks have not needed a
// depth that is a multiple of 4 since chunk_planes takes any length; other depths are
// untried here and take the two-pass step.
bool sc_stage_fits(int W, int H, int D) { return W % 32 == 0 && H % ST_TY == 0 && D % 4 == 0; }

namespace {

template <typename S> PairD3 pair_d3(const D3Args &a) {
    const auto two = [](float v) { return make_float2(v, v); };
    if (sizeof(S) == 4)
        return PairD3{two(a.tau_inv), two(-a.w0), two(-a.w1), two(-a.w7), two(-a.tau_inv),
                      two(0.f), two(0.f), two(0.f), two(0.f)};
    return PairD3{two(a.tau_inv), two(a.w0), two(a.w1), two(a.w7), two(1.f - a.tau_inv),
                  two(-(a.tau_inv * a.wr[0])), two(-(a.tau_inv * a.wr[1])),
                  two(-(a.tau_inv * a.wr[7])), two(a.rho_ref)};
}

// Planes of a chunk: the fewest plane steps, a chunk's planes and the two beyond
// its ends times the waves of blocks; a single wave that leaves SMs part empty
// runs its blocks somewhat faster.  256^3 in FP16: 37 planes, 2.95 waves, 54.5
// GLUPS; 32 planes (3.4 waves) 53.0, 16 planes 51.4, 64 planes 47.4.
int chunk_planes(long tiles, int D, int resident) {
    int pick = 1;
    double best = 0;
    for (int n = 1; n <= D; n++) {
        const int zc = (D + n - 1) / n;
        const double w = (double)tiles * ((D + zc - 1) / zc) / (152. * resident);
        const double cost = (zc + 2) * (w <= 1. ? 0.65 + 0.35 * w : std::ceil(w));
        if (best == 0 || cost < best) {
            best = cost;
            pick = zc;
        }
    }
    return pick;
}

template <typename S, bool MOM, int PSI, int TX>
cudaError_t stage_launch(const D3Args &a, cudaStream_t s) {
    using SS = StageShape<S, TX>;
    static_assert(SS::MIN_BLOCKS * (SS::SMEM + 1024) <= 228 * 1024, "resident blocks per SM");
    // once per instantiation
    static const cudaError_t attr_e =
        cudaFuncSetAttribute(d3q19_sc_stage_kernel<S, MOM, PSI, TX>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, SS::SMEM);
    if (attr_e != cudaSuccess) return attr_e;
    const int nx = a.W / TX, ny = a.H / ST_TY;
    const int zc = chunk_planes((long)nx * ny, a.D, SS::MIN_BLOCKS);
    return launch_dependent_smem(d3q19_sc_stage_kernel<S, MOM, PSI, TX>,
                                 dim3(nx, ny, (a.D + zc - 1) / zc), dim3(SS::THREADS), SS::SMEM, s,
                                 a, zc, ST_WAIT, pair_constants(), pair_d3<S>(a));
}

// 16-bit storage takes the wide tile where the width allows it (256^3: 54.5
// GLUPS, the narrow one 51); in FP32 two stages of it leave room for one block
// per SM (34.0, three blocks of the narrow tile 36.0).
template <typename S, bool MOM, int PSI>
cudaError_t stage_launch(const D3Args &a, cudaStream_t s) {
    if constexpr (sizeof(S) == 2)
        if (a.W % 64 == 0) return stage_launch<S, MOM, PSI, 64>(a, s);
    return stage_launch<S, MOM, PSI, 32>(a, s);
}

template <typename S>
cudaError_t stage_launch(const D3Args &a, bool mom, cudaStream_t s) {
    if (a.psi_form == 0)
        return mom ? stage_launch<S, true, 0>(a, s) : stage_launch<S, false, 0>(a, s);
    return mom ? stage_launch<S, true, 1>(a, s) : stage_launch<S, false, 1>(a, s);
}

}  // namespace

// The give-up path of the staged step on a 32 x 8 x 4 FP32 lattice: every
// first stage wait is given no polls, so each block reports through *err,
// waits for the stages its prologue issued and returns.
cudaError_t sc_stage_wait_selftest(int *err) {
    constexpr int W = 32, H = ST_TY, D = 4, N = W * H * D;
    using SS = StageShape<float, W>;
    const auto kernel = d3q19_sc_stage_kernel<float, false, 1, W>;
    float *buf = nullptr;
    cudaError_t e = cudaMalloc(&buf, sizeof(float) * 2 * 19 * N);
    if (e != cudaSuccess) return e;
    e = cudaMemset(buf, 0, sizeof(float) * 2 * 19 * N);
    D3Args a{};
    for (int k = 0; k < 19; k++) {
        a.src.f[k] = buf + (long)k * N;
        a.dst.f[k] = buf + (long)(19 + k) * N;
    }
    a.W = W; a.H = H; a.D = D; a.ndev = 1;
    a.tau_inv = 1.f; a.G = -5.f; a.psi_form = 1;
    a.err = err;
    static const cudaError_t attr_e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SS::SMEM);
    if (e == cudaSuccess) e = attr_e;
    if (e == cudaSuccess) {
        kernel<<<dim3(1, 1, 1), SS::THREADS, SS::SMEM>>>(a, D, 0, pair_constants(),
                                                         pair_d3<float>(a));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    cudaFree(buf);
    return e;
}

cudaError_t launch_d3q19_sc_stage(const D3Args &a, int storage, bool mom, cudaStream_t s) {
    if (!sc_stage_fits(a.W, a.H, a.D)) return cudaErrorInvalidValue;
    switch (storage) {
    case 0: return stage_launch<float>(a, mom, s);
    case 1: return stage_launch<__half>(a, mom, s);
    case 2: return stage_launch<__nv_bfloat16>(a, mom, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace lb
