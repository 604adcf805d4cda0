// kb_umma_roll.cuh -- convolutions and weight gradients of the warm-start
// network that walk down the rows of a pixel column, so that every input row
// is copied to shared memory once (engine 2, kb_umma_tma.cuh).
#pragma once
#include "kb_umma_tma.cuh"

namespace kb {
namespace umma {

// Convolution (forward or data gradient) rolling down the rows: layers of
// 128-pixel row tiles whose weights fit beside a ring of strips.  A row tile is 128
// pixels of one row; a CTA takes a contiguous range of row tiles, numbered
// down the rows of each 128-pixel column, and walks it.  Each input row is
// copied ONCE (one strip of 130 pixels per channel chunk) and feeds the three
// output rows it belongs to, which accumulate in a ring of four TMEM
// accumulators: row y is complete when row y + 1 has been read.  With one tile
// per row and three copies of every input row the ring of four CTAs per SM held
// a single tile, and bytes in flight over latency bound the layer (32 channels,
// 256^2, batch 16: 50 us against 20 us of HBM traffic).  The batch-16 256^2
// network: inference 734 -> 674 us, gradient 2482 -> 2383 us.
// The three kernel rows of a tap share one MMA: their weight blocks lie one
// after another in shared memory (kernel rows 2, 1, 0) and their output rows in
// neighbouring accumulators, bn columns apart, so an N of 3 bn reads the strip
// once where three MMAs read it three times (an MMA of N = 32 is bound by
// reading its 4 KB A operand).  The ring splits a run where it wraps, the row
// that starts from 0 is a run of its own on the first tap, and N stops at 256.
// The 96-channel decoder layer's forward 95 -> 73 us, the 32-channel layers 2 to
// 5 us less; inference 671 -> 642 us, gradient 2335 -> 2310 us.
// The epilogue reads 16 TMEM columns per wait.  A lane is a pixel, so an access
// of a warp touches up to 32 lines whatever its width, and the load-store unit
// bounds the epilogue: masks and outputs move 32 bytes per access (the 96-channel
// data gradient 120 -> 92 us, 32 -> 32 channels forward 36 -> 31; inference 640 ->
// 607 us, gradient 2255 -> 2171).  The ReLU mask of a row is loaded while the
// accumulator is still being computed, with more than 32 columns one row ahead
// (2171 -> 2155 us; with four CTAs per SM there are no registers for it).
struct ConvRoll : ConvStore {
    CUtensorMap x1, x2, w;
    int e, c1, C, H, W, nck;
    int rows;                          // row tiles: images x W / 128 x H
    uint32_t strip_bytes, tx;          // a ring stage: one chunk of one input row
    uint32_t res_bytes, tmem_cols;     // resident weights; TMEM columns of the accumulators, bn apart
    int ncols, cps;
};
constexpr int ROLL_ACC = 4;

// A CTA's range of row tiles as segments of one column: rows [ya, yb) of the
// column at pixel x0 of image b.
struct RollSegment {
    int r, r1, b, x0, ya, yb;
    __device__ __forceinline__ RollSegment(const ConvRoll &op)
        : r((int)((long long)op.rows * blockIdx.x / gridDim.x)),
          r1((int)((long long)op.rows * (blockIdx.x + 1) / gridDim.x)), b(0), x0(0), ya(0), yb(0) {}
    __device__ __forceinline__ bool next(const ConvRoll &op) {
        if (r >= r1) return false;
        const int nx = op.W / BM, col = r / op.H;
        ya = r - col * op.H;
        yb = min(op.H, ya + (r1 - r));
        b = col / nx;
        x0 = (col - b * nx) * BM;
        r += yb - ya;
        return true;
    }
};

// KK = e / 16 MMAs per tap and chunk; NQ 16-column groups per epilogue warp.
template <int KK, int NQ>
__global__ void __launch_bounds__(TM_THREADS, NQ == 1 ? 4 : (NQ == 2 ? 2 : 1))
    conv_roll_k(const __grid_constant__ ConvRoll op, const int nstages, int *__restrict__ err,
                const long long spin) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t stage_bytes = op.strip_bytes;
    const uint32_t res = base + (uint32_t)nstages * stage_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw + (base - raw) + (size_t)nstages * stage_bytes +
                                                  op.res_bytes);
    uint64_t *empty = full + nstages;
    uint64_t *acc_full = empty + nstages, *acc_empty = acc_full + ROLL_ACC, *drain = acc_empty + ROLL_ACC;
    uint64_t *resbar = drain + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(resbar + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t cols = (uint32_t)op.bn;

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(op.tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < nstages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < ROLL_ACC; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 128 * TM_EPI);
        }
        mbar_init(drain, 1);
        mbar_init(resbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    RollSegment seg(op);

    if (warp == 0) {
        // ---------------------------------------------------------- producer
        if (elect_one()) {
            prefetch_map(&op.x1);
            if (op.c1 < op.C) prefetch_map(&op.x2);
            prefetch_map(&op.w);
            const uint32_t blk = (uint32_t)(op.bn * 32 * KK);
            expect_tx(smem_u32(resbar), op.res_bytes);
            // (dx, chunk) blocks of the kernel rows 2, 1, 0, one after another
            for (int j = 0; j < 9 * op.nck; ++j) {
                const int k = j % 3, g = j / 3, dx = g / op.nck, ci = g - dx * op.nck;
                tma2(res + (uint32_t)j * blk, &op.w, (((2 - k) * 3 + dx) * op.nck + ci) * 16 * KK, 0, smem_u32(resbar));
            }
        }
        long long g = 0;
        int s = 0;
        uint32_t par = 0;
        while (ok && seg.next(op)) {
            for (int t = seg.ya - 1; t <= seg.yb && ok; ++t)
                for (int ci = 0; ci < op.nck; ++ci, ++g) {
                    if (g >= nstages && !(ok = mbar_wait_warp(&empty[s], par ^ 1u, spin))) break;
                    if (elect_one()) {
                        const uint32_t bar = smem_u32(&full[s]), sa = base + (uint32_t)s * stage_bytes;
                        const int c = ci * 16 * KK;
                        expect_tx(bar, op.tx);
                        if (c < op.c1) tma4(sa, &op.x1, c, seg.x0 - 1, t, seg.b, bar);
                        else tma4(sa, &op.x2, c - op.c1, seg.x0 - 1, t, seg.b, bar);
                    }
                    if (++s == nstages) {
                        s = 0;
                        par ^= 1u;
                    }
                }
        }
        // the copies issued have all landed before the CTA leaves
        for (long long i = 0; i < g && i < nstages; ++i) {
            if (s == 0) {
                s = nstages;
                par ^= 1u;
            }
            --s;
            if (!mbar_wait_warp(&full[s], par, spin)) ok = false;
        }
        if (!mbar_wait_warp(resbar, 0u, spin)) ok = false;
    } else if (warp == 1) {
        // ---------------------------------------------------------- MMA issue
        const uint32_t idesc1 = idesc_bf16(op.bn, false, false), idesc_step = idesc_bf16(2 * op.bn, false, false) - idesc1;
        const int gmax = 256 / op.bn;
        constexpr uint32_t S = 32u * KK, row = S / 16u;
        const uint32_t blk = (uint32_t)op.bn * row;
        const Desc bw = desc_k(res, S);
        int s = 0, nb = 0;  // nb: row tiles of earlier segments
        uint32_t par = 0;
        ok = mbar_wait_warp(resbar, 0u, spin);
        while (ok && seg.next(op)) {
            for (int t = seg.ya - 1; t <= seg.yb && ok; ++t) {
                const int n = nb + t - seg.ya;  // accumulator use of output row t
                if (t + 1 < seg.yb && n + 1 >= ROLL_ACC) {
                    const int u = n + 1;
                    if (!(ok = mbar_wait_warp(&acc_empty[u % ROLL_ACC], (uint32_t)((u / ROLL_ACC - 1) & 1), spin)))
                        break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                for (int ci = 0; ci < op.nck; ++ci) {
                    if (!(ok = mbar_wait_warp(&full[s], par, spin))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
                        const Desc a = desc_k(base + (uint32_t)s * stage_bytes, S);
                        // kernel row 2 - o feeds output row t - 1 + o; rows in
                        // neighbouring accumulators share one MMA
                        const int o0 = max(0, seg.ya - t + 1), o1 = min(2, seg.yb - t);
#pragma unroll
                        for (int dx = 0; dx < 3; ++dx)
                            for (int o = o0; o <= o1;) {
                                const int slot = (n - 1 + o) % ROLL_ACC;
                                const bool first = dx == 0 && ci == 0;  // row t + 1 starts from 0
                                const int run = min(min((first && o < 2 ? min(o1, 1) : o1) + 1 - o, ROLL_ACC - slot), gmax);
                                mma_run<KK>(tmem + (uint32_t)slot * cols, a, (uint32_t)dx * row, 2u, bw,
                                            (uint32_t)((dx * op.nck + ci) * 3 + o) * blk, 2u, idesc1 + (uint32_t)(run - 1) * idesc_step,
                                            first && o == 2 ? 0u : 1u);
                                o += run;
                            }
                        mma_commit(&empty[s]);
                        if (ci == op.nck - 1 && t - 1 >= seg.ya) mma_commit(&acc_full[(n - 1) % ROLL_ACC]);
                    }
                    __syncwarp();
                    if (++s == nstages) {
                        s = 0;
                        par ^= 1u;
                    }
                }
            }
            nb += seg.yb - seg.ya;
        }
        // every MMA issued above is complete once this commit arrives
        if (elect_one()) mma_commit(drain);
        if (!mbar_wait_warp(drain, 0u, spin)) ok = false;
    } else {
        // ---------------------------------------------------------- epilogue
        const int q = warp & 3, grp = (warp - 2) >> 2;
        const int px = q * 32 + lane;
        int n = 0;
        // the ReLU mask of the warp's columns at pixel x of row y
        auto load_mask = [&](int x, int y, uint32_t (*mk)[8]) {
            const int up = op.mask.up1;
            const size_t m = ((size_t)seg.b * op.H + y) * op.W + x;
            const __nv_bfloat16 *m1 =
                op.mask.s1 + (((size_t)seg.b * (op.H >> up) + (y >> up)) * (op.W >> up) + (x >> up)) * op.mask.c1;
            const __nv_bfloat16 *m2 = op.mask.s2 ? op.mask.s2 + m * op.mask.c2 - op.mask.c1 : m1;
#pragma unroll
            for (int g = 0; g < NQ; ++g) {
                const int c16 = g * 16 * TM_EPI + grp * 16;
                if (c16 < op.ncols) ld32(mk[g], (c16 < op.mask.c1 ? m1 : m2) + c16);
            }
        };
        uint32_t mk[NQ][8], next[NQ][8];
        while (ok && seg.next(op))
            for (int y = seg.ya; y < seg.yb; ++y, ++n) {
                const int x = seg.x0 + px;
                const size_t m = ((size_t)seg.b * op.H + y) * op.W + x;
                if (op.mask.s1) {
                    if (NQ == 1 || y == seg.ya) {
                        load_mask(x, y, mk);
                    } else {
#pragma unroll
                        for (int k = 0; k < NQ; ++k)
#pragma unroll
                            for (int i = 0; i < 8; ++i) mk[k][i] = next[k][i];
                    }
                    if (NQ > 1 && y + 1 < seg.yb) load_mask(x, y + 1, next);
                }
                if (!(ok = mbar_wait_warp(&acc_full[n % ROLL_ACC], (uint32_t)((n / ROLL_ACC) & 1), spin))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tacc = tmem + (uint32_t)(n % ROLL_ACC) * cols + ((uint32_t)(q * 32) << 16);
#pragma unroll
                for (int g = 0; g < NQ; ++g) {
                    const int c16 = g * 16 * TM_EPI + grp * 16;
                    if (c16 >= op.ncols) break;
                    float v[16];
                    tmem_ld16(tacc + (uint32_t)c16, v);
                    if (op.bias) {
#pragma unroll
                        for (int i = 0; i < 16; i += 4) {
                            const float4 b4 = __ldg(reinterpret_cast<const float4 *>(op.bias + c16 + i));
                            v[i] += b4.x; v[i + 1] += b4.y; v[i + 2] += b4.z; v[i + 3] += b4.w;
                        }
                    }
                    if (op.relu)
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.f);
                    if (op.mask.s1)
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const uint32_t w = mk[g][i >> 1];
                            const float f = __uint_as_float((i & 1) ? (w & 0xffff0000u) : (w << 16));
                            if (!(f > 0.f)) v[i] = 0.f;
                        }
                    if (op.out_f32) {
#pragma unroll
                        for (int i = 0; i < 16; i += 4) {
                            if (op.store_cols && c16 + i >= op.store_cols) break;
                            *reinterpret_cast<float4 *>((float *)op.out + m * op.Nout + c16 + i) =
                                make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                        }
                    } else {
                        uint32_t o[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                            o[i] = *reinterpret_cast<const uint32_t *>(&h);
                        }
                        st32((__nv_bfloat16 *)op.out + m * op.Nout + c16, o);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(&acc_empty[n % ROLL_ACC]);
            }
    }
    if (!ok) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(op.tmem_cols));
}

// Weight gradient of rows that are a multiple of 64 pixels wide, rolling down
// the rows: a CTA takes one group of channel chunks and a contiguous range of
// 64-pixel steps, numbered down the rows of each 64-pixel column, and keeps the
// gradient rows r = tap C + c of its chunks (and the bias row) in TMEM.  A ring
// stage holds the strips of input row t (one per chunk: pixels x-1 .. x+sr-2,
// box ea x sr, MN-major, swizzle 2ea) and the output gradient of row t + 1 (nb
// blocks of eb channels x 64 pixels); the step of input row t multiplies its
// strips with the output gradients of rows t - 1, t and t + 1 (kernel rows 2, 1
// and 0) from the last three stages, so a row of either is copied once, not once
// per kernel row (17 -> 9 KB per step at 32 channels, and four or five stages
// where two fitted).  The three output gradients are one operand of N = 3 bn
// (its blocks lie a stage apart; two MMAs where the ring wraps, and on the first
// rows, where a kernel row starts from 0 beside one that adds): with an MMA per
// kernel row each read the 4 KB strip again, which bounds an MMA of N = 32 (32
// channels 51 -> 41 us, 96 -> 32 channels 130 -> 94, the gradient 2069 -> 2011).
// An M-tile (chunk, h) reads its strip with the blocks one row apart (LBO = 2ea
// bytes): block j is the strip shifted by j pixels, i.e. tap dx = 2h - 1 + j
// (blocks of taps beyond +1 are computed and not stored).  The bias M-tile reads
// the resident `ones` rows (1 in channel 0).  Columns [(3 (chunk mtp + h) + 2 -
// kernel row) bn, + bn) hold a tile's kernel row, the last bn the bias.
// 64-channel chunks take this form too, with one CTA per SM: per-tap boxes
// (WgradTma) copy 120 KB per step there, this form 17 KB.  The whole gradient
// of the batch-16 256^2 network: 2382 -> 2340 us.
struct WgradRoll {
    CUtensorMap x1, x2, ones, dy;
    float *part;  // [splits][9C + 1][Nout]
    int bn, ea, eb, c1, C, H, W, Nout, nsteps;
    int cpt, mtp, nb, nmt, ea_shift, bn_shift;  // chunks per CTA, M-tiles per strip (1, 2), dY blocks, strip M-tiles
    uint32_t strip_bytes, tx;                    // a strip in the stage, and as copied
    uint32_t stage_bytes, res_bytes, acc_cols;
    int ncols, cps, groups, splits;              // CTAs: chunk group fastest

    __device__ void store(int row, int col, const float *v, const uint3 &t) const {
        const int m = col >> bn_shift, n = col & (bn - 1);
        const int R = 9 * C;
        int r;
        if (m == nmt) {
            if (row != 0 || t.x != 0) return;
            r = R;
        } else {
            const int st = m / 3, dyi = 2 - (m - 3 * st);
            const int cl = mtp == 2 ? (st >> 1) : st, h = st - cl * mtp, ci = (int)t.x * cpt + cl;
            const int j = row >> ea_shift, c = row & (ea - 1);
            const int dx = 2 * h - 1 + j;
            if (dx > 1) return;
            r = (dyi * 3 + dx + 1) * C + ci * ea + c;
        }
        st32(part + ((size_t)t.z * (R + 1) + r) * Nout + n, v);
    }
};

__global__ void __launch_bounds__(TM_THREADS, TM_MAX_CPS)
    wgrad_roll_k(const __grid_constant__ WgradRoll op, const int nstages, int *__restrict__ err,
                 const long long spin) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t stage_bytes = op.stage_bytes;
    const uint32_t res = base + (uint32_t)nstages * stage_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw + (base - raw) + (size_t)nstages * stage_bytes +
                                                  op.res_bytes);
    uint64_t *empty = full + nstages;
    uint64_t *acc_full = empty + nstages, *resbar = acc_full + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(resbar + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t cols = op.acc_cols;

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < nstages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(resbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    const int grp = (int)blockIdx.x % op.groups, z = (int)blockIdx.x / op.groups;
    const int nx = op.W / BK;
    const int r0 = (int)((long long)op.nsteps * z / op.splits), r1 = (int)((long long)op.nsteps * (z + 1) / op.splits);

    if (warp == 0) {
        // ---------------------------------------------------------- producer
        if (elect_one()) {
            prefetch_map(&op.x1);
            if (op.c1 < op.C) prefetch_map(&op.x2);
            prefetch_map(&op.ones);
            prefetch_map(&op.dy);
            expect_tx(smem_u32(resbar), op.res_bytes);
            tma2(res, &op.ones, 0, 0, smem_u32(resbar));
        }
        const int cg = grp * op.cpt * op.ea;  // first channel of the chunk group
        const uint32_t txs = (uint32_t)(op.cpt) * op.tx, txd = (uint32_t)(op.bn * BK * 2);
        const uint32_t dyo = (uint32_t)op.cpt * op.strip_bytes;
        long long g = 0;
        int s = 0;
        uint32_t par = 0;
        for (int r = r0; r < r1 && ok;) {
            const int col = r / op.H, ya = r - col * op.H, yb = min(op.H, ya + (r1 - r));
            const int b = col / nx, x0 = (col - b * nx) * BK;
            r += yb - ya;
            for (int t = ya - 1; t <= yb; ++t, ++g) {
                if (g >= nstages && !(ok = mbar_wait_warp(&empty[s], par ^ 1u, spin))) break;
                if (elect_one()) {
                    const uint32_t bar = smem_u32(&full[s]), sa = base + (uint32_t)s * stage_bytes;
                    expect_tx(bar, txs + (t + 1 < yb ? txd : 0u));
                    for (int ci = 0, c = cg; ci < op.cpt; ++ci, c += op.ea) {
                        const uint32_t dst = sa + (uint32_t)ci * op.strip_bytes;
                        if (c < op.c1) tma4(dst, &op.x1, c, x0 - 1, t, b, bar);
                        else tma4(dst, &op.x2, c - op.c1, x0 - 1, t, b, bar);
                    }
                    if (t + 1 < yb)
                        for (int j = 0; j < op.nb; ++j)
                            tma4(sa + dyo + (uint32_t)(j * 128 * op.eb), &op.dy, j * op.eb, x0, t + 1, b, bar);
                }
                if (++s == nstages) {
                    s = 0;
                    par ^= 1u;
                }
            }
        }
        // the copies issued have all landed before the CTA leaves
        for (long long i = 0; i < g && i < nstages; ++i) {
            if (s == 0) {
                s = nstages;
                par ^= 1u;
            }
            --s;
            if (!mbar_wait_warp(&full[s], par, spin)) ok = false;
        }
        if (!mbar_wait_warp(resbar, 0u, spin)) ok = false;
    } else if (warp == 1) {
        // ---------------------------------------------------------- MMA issue
        const uint32_t idesc1 = idesc_bf16(op.bn, true, true), idesc_step = idesc_bf16(2 * op.bn, true, true) - idesc1;
        const int gmax = op.nb == 1 ? 256 / op.bn : 1;
        const uint32_t sA = 2u * (uint32_t)op.ea, sB = 2u * (uint32_t)op.eb;
        const uint32_t strip = op.strip_bytes >> 4, half = sA >> 3;  // 2 sA bytes
        const uint32_t dyo = (uint32_t)op.cpt * op.strip_bytes, lbo = op.nb == 1 ? stage_bytes : 64u * sB;
        const Desc ones = desc_sw(res, sA, 8u * sA, sA);
        int s = 0, s1 = 0, s2 = 0;  // this stage's slot and the two before
        uint32_t par = 0, begun = 0;  // begun: kernel rows (bit 2 - row) and bias (bit 3) that hold a sum
        ok = mbar_wait_warp(resbar, 0u, spin);
        for (int r = r0; r < r1 && ok;) {
            const int col = r / op.H, ya = r - col * op.H, yb = min(op.H, ya + (r1 - r));
            r += yb - ya;
            for (int t = ya - 1; t <= yb; ++t) {
                if (!(ok = mbar_wait_warp(&full[s], par, spin))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // input row t meets output rows t - 1 + o, kernel row 2 - o
                const int o0 = max(0, ya - t + 1), o1 = min(2, yb - t);
                if (elect_one()) {
                    const Desc a = desc_sw(base + (uint32_t)s * stage_bytes, sA, 8u * sA, sA);
                    uint32_t was = begun;
                    for (int o = o0; o <= o1;) {
                        const int slot = o == 0 ? s2 : (o == 1 ? s1 : s);
                        const uint32_t on = was >> o & 1u;
                        int run = 1;
                        while (o + run <= o1 && run < gmax && slot + run < nstages && (was >> (o + run) & 1u) == on) ++run;
                        const Desc b = desc_sw(base + (uint32_t)slot * stage_bytes + dyo, lbo, 8u * sB, sB);
                        const uint32_t idesc = idesc1 + (uint32_t)(run - 1) * idesc_step;
                        uint32_t accm = tmem + (uint32_t)(o * op.bn), a0 = 0;
                        for (int ci = 0; ci < op.cpt; ++ci, a0 += strip)
                            for (int h = 0; h < op.mtp; ++h, accm += (uint32_t)(3 * op.bn))
                                mma_run<BK / 16>(accm, a, a0 + (uint32_t)h * half, sA, b, 0u, sB, idesc, on);
                        o += run;
                    }
                    if (grp == 0 && t + 1 < yb)
                        mma_run<BK / 16>(tmem + (uint32_t)(op.nmt * op.bn), ones, 0u, sA,
                                         desc_mn(base + (uint32_t)s * stage_bytes + dyo, sB), 0u, sB, idesc1, was >> 3);
                    if (t > ya) mma_commit(&empty[s2]);
                    if (t == yb) {
                        mma_commit(&empty[s1]);
                        mma_commit(&empty[s]);
                    }
                }
                __syncwarp();
                for (int o = o0; o <= o1; ++o) begun |= 1u << o;
                if (t + 1 < yb) begun |= 8u;
                s2 = s1;
                s1 = s;
                if (++s == nstages) {
                    s = 0;
                    par ^= 1u;
                }
            }
        }
        // every MMA issued above is complete once this commit arrives
        if (elect_one()) mma_commit(acc_full);
        if (!mbar_wait_warp(acc_full, 0u, spin)) ok = false;
    } else {
        // ---------------------------------------------------------- epilogue
        const int q = warp & 3, eg = (warp - 2) >> 2;
        const int row = q * 32 + lane;
        const uint3 t = make_uint3((unsigned)grp, 0u, (unsigned)z);
        ok = mbar_wait_warp(acc_full, 0u, spin);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (ok)
            for (int c0 = eg * 16; c0 < op.ncols; c0 += 16 * TM_EPI) {
                float v[16];
                tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
                op.store(row, c0, v, t);
                op.store(row, c0 + 8, v + 8, t);
            }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    if (!ok) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}

// ---------------------------------------------------------------- host side
inline int launch_wgrad_roll(const WgradRoll &w, int *err, cudaStream_t stream, long long spin = 1ll << 22) {
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(wgrad_roll_k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)TM_SMEM_MAX);
        if (e != cudaSuccess) return kb::check_launch("wgrad_roll_k: shared-memory attribute");
        configured[dev] = true;
    }
    const int ns = tma_stages(w.stage_bytes, w.res_bytes, w.cps);
    if (ns < 4 || w.cps < 1 || (uint32_t)w.cps * w.acc_cols > 512u || w.splits < 1 || w.splits > w.nsteps)
        return kb::set_error(KB_ERR_ARG, "wgrad_roll_k: shape does not fit");
    wgrad_roll_k<<<(unsigned)(w.groups * w.splits), TM_THREADS,
                   tma_smem_bytes(ns, w.stage_bytes, w.res_bytes), stream>>>(w, ns, err, spin);
    return 0;
}

// Ring stages and shared memory of a rolling convolution with cps CTAs per SM.
inline int roll_stages(const ConvRoll &c, int cps) { return tma_stages(c.strip_bytes, c.res_bytes, cps); }
inline size_t roll_smem_bytes(const ConvRoll &c, int ns) {
    return 1024 + (size_t)ns * c.strip_bytes + c.res_bytes + (size_t)(2 * ns + 2 * ROLL_ACC + 2) * 8 + 16;
}
// Most CTAs per SM whose four accumulators fit TMEM together, whose ring holds
// two strips and whose epilogue registers fit; 0 if the weights leave no ring.
inline int roll_fit(const ConvRoll &c) {
    const int nq = (c.ncols + 31) / 32, most = nq == 1 ? 4 : (nq == 2 ? 2 : 1);
    for (int k = most; k >= 1; --k)
        if ((uint32_t)k * c.tmem_cols <= 512u && roll_stages(c, k) >= 2) return k;
    return 0;
}

template <int KK, int NQ>
int launch_roll_t(const ConvRoll &c, int *err, cudaStream_t stream, long long spin) {
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(conv_roll_k<KK, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)TM_SMEM_MAX);
        if (e != cudaSuccess) return kb::check_launch("conv_roll_k: shared-memory attribute");
        configured[dev] = true;
    }
    const int ns = roll_stages(c, c.cps);
    const int slots = kb::sm_count() * c.cps, ctas = c.rows < slots ? c.rows : slots;
    conv_roll_k<KK, NQ><<<(unsigned)ctas, TM_THREADS, roll_smem_bytes(c, ns), stream>>>(c, ns, err, spin);
    return 0;
}

inline int launch_roll(const ConvRoll &c, int *err, cudaStream_t stream, long long spin = 1ll << 22) {
    const int nq = (c.ncols + 31) / 32;
    if (c.cps < 1 || c.cps > TM_MAX_CPS || roll_stages(c, c.cps) < 2 || nq > 4 || c.rows < 1 ||
        (uint32_t)c.cps * c.tmem_cols > 512u || (uint32_t)(ROLL_ACC * c.bn) > c.tmem_cols)
        return kb::set_error(KB_ERR_ARG, "conv_roll_k: shape does not fit");
#define KB_ROLL(KK)                                                                          \
    do {                                                                                     \
        if (nq == 1) return launch_roll_t<KK, 1>(c, err, stream, spin);                      \
        if (nq == 2) return launch_roll_t<KK, 2>(c, err, stream, spin);                      \
        if (nq == 3) return launch_roll_t<KK, 3>(c, err, stream, spin);                      \
        return launch_roll_t<KK, 4>(c, err, stream, spin);                                   \
    } while (0)
    if (c.e == 64) KB_ROLL(4);
    if (c.e == 32) KB_ROLL(2);
    KB_ROLL(1);
#undef KB_ROLL
}

}  // namespace umma
}  // namespace kb
