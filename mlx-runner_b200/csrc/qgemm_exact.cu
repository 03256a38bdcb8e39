// Prefill GEMM for sm_100a that rounds no operand to fp16's 11 bits or range: Y[T, O] = X[T, K] . W[O, K]^T, any MLX bit
// width, fp32 / fp16 / bf16 activations of any magnitude, scales, biases and sums over groups in fp32.
//
// What it replaces: batches whose weights or activations may not be rounded to fp16 (everything but 4-bit layers with
// 16-bit activations) ran eight or sixteen tokens at a time on the token-major decode kernel, or on the CUDA cores when
// the rows were too long for it -- the whole layer was read and unpacked again for every eight tokens.
//
// Operands.  The A operand is the raw codes, centred: q - 2^(bits-1) is exact in fp16, and unpacking costs three to five
// instructions per pair of codes.  fp16 activations are the B operand as they are; bf16 and fp32 ones are scaled by a
// power of two per token first, which the stored outputs undo, and are then one fp16 number and two (x = x1 + x2): one or
// two tcgen05 products per term.  The products of one quantisation group -- 64 codes, or 32
// where the group is that short -- accumulate in fp32 in tensor memory; then every thread adds
// scale * sum + (bias + scale * 2^(bits-1)) * (sum of the group's activations) to fp32 accumulators in its registers.
// (Folding scale and bias into an A operand of two fp16 numbers needs no such drain, but tcgen05 cuts every sum off
// below about 2^-25 of the accumulator, always towards zero: over 1024 products that came to 1.2e-6 of the result,
// against 1.8e-7 here.)
//
// Tile: 128 rows x up to 128 tokens, K in stages of 64.  The codes are the A operand in tensor memory, written by four
// unpacking warps, one per lane quadrant: a lane owns a row, its warp fetches the 32 rows' packed bytes of a stage with
// warp-private cp.async copies, eight stages ahead, into rows padded so that the lanes' reads meet no bank twice.  The
// activations are the B operand, fetched by TMA with the 128-byte swizzle.  Three accumulators in tensor memory take the
// drain steps in turn; sixteen draining warps own a lane quadrant and a quarter of the tile's tokens each.  (With the
// same sixteen warps unpacking by turns and draining, every step waited for the group that was unpacking.)  One warp
// issues the MMAs with its lanes together and one lane elected for the instruction itself: from a branch that only lane 0
// takes, an MMA costs 110 cycles to issue, here 50.
//
// Split K.  A layer of few rows leaves most SMs without a tile, so K is cut into `S` segments worked on by different
// CTAs; the warp that finishes a piece of the tile last adds the segments' partial sums in their order.  S depends on
// the layer and the activations' type alone, not on the batch: a token's result is the same whatever batch it rides in.
// Measured (pre-pass included, one decode-kernel pass per eight tokens before): 12288 x 4096, 4 bits, 512 fp32 tokens
// 1398 -> 165 us (312 TFLOP/s counted once per term); 8 bits, 384 bf16 tokens 717 -> 121 us.  What bounds it now is the
// drain: 128 x 128 sums leave tensor memory per 64 codes, two packed FMAs per pair of them, some 1700 cycles a stage
// against 512 of the MMAs.
// Every wait is bounded: a wait that runs out sets the device error word, raises the CTA's abort flag and all roles
// fall through to the common exit, where tensor memory is released.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <mutex>

#include "dependent_launch.h"
#include "mlxq_device.cuh"
#include "qgemm_exact.cuh"
#include "qmv_pipe.cuh"
#include "sm100_ptx.cuh"

namespace mlxq {

namespace {

constexpr int BM = 128, BN_MAX = 128, BK = 64;
constexpr int S_X = 4;                         // activation stages
constexpr int S_A = 4;                         // tensor-memory stages of A
constexpr int S_D = 3;                         // accumulators
constexpr int S_W = 8;                         // stages of packed rows in flight per unpacking warp
constexpr int S_T = 8;                         // drain steps' scales, biases and activation sums in flight
constexpr int T_SLOT = BM * 8 + BN_MAX * 4;    // one step's: 1 KB of (scale, bias) pairs, up to 512 bytes of sums
constexpr int X_TILE = BN_MAX * BK * 2;        // 16 KB per part
constexpr int UNPACKERS = 4, WORKERS = 16;     // warps 0-3 unpack, 4-19 drain
constexpr int WORKER0 = UNPACKERS, X_PRODUCER = WORKER0 + WORKERS, MMA_WARP = X_PRODUCER + 1;
constexpr int NUM_THREADS = (MMA_WARP + 1) * 32;
constexpr int TMEM_COLS = 512;
constexpr int A_COL0 = S_D * BN_MAX;           // after the accumulators

// bytes of a row per stage, the padded pitch of such a row in shared memory, the copies' size
template <int BITS> struct Row {
    static constexpr int BYTES = BK * BITS / 8;
    static constexpr int PIECE = BYTES % 16 == 0 ? 16 : 8;
    static constexpr int PPR = BYTES / PIECE;                               // pieces per row = pieces per lane
    static constexpr int PITCH = BITS == 4 ? 48 : BITS == 8 ? 80 : BYTES;   // consecutive rows start in different banks
    static constexpr int SLOT = 32 * PITCH;
};

struct Barriers {
    uint64_t full_x[S_X];
    uint64_t empty_x[S_X];
    uint64_t full_a[S_A];
    uint64_t empty_a[S_A];
    uint64_t d_full[S_D], d_empty[S_D];
    uint64_t full_t[S_T], empty_t[S_T];
    uint32_t tmem_base;
    int abort_flag;
};

template <int BITS, int XS> constexpr int smem_bytes() {
    return S_X * XS * X_TILE + UNPACKERS * S_W * Row<BITS>::SLOT + S_T * T_SLOT + static_cast<int>(sizeof(Barriers)) + 1024;
}

struct ExactArgs {
    const uint8_t* w;
    const void* bias;
    void* y;
    unsigned* err;
    const float2* table;        // [group][o_pad] (scale, bias + scale * 2^(bits-1))
    const float* xsum;          // [drain step][t_pad] sums of the activations
    const float* unscale;       // [t_pad] the inverse of each token's power of two
    float* partial;             // [tile][segment][token][row of the tile] (S > 1)
    unsigned* counters;         // [tile][draining warp] (S > 1)
    long long y_stride;
    int bias_dtype, y_dtype;
    int O, K, gs_shift, T;
    int m_tiles, n_tiles, S, t_pad;
    int steps_shift;            // log2(drain steps per stage): 1 for groups of 32, else 0
    uint32_t idesc;
};

__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFF) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr) : "memory");
}

template <int BYTES> __device__ __forceinline__ void cp_piece(uint32_t dst, const void* src) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
// two fp32 FMAs: d += a * b
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }

// code J of a row's stage in the low bits of the result (with other codes' bits above it)
template <int BITS, int J>
__device__ __forceinline__ uint32_t code_at(const uint32_t (&w)[2 * BITS]) {
    constexpr int bit = J * BITS, word = bit / 32, off = bit % 32;
    if constexpr (off + BITS > 32) return __funnelshift_r(w[word], w[word + 1 < 2 * BITS ? word + 1 : word], off);
    else return w[word] >> off;
}

// Registers I0 ... I0 + 15 of a row's stage: pairs of codes as fp16 numbers minus 2^(bits-1).  A code is or'ed into the
// mantissa of 1024.  Pair I is codes (2I, 2I + 1); at 4 bits the codes (i, i + 4) of each eight, which one mask picks out
// of a word -- the activations are staged in the matching order 0,4,1,5,2,6,3,7.
template <int BITS, int I0, int I = 0>
__device__ __forceinline__ void code_pairs(const uint32_t (&w)[2 * BITS], uint32_t (&v)[16]) {
    if constexpr (I < 16) {
        constexpr int P = I0 + I;
        uint32_t u;
        if constexpr (BITS == 4) {
            u = ((w[P / 4] >> (4 * (P % 4))) & 0x000F000Fu) | 0x64006400u;
        } else if constexpr (BITS == 8) {
            u = __byte_perm(w[P / 2], 0x64646464u, (P & 1) ? 0x4342 : 0x4140);
        } else {
            constexpr uint32_t mask = (1u << BITS) - 1u;
            u = (__byte_perm(code_at<BITS, 2 * P>(w), code_at<BITS, 2 * P + 1>(w), 0x5410) & (mask | (mask << 16))) | 0x64006400u;
        }
        const __half2 c = __float2half2_rn(1024.0f + static_cast<float>(1 << (BITS - 1)));
        const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&u), c);
        v[I] = *reinterpret_cast<const uint32_t*>(&h);
        code_pairs<BITS, I0, I + 1>(w, v);
    }
}

// XS: fp16 parts per activation (1 for 16-bit activations, 2 for fp32).  NC: tokens per draining warp, a quarter of the tile.
template <int BITS, int XS, int NC>
__global__ void __launch_bounds__(NUM_THREADS, 1)
qgemm_exact_kernel(const __grid_constant__ CUtensorMap map_x, const ExactArgs a) {
    using R = Row<BITS>;
    constexpr int BN = 4 * NC;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* x_tiles = smem;                                                  // S_X x XS x 16 KB
    uint8_t* w_ring = smem + S_X * XS * X_TILE;
    uint8_t* t_ring = w_ring + UNPACKERS * S_W * R::SLOT;
    Barriers* bars = reinterpret_cast<Barriers*>(t_ring + S_T * T_SLOT);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int k_stages = a.K / BK;
    const int total = a.m_tiles * a.n_tiles * a.S;
    const int spst = 1 << a.steps_shift;
    // unit u: row tiles vary fastest (CTAs running together share activation tiles in L2), then segments, then tokens
    auto seg_of = [&](int u) { return (u / a.m_tiles) % a.S; };
    auto k_begin = [&](int seg) { return k_stages * seg / a.S; };

    if (threadIdx.x == 0) {
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        for (int i = 0; i < S_X; i++) { mbar_init(&bars->full_x[i], 1); mbar_init(&bars->empty_x[i], 1); }
        for (int i = 0; i < S_A; i++) { mbar_init(&bars->full_a[i], UNPACKERS); mbar_init(&bars->empty_a[i], 1); }
        for (int i = 0; i < S_D; i++) { mbar_init(&bars->d_full[i], 1); mbar_init(&bars->d_empty[i], WORKERS); }
        for (int i = 0; i < S_T; i++) { mbar_init(&bars->full_t[i], 1); mbar_init(&bars->empty_t[i], WORKERS); }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base), 0);

    // (the unpacking warps do not wait for the pre-pass, which lets this grid start when all before it is complete)
    if (warp >= WORKER0) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (warp == X_PRODUCER) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_x)) : "memory");
            uint32_t it = 0, step = 0;
            bool ok = true;
            constexpr uint32_t bytes = BN * (BK * 2) * XS, t_bytes = BM * 8 + BN * 4;
            const int o_pad = a.m_tiles * BM;
            for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
                const int seg = seg_of(u), tok0 = u / (a.m_tiles * a.S) * BN, row0 = (u % a.m_tiles) * BM;
                const int k1 = k_begin(seg + 1);
                for (int ks = k_begin(seg); ok && ks < k1; ks++, it++) {
                    const int s = it % S_X;
                    if (it >= S_X && !mbar_wait(&bars->empty_x[s], ((it / S_X) - 1) & 1, &bars->abort_flag, a.err)) { ok = false; break; }
                    mbar_expect_tx(&bars->full_x[s], bytes);
                    tma_load_2d(x_tiles + s * (XS * X_TILE), &map_x, &bars->full_x[s], ks * BK, tok0);
                    // (the second parts are the rows T ... 2T - 1 of the staged array)
                    if constexpr (XS == 2) tma_load_2d(x_tiles + s * (XS * X_TILE) + X_TILE, &map_x, &bars->full_x[s], ks * BK, a.T + tok0);
                    for (int j = 0; j < spst; j++, step++) {
                        const int sl = step % S_T, st = (ks << a.steps_shift) + j;
                        if (step >= S_T && !mbar_wait(&bars->empty_t[sl], ((step / S_T) - 1) & 1, &bars->abort_flag, a.err)) { ok = false; break; }
                        mbar_expect_tx(&bars->full_t[sl], t_bytes);
                        bulk_load(t_ring + sl * T_SLOT, a.table + static_cast<size_t>((st * (BK >> a.steps_shift)) >> a.gs_shift) * o_pad + row0, BM * 8, &bars->full_t[sl]);
                        bulk_load(t_ring + sl * T_SLOT + BM * 8, a.xsum + static_cast<size_t>(st) * a.t_pad + tok0, BN * 4, &bars->full_t[sl]);
                    }
                    if (!ok) { it++; break; }
                }
            }
            // see every copy this thread issued land (bounded) before the CTA may exit
            for (uint32_t j = it > S_X ? it - S_X : 0; j < it; j++) {
                const uint64_t t0 = global_ns();
                while (!mbar_try_wait(&bars->full_x[j % S_X], (j / S_X) & 1))
                    if (global_ns() - t0 > WAIT_NS) break;
            }
            for (uint32_t j = step > S_T ? step - S_T : 0; j < step; j++) {
                const uint64_t t0 = global_ns();
                while (!mbar_try_wait(&bars->full_t[j % S_T], (j / S_T) & 1))
                    if (global_ns() - t0 > WAIT_NS) break;
            }
        }
    } else if (warp == MMA_WARP) {
        // ---- MMA issuer: the warp's lanes stay together, one is elected for the instructions -----------------------------
        uint32_t it = 0, buf = 0, d_phase = 1;                  // (the first turn of every accumulator waits for nothing)
        bool ok = true;
        const uint64_t x_desc = desc_sw128(smem_u32(x_tiles));
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            const int seg = seg_of(u), n = k_begin(seg + 1) - k_begin(seg);
            for (int i = 0; ok && i < n; i++, it++) {
                const uint32_t s = it % S_X, sa = it % S_A;
                const uint64_t x1 = x_desc + static_cast<uint64_t>(s * (XS * X_TILE / 16)), x2 = x1 + X_TILE / 16;
                const uint32_t a_addr = tmem + A_COL0 + sa * 32;
                for (int j = 0; j < spst; j++) {
                    if (!mbar_wait_three(&bars->d_empty[buf], d_phase, &bars->full_x[s], (it / S_X) & 1, &bars->full_a[sa], (it / S_A) & 1,
                                    &bars->abort_flag, a.err)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t d_addr = tmem + buf * BN_MAX;
                    if (elect_one()) {
                        if (spst == 1) {
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) {
                                tc_mma_ts(d_addr, a_addr + kk * 8, x1 + static_cast<uint64_t>(kk * 2), a.idesc, kk != 0);
                                if constexpr (XS == 2) tc_mma_ts(d_addr, a_addr + kk * 8, x2 + static_cast<uint64_t>(kk * 2), a.idesc, 1u);
                            }
                        } else {                                // half a stage: two K slices of 16
#pragma unroll
                            for (int kk = 0; kk < 2; kk++) {
                                tc_mma_ts(d_addr, a_addr + (2 * j + kk) * 8, x1 + static_cast<uint64_t>((2 * j + kk) * 2), a.idesc, kk != 0);
                                if constexpr (XS == 2) tc_mma_ts(d_addr, a_addr + (2 * j + kk) * 8, x2 + static_cast<uint64_t>((2 * j + kk) * 2), a.idesc, 1u);
                            }
                        }
                        tc_commit(&bars->d_full[buf]);
                        if (j == spst - 1) {
                            tc_commit(&bars->empty_x[s]);
                            tc_commit(&bars->empty_a[sa]);
                        }
                    }
                    __syncwarp();
                    if (++buf == S_D) { buf = 0; d_phase ^= 1; }
                }
            }
        }
    } else if (warp < UNPACKERS) {
        // ---- unpacking warps: a lane quadrant's 32 rows of every stage ----------------------------------------------------
        const int quad = warp;
        const size_t row_bytes = static_cast<size_t>(a.K) * BITS / 8;
        const uint32_t ring = smem_u32(w_ring + quad * (S_W * R::SLOT));
        const uint32_t a_base = tmem + (static_cast<uint32_t>(quad * 32) << 16) + A_COL0;
        // the copy stream: (unit, stage) pairs in order, S_W of them in flight
        int l_u = blockIdx.x, l_left = 0;
        const uint8_t* l_src[R::PPR];
        uint32_t l_dst[R::PPR];
#pragma unroll
        for (int m = 0; m < R::PPR; m++) {
            const int pc = lane + 32 * m, rr = pc / R::PPR, part = pc - rr * R::PPR;
            l_dst[m] = ring + rr * R::PITCH + part * R::PIECE;
            l_src[m] = nullptr;
        }
        auto enter = [&]() {                                    // the cursor moves to unit l_u
            const int seg = seg_of(l_u), k0 = k_begin(seg);
            l_left = k_begin(seg + 1) - k0;
#pragma unroll
            for (int m = 0; m < R::PPR; m++) {
                const int pc = lane + 32 * m, rr = pc / R::PPR, part = pc - rr * R::PPR;
                const int row = min((l_u % a.m_tiles) * BM + quad * 32 + rr, a.O - 1);   // rows past the end read a valid row; never stored
                l_src[m] = a.w + static_cast<size_t>(row) * row_bytes + static_cast<size_t>(k0) * R::BYTES + part * R::PIECE;
            }
        };
        auto issue = [&](uint32_t slot_off) {
            if (l_u < total) {
#pragma unroll
                for (int m = 0; m < R::PPR; m++) {
                    cp_piece<R::PIECE>(l_dst[m] + slot_off, l_src[m]);
                    l_src[m] += R::BYTES;
                }
                if (--l_left == 0) {
                    l_u += gridDim.x;
                    if (l_u < total) enter();
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        enter();                                                // (the grid has no more CTAs than units)
        for (int i = 0; i < S_W; i++) issue(i * R::SLOT);
        uint32_t it = 0, slot = 0;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            const int seg = seg_of(u), n = k_begin(seg + 1) - k_begin(seg);
            for (int i = 0; i < n; i++, it++) {
                asm volatile("cp.async.wait_group %0;" ::"n"(S_W - 1) : "memory");
                __syncwarp();                                   // (a lane's row was copied by several lanes)
                const uint32_t src = ring + slot + lane * R::PITCH, sa = it % S_A;
                uint32_t wd[2 * BITS];
#pragma unroll
                for (int m = 0; m < R::PPR; m++) {
                    if constexpr (R::PIECE == 16)
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(wd[4 * m]), "=r"(wd[4 * m + 1]), "=r"(wd[4 * m + 2]), "=r"(wd[4 * m + 3]) : "r"(src + 16 * m));
                    else
                        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(wd[2 * m]), "=r"(wd[2 * m + 1]) : "r"(src + 8 * m));
                }
                uint32_t v[16], v2[16];
                code_pairs<BITS, 0>(wd, v);
                code_pairs<BITS, 16>(wd, v2);
                __syncwarp();                                   // every lane has read the slot
                issue(slot);
                slot = slot == (S_W - 1) * R::SLOT ? 0 : slot + R::SLOT;
                if (it >= S_A && !mbar_wait_warp(&bars->empty_a[sa], ((it / S_A) - 1) & 1, &bars->abort_flag, a.err)) { ok = false; break; }
                __syncwarp();
                tc_fence_after();
                tc_st16(a_base + sa * 32, v);
                tc_st16(a_base + sa * 32 + 16, v2);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->full_a[sa]);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
        // ---- draining warps: a lane quadrant's 32 rows x a quarter of the tokens ---------------------------------------------
        const int dw = warp - WORKER0, par = dw >> 2;
        const int quad = warp & 3;                              // tensor-memory lane quadrant this warp may touch
        const uint32_t base = tmem + (static_cast<uint32_t>(quad * 32) << 16) + par * NC;
        uint32_t buf = 0, d_phase = 0, step = 0;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            const int m_tile = u % a.m_tiles, seg = seg_of(u);
            const int trow = quad * 32 + lane, row = m_tile * BM + trow;
            const int n_tile = u / (a.m_tiles * a.S), tok0 = n_tile * BN + par * NC;
            const float unscale = lane < NC ? __ldcg(a.unscale + tok0 + lane) : 0.0f;     // lane c: token c of this warp's
            uint64_t acc[NC / 2];
#pragma unroll
            for (int i = 0; i < NC / 2; i++) acc[i] = 0ull;
            const int n = (k_begin(seg + 1) - k_begin(seg)) << a.steps_shift;
            for (int i = 0; i < n; i++, step++) {
                // the step's scales, biases and sums (copied by the producer, far ahead), then its products
                const uint32_t sl = step % S_T;
                const uint8_t* ts = t_ring + sl * T_SLOT;
                if (!mbar_wait_both(&bars->full_t[sl], (step / S_T) & 1, &bars->d_full[buf], d_phase, &bars->abort_flag, a.err)) { ok = false; break; }
                tc_fence_after();
                uint32_t d[NC];
#pragma unroll
                for (int c = 0; c < NC; c += 8) tc_ld8(base + buf * BN_MAX + c, d + c);
                const float2 sb = *reinterpret_cast<const float2*>(ts + trow * 8);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->d_empty[buf]);
                if (++buf == S_D) { buf = 0; d_phase ^= 1; }
                const uint64_t s2 = pack2(sb.x, sb.x), b2 = pack2(sb.y, sb.y);
                const float4* xv = reinterpret_cast<const float4*>(ts + BM * 8) + par * (NC / 4);
#pragma unroll
                for (int c = 0; c < NC; c += 4) {
                    const float4 x4 = xv[c / 4];
                    fma2(acc[c / 2], s2, pack2(__uint_as_float(d[c]), __uint_as_float(d[c + 1])));
                    fma2(acc[c / 2 + 1], s2, pack2(__uint_as_float(d[c + 2]), __uint_as_float(d[c + 3])));
                    fma2(acc[c / 2], b2, pack2(x4.x, x4.y));
                    fma2(acc[c / 2 + 1], b2, pack2(x4.z, x4.w));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->empty_t[sl]);
            }
            if (!ok) break;

            // ---- the unit is done: this warp's 32 rows x NC tokens ----------------------------------------------------------
            const float rb = (a.bias != nullptr && row < a.O) ? load_scalar(a.bias, a.bias_dtype, row) : 0.0f;
            auto store = [&](int c, float v) {
                const int tok = tok0 + c;
                const float u = __shfl_sync(0xffffffffu, unscale, c);
                if (row < a.O && tok < a.T) store_scalar(a.y, a.y_dtype, static_cast<size_t>(tok) * a.y_stride + row, fmaf(v, u, rb));
            };
            if (a.S == 1) {
#pragma unroll
                for (int i = 0; i < NC / 2; i++) {
                    float f0, f1;
                    unpack2(acc[i], f0, f1);
                    store(2 * i, f0);
                    store(2 * i + 1, f1);
                }
            } else {
                // partial sums to memory; the warp that is last among the segments' CTAs for this piece of the tile adds
                // them up, in the order of the segments
                const int tile = n_tile * a.m_tiles + m_tile;
                const size_t seg_step = static_cast<size_t>(BN) * BM;
                float* part = a.partial + static_cast<size_t>(tile) * a.S * seg_step + static_cast<size_t>(par * NC) * BM + trow;
#pragma unroll
                for (int i = 0; i < NC / 2; i++) {
                    float f0, f1;
                    unpack2(acc[i], f0, f1);
                    __stcg(part + seg * seg_step + static_cast<size_t>(2 * i) * BM, f0);
                    __stcg(part + seg * seg_step + static_cast<size_t>(2 * i + 1) * BM, f1);
                }
                __threadfence();
                __syncwarp();
                unsigned before = 0;
                if (lane == 0) before = atomicInc(a.counters + tile * WORKERS + par * 4 + quad, static_cast<unsigned>(a.S - 1));
                before = __shfl_sync(0xffffffffu, before, 0);
                if (before == static_cast<unsigned>(a.S - 1)) {
                    __threadfence();
                    float f[NC];
#pragma unroll
                    for (int i = 0; i < NC; i++) f[i] = __ldcg(part + static_cast<size_t>(i) * BM);
#pragma unroll 1
                    for (int sg = 1; sg < a.S; sg++)
#pragma unroll
                        for (int i = 0; i < NC; i++) f[i] += __ldcg(part + sg * seg_step + static_cast<size_t>(i) * BM);
#pragma unroll
                    for (int i = 0; i < NC; i++) store(i, f[i]);
                }
                __syncwarp();
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ---- the pre-pass: activations -> fp16 parts and their sums per drain step, scales and biases -> the table by row, the
// counters -> 0 -----------------------------------------------------------------------------------------------------------
struct ExactStage {
    const void* x; int x_dtype; long long x_stride; __half* xs; int T, K, xs_parts, permuted;
    float* xsum; int t_pad, step_chunks;     // chunks of eight activations per drain step: 8 or 4
    float* unscale;                          // [t_pad] what a token's outputs are multiplied by
    const void* s; const void* b; int s_dtype; int s_vec; int O, o_pad, groups; float centre; float2* table;
    unsigned* counters; int n_counters;
    unsigned x_blocks;
};

// Activations are scaled by a power of two per token (token_scale_exponent): unscaled, one of 1e5 became infinity, and fp32
// ones of 1e-4 kept 13 of their 24 bits.  fp16 activations are what they are: factor one.
constexpr int STAGE_THREADS = 256;
constexpr int STAGE_KEEP = 6;                // chunks of a thread that stay in registers between the two passes: 12288 codes

__global__ void __launch_bounds__(STAGE_THREADS) exact_stage_kernel(const ExactStage g) {
    asm volatile("griddepcontrol.wait;" ::: "memory");           // a dependent of the previous kernel; what that wrote is read through L2
    // The GEMM may start now and not before: it reads packed weights without a wait of its own, and everything ahead in the
    // stream, which may have written them, is complete here.
    if (threadIdx.x == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (blockIdx.x < g.x_blocks) {
        // a block per token: the largest magnitude first, then the parts
        __shared__ float warp_max[STAGE_THREADS / 32];
        const int chunks = g.K / 8;                              // a multiple of 16
        const int lane = threadIdx.x & 31;
        for (int t = blockIdx.x; t < g.T; t += g.x_blocks) {
            const size_t row = static_cast<size_t>(t) * g.x_stride;
            float kept[STAGE_KEEP][8], largest = 0.0f;
#pragma unroll
            for (int k = 0; k < STAGE_KEEP; k++) {
                const int c = k * STAGE_THREADS + threadIdx.x;
                if (c < chunks) load8_coherent(g.x, g.x_dtype, row + c * 8, kept[k]);
            }
            float factor = 1.0f, inverse = 1.0f;
            if (g.x_dtype != DT_F16) {
#pragma unroll
                for (int k = 0; k < STAGE_KEEP; k++)
                    if (k * STAGE_THREADS + static_cast<int>(threadIdx.x) < chunks)
#pragma unroll
                        for (int j = 0; j < 8; j++) largest = fmaxf(largest, fabsf(kept[k][j]));
                for (int c = STAGE_KEEP * STAGE_THREADS + threadIdx.x; c < chunks; c += STAGE_THREADS) {
                    float v[8];
                    load8_coherent(g.x, g.x_dtype, row + c * 8, v);
#pragma unroll
                    for (int j = 0; j < 8; j++) largest = fmaxf(largest, fabsf(v[j]));
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, o));
                __syncthreads();                                 // (the previous token's maxima have been read)
                if (lane == 0) warp_max[threadIdx.x >> 5] = largest;
                __syncthreads();
#pragma unroll
                for (int w = 0; w < STAGE_THREADS / 32; w++) largest = fmaxf(largest, warp_max[w]);
                const uint32_t e = token_scale_exponent(largest);
                factor = __uint_as_float(e << 23);
                inverse = __uint_as_float((254u - e) << 23);
            }
            if (threadIdx.x == 0) g.unscale[t] = inverse;
            // one chunk of eight; whole warps come here together: the sums are formed by 4 or 8 lanes, which are live together
            auto emit = [&](int c, const float (&v)[8], bool live) {
                float sum = 0.0f, f[8];
#pragma unroll
                for (int j = 0; j < 8; j++) { f[j] = v[j] * factor; sum += f[j]; }
                for (int o = 1; o < g.step_chunks; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (!live) return;
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float p = g.permuted ? f[j] : f[2 * j], q = g.permuted ? f[j + 4] : f[2 * j + 1];
                    const __half2 h = __floats2half2_rn(p, q);
                    const float2 b = __half22float2(h);
                    const __half2 l = __floats2half2_rn(p - b.x, q - b.y);
                    hi[j] = *reinterpret_cast<const uint32_t*>(&h);
                    lo[j] = *reinterpret_cast<const uint32_t*>(&l);
                }
                __half* out = g.xs + static_cast<size_t>(t) * g.K + c * 8;
                *reinterpret_cast<uint4*>(out) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                if (g.xs_parts == 2) *reinterpret_cast<uint4*>(out + static_cast<size_t>(g.T) * g.K) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                if ((c & (g.step_chunks - 1)) == 0) g.xsum[static_cast<size_t>(c / g.step_chunks) * g.t_pad + t] = sum;
            };
#pragma unroll
            for (int k = 0; k < STAGE_KEEP; k++)
                if (k * STAGE_THREADS < chunks) {
                    const int c = k * STAGE_THREADS + threadIdx.x;
                    emit(c, kept[k], c < chunks);
                }
            for (int c0 = STAGE_KEEP * STAGE_THREADS; c0 < chunks; c0 += STAGE_THREADS) {
                const int c = c0 + threadIdx.x;
                float v[8] = {};
                if (c < chunks) load8_coherent(g.x, g.x_dtype, row + c * 8, v);
                emit(c, v, c < chunks);
            }
        }
        return;
    }
    const unsigned block = blockIdx.x - g.x_blocks, blocks = gridDim.x - g.x_blocks;
    for (int i = block * 256 + threadIdx.x; i < g.n_counters; i += blocks * 256) g.counters[i] = 0u;
    // eight groups of a row per thread, rows in consecutive threads
    const int row_chunks = (g.groups + 7) / 8;
    const long long n = static_cast<long long>(row_chunks) * g.o_pad;
    for (long long i = block * 256ll + threadIdx.x; i < n; i += blocks * 256ll) {
        const int row = static_cast<int>(i % g.o_pad), g0 = static_cast<int>(i / g.o_pad) * 8;
        const size_t at = static_cast<size_t>(min(row, g.O - 1)) * g.groups + g0;
        float s[8], b[8];
        if (g.s_vec) {
            if (g.s_dtype == DT_F16) {
                XLoad<__half>::load8(static_cast<const __half*>(g.s) + at, s);
                XLoad<__half>::load8(static_cast<const __half*>(g.b) + at, b);
            } else {
                XLoad<__nv_bfloat16>::load8(static_cast<const __nv_bfloat16*>(g.s) + at, s);
                XLoad<__nv_bfloat16>::load8(static_cast<const __nv_bfloat16*>(g.b) + at, b);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++) {
                s[k] = g0 + k < g.groups ? load_scalar(g.s, g.s_dtype, at + k) : 0.0f;
                b[k] = g0 + k < g.groups ? load_scalar(g.b, g.s_dtype, at + k) : 0.0f;
            }
        }
        // (rows past the end hold the last row's values; what is computed from them is never stored)
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (g0 + k < g.groups) g.table[static_cast<size_t>(g0 + k) * g.o_pad + row] = make_float2(s[k], fmaf(s[k], g.centre, b[k]));
    }
}

template <int BITS, int XS, int NC>
cudaError_t launch_one(const CUtensorMap& map_x, const ExactArgs& a, int device, int grid, cudaStream_t st) {
    static_assert(smem_bytes<BITS, XS>() <= 227 * 1024, "shared memory of a CTA");
    // the shared-memory opt-in is an attribute of the function in one device's context
    static std::mutex mu;
    static bool done[64] = {};
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!done[device]) {
            const cudaError_t e = cudaFuncSetAttribute(qgemm_exact_kernel<BITS, XS, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<BITS, XS>());
            if (e != cudaSuccess) return e;
            done[device] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = smem_bytes<BITS, XS>();
    cfg.stream = st;
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;          // a dependent of the pre-pass
    la[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = la;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, qgemm_exact_kernel<BITS, XS, NC>, map_x, a);
}

template <int BITS, int XS>
cudaError_t launch_nc(int bn, const CUtensorMap& map_x, const ExactArgs& a, int device, int grid, cudaStream_t st) {
    if (bn <= 32) return launch_one<BITS, XS, 8>(map_x, a, device, grid, st);
    if (bn <= 64) return launch_one<BITS, XS, 16>(map_x, a, device, grid, st);
    return launch_one<BITS, XS, 32>(map_x, a, device, grid, st);
}

template <int XS>
cudaError_t launch_bits(int bits, int bn, const CUtensorMap& map_x, const ExactArgs& a, int device, int grid, cudaStream_t st) {
    switch (bits) {
        case 2: return launch_nc<2, XS>(bn, map_x, a, device, grid, st);
        case 3: return launch_nc<3, XS>(bn, map_x, a, device, grid, st);
        case 4: return launch_nc<4, XS>(bn, map_x, a, device, grid, st);
        case 5: return launch_nc<5, XS>(bn, map_x, a, device, grid, st);
        case 6: return launch_nc<6, XS>(bn, map_x, a, device, grid, st);
        case 8: return launch_nc<8, XS>(bn, map_x, a, device, grid, st);
        default: return cudaErrorNotSupported;
    }
}

size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

// Segments of K: the count that leaves the busiest CTA the least to do on one tile of tokens, from the layer alone (a
// unit's fixed cost is about six stages; a segment keeps eight stages or more), but no fewer than `least`.  Never from the
// device or the batch: the order of the sums must not change with them.
int segments(int m_tiles, int k_stages, int least) {
    constexpr int SMS = 148;
    int best = least;
    long long best_cost = -1;
    for (int s = least; s == least || (s <= 8 && k_stages / s >= 8); s++) {
        const long long waves = (static_cast<long long>(m_tiles) * s + SMS - 1) / SMS;
        const long long cost = waves * ((k_stages + s - 1) / s + 6);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = s; }
    }
    return best;
}

// With 16-bit activations the products are exact and the roundings of the running sum are what is left; they grow with its
// length, and the kernels that serve such calls otherwise have shorter sums.  So that the error is not above theirs:
// * 8-bit rows of more than 8192 codes, the CUDA-core kernel's: segments of 24 drain steps at most, 16 of them at most.  In
//   sums of 48 and 96 steps the error was 1.34e-7 and 1.82e-7 of the result (12288 codes in groups of 64 and 32), in sums of
//   24 it is 1.1e-7 and 1.2e-7, there 1.2e-7.  (4096 x 12288 with 384 bf16 tokens: 125 -> 150 us in groups of 64, 206 -> 252
//   in groups of 32.)
// * 6 and 8 bits in groups of 32: 64 steps.  (14336 x 4096 in sums of 128 2.1e-7, of 64 1.5e-7; the token-major kernel 1.7e-7.)
int least_segments(const GemmLayer& L, int parts) {
    if (L.bits < 6 || parts != 1) return 1;
    const int steps = L.K / (L.gs == 32 ? 32 : BK), limit = L.bits == 8 && L.K > 8192 ? 24 : L.gs == 32 ? 64 : steps;
    const int s = (steps + limit - 1) / limit;
    return s < 16 ? s : 16;
}

constexpr long long SLICE_BYTES = 96ll << 20;          // scratch of one slice of tokens, about

}  // namespace

bool qgemm_exact_takes(const GemmLayer& L, int x_dtype, long long x_stride, const void* x, long long T) {
    if (T < 17 || T > 0x7FFFFFFFLL || L.O < 1) return false;
    if (L.bits != 2 && L.bits != 3 && L.bits != 4 && L.bits != 5 && L.bits != 6 && L.bits != 8) return false;
    if (L.gs != 32 && L.gs != 64 && L.gs != 128) return false;
    if (L.s_dtype != DT_F16 && L.s_dtype != DT_BF16) return false;
    if (L.K % 128 != 0) return false;
    if ((reinterpret_cast<uintptr_t>(L.w) & 15u) != 0 || (reinterpret_cast<uintptr_t>(x) & 15u) != 0) return false;
    return (x_stride * dtype_size(x_dtype)) % 16 == 0;
}

cudaError_t launch_qgemm_exact(const GemmLayer& L, const GemmCall& c, cudaStream_t st, const char** why) {
    *why = "";
    const int parts = c.x_dtype == DT_F32 ? 2 : 1;
    ExactArgs a = {};
    a.w = L.w; a.bias = L.bias; a.err = c.err;
    a.y_stride = c.y_stride; a.bias_dtype = L.bias_dtype; a.y_dtype = c.y_dtype;
    a.O = L.O; a.K = L.K;
    while ((1 << a.gs_shift) < L.gs) a.gs_shift++;
    a.steps_shift = L.gs == 32 ? 1 : 0;
    a.m_tiles = (L.O + BM - 1) / BM;
    a.S = segments(a.m_tiles, L.K / BK, least_segments(L, parts));
    const int steps = (L.K / BK) << a.steps_shift, groups = L.K / L.gs, o_pad = a.m_tiles * BM;
    // Long batches run in slices of tokens, so that the scratch memory stays bounded whatever the batch.
    const long long per_token = static_cast<long long>(L.K) * 2 * parts + 4ll * steps + (a.S > 1 ? 4ll * a.S * o_pad : 0);
    long long slice = SLICE_BYTES / per_token / BN_MAX * BN_MAX;
    if (slice < BN_MAX) slice = BN_MAX;
    if (slice > c.T) slice = c.T;
    const int bn = slice <= 32 ? 32 : slice <= 64 ? 64 : BN_MAX;
    const long long n_tiles = (slice + bn - 1) / bn;
    a.t_pad = static_cast<int>(n_tiles) * bn;
    const size_t x_b = align256(static_cast<size_t>(slice) * L.K * 2 * parts), tab_b = align256(static_cast<size_t>(groups) * o_pad * sizeof(float2));
    const size_t sum_b = align256(static_cast<size_t>(steps) * a.t_pad * 4), un_b = align256(static_cast<size_t>(a.t_pad) * 4);
    const size_t ctr_b = a.S > 1 ? align256(static_cast<size_t>(n_tiles) * a.m_tiles * WORKERS * 4) : 0;
    const size_t part_b = a.S > 1 ? static_cast<size_t>(n_tiles) * a.m_tiles * a.S * bn * BM * 4 : 0;
    cudaMemPool_t pool = gemm_scratch_pool(L.device);
    if (!pool) { *why = "scratch pool"; return cudaErrorMemoryAllocation; }
    uint8_t* scratch = nullptr;
    if (cudaMallocFromPoolAsync(reinterpret_cast<void**>(&scratch), x_b + tab_b + sum_b + un_b + ctr_b + part_b, pool, st) != cudaSuccess) {
        cudaGetLastError();
        *why = "scratch allocation";
        return cudaErrorMemoryAllocation;
    }
    __half* xs = reinterpret_cast<__half*>(scratch);
    float2* table = reinterpret_cast<float2*>(scratch + x_b);
    float* xsum = reinterpret_cast<float*>(scratch + x_b + tab_b);
    a.table = table;
    a.xsum = xsum;
    float* unscale = reinterpret_cast<float*>(scratch + x_b + tab_b + sum_b);
    a.unscale = unscale;
    a.counters = reinterpret_cast<unsigned*>(scratch + x_b + tab_b + sum_b + un_b);
    a.partial = reinterpret_cast<float*>(scratch + x_b + tab_b + sum_b + un_b + ctr_b);
    // fp32 accumulate, A and B fp16, both K-major, N = bn, M = 128
    a.idesc = (1u << 4) | (static_cast<uint32_t>(bn >> 3) << 17) | (static_cast<uint32_t>(BM >> 4) << 24);
    cudaError_t err = cudaSuccess;
    for (long long t0 = 0; t0 < c.T && err == cudaSuccess; t0 += slice) {
        const int T = static_cast<int>(c.T - t0 < slice ? c.T - t0 : slice);
        a.T = T;
        a.n_tiles = (T + bn - 1) / bn;
        a.y = static_cast<char*>(c.y) + static_cast<size_t>(t0) * c.y_stride * dtype_size(c.y_dtype);
        ExactStage g = {};
        g.x = static_cast<const char*>(c.x) + static_cast<size_t>(t0) * c.x_stride * dtype_size(c.x_dtype);
        g.x_dtype = c.x_dtype; g.x_stride = c.x_stride; g.xs = xs; g.T = T; g.K = L.K; g.xs_parts = parts; g.permuted = L.bits == 4;
        g.xsum = xsum; g.unscale = unscale; g.t_pad = a.t_pad; g.step_chunks = 8 >> a.steps_shift;
        g.s = L.s; g.b = L.b; g.s_dtype = L.s_dtype; g.O = L.O; g.o_pad = o_pad; g.groups = groups;
        g.s_vec = groups % 8 == 0 && ((reinterpret_cast<uintptr_t>(L.s) | reinterpret_cast<uintptr_t>(L.b)) & 15u) == 0;
        g.centre = static_cast<float>(1 << (L.bits - 1)); g.table = table;
        g.counters = a.counters; g.n_counters = a.S > 1 ? a.n_tiles * a.m_tiles * WORKERS : 0;
        const long long ns = (static_cast<long long>((groups + 7) / 8) * o_pad + 255) / 256;
        g.x_blocks = static_cast<unsigned>(T < 148 * 6 ? T : 148 * 6);
        cudaLaunchConfig_t sc = {};
        sc.gridDim = dim3(g.x_blocks + static_cast<unsigned>(ns < 148 * 4 ? ns : 148 * 4));
        sc.blockDim = dim3(STAGE_THREADS);
        sc.stream = st;
        cudaLaunchAttribute sa[1];
        sa[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        sa[0].val.programmaticStreamSerializationAllowed = 1;
        sc.attrs = sa;
        sc.numAttrs = pdl_enabled() ? 1 : 0;
        err = cudaLaunchKernelEx(&sc, exact_stage_kernel, g);
        if (err != cudaSuccess) { *why = "pre-pass"; break; }
        CUtensorMap map_x;
        if (!gemm_map_2d(&map_x, xs, static_cast<uint64_t>(L.K), static_cast<uint64_t>(T) * parts, static_cast<uint64_t>(L.K) * 2, BK, bn)) {
            *why = "tensor map of the activations";
            err = cudaErrorInvalidValue;
            break;
        }
        const long long units = static_cast<long long>(a.m_tiles) * a.n_tiles * a.S;
        const int sms = gemm_sm_count(L.device), grid = static_cast<int>(units < sms ? units : sms);
        err = parts == 2 ? launch_bits<2>(L.bits, bn, map_x, a, L.device, grid, st) : launch_bits<1>(L.bits, bn, map_x, a, L.device, grid, st);
        if (err != cudaSuccess) *why = "launch";
    }
    cudaFreeAsync(scratch, st);                        // stream-ordered: released after the last slice has read it
    return err;
}

}  // namespace mlxq
