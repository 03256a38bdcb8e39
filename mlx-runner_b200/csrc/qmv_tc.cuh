// Decode matvec for up to sixteen tokens on the fifth-generation tensor cores: raw codes as the A operand in tensor memory,
// the tokens as accumulator columns, scales and biases per group in fp32.
//
// What bounds the kernels on mma.sync (qmv_tok.cuh): an MMA of theirs covers sixteen rows, so every sixteen rows the batch's
// activations are read from shared memory again (two 128-bit loads per 1024 codes, eight columns and 32 codes of K), every CTA
// stages all of K of them, and a warp's turn of one group is one chain of waits, loads, MMAs and shuffles.  Here an MMA covers
// 128 rows, reads the activations once for all of them and its operands in no warp's registers (M = 128, N = 16, K = 16 takes
// nine cycles), and a CTA stages a slice of K.
//
// A CTA takes 128-row blocks and a slice of K.  Its parts:
// * four unpacking warps, a lane a row, fetch 32 packed rows each with warp-private cp.async copies, a stage of 128 codes a row
//   at a time and several ahead (no barrier to wait at: a wait for an mbarrier costs 150 cycles, a quarter of a stage), into
//   rows padded so that the lanes' reads meet no bank twice, and turn a stage into fp16 registers -- a code less
//   2^(bits-1); codes further up in their halves are undone by the staged activations (see qmv_mma.cuh, code_plan.cuh) -- and
//   store them to tensor memory.  (As subnormal numbers, q * 2^-24, which the mma.sync kernels multiply, the products lose
//   their low bits: the error was 1e-6 of the result at 4 bits, up to 1.7 times the token-major kernel's);
// * one warp issues the MMAs.  Every group of codes sums up in sixteen columns of its own; an fp32 token's activations are two
//   fp16 parts, multiplied into the same column one after the other;
// * four draining warps, a lane a row, add  (bias + 2^(bits-1) * scale) * (sum of the group's activations) + scale * sum  to
//   fp32 registers.  (With
//   eight of them, a group of a slot each, 24576 x 4096 at 4 bits with 6 fp32 tokens took 33 us and not 26: what waits, polls.)
// The activations of the slice are staged once per CTA, scaled by a power of two per token and group, so that any magnitude is
// served.
//
// K is cut into `kz` slices, worked on by the CTAs of a cluster: that gives layers of few rows enough CTAs, and a CTA's
// activations are few.  At the end of a block every CTA stores its sums into the shared memory of the CTA that finishes
// those rows, which adds them up in the order of the slices, a block later than it could, so that nobody waits.
//
// Two CTAs share an SM: one's waits are the other's turns, and the next launch of the stream can fetch its first stages
// while this one's last CTAs run.  (Never three: a CTA asks for 80 KB at the least.  And the library's other kernels that allocate
// tensor memory fill an SM's registers, so that no two launches wait for each other's.)  Every wait but the cluster's start and end
// is bounded: a wait that runs out sets the
// device error word and the CTA's abort flag, and all roles run on to the common exit.
#pragma once

#include "code_plan.cuh"
#include "qmv_pipe.cuh"
#include "sm100_ptx.cuh"

namespace mlxq {

constexpr int TC_STAGE = 128;                  // codes of a row per stage
constexpr int TC_DRAINERS = 4, TC_UNPACKERS = 4;                // warps (four each: warp w touches lane quadrant w % 4)
constexpr int TC_ISSUER = TC_DRAINERS + TC_UNPACKERS, TC_HELPER = TC_ISSUER + 1;     // (the helper stages activations and no more)
constexpr int TC_THREADS = (TC_HELPER + 1) * 32;
constexpr int TC_STAGERS = TC_THREADS - TC_UNPACKERS * 32;      // threads that stage the activations
constexpr int TC_TMEM = 256;                   // columns: two CTAs an SM
constexpr int TC_BN = 16;                      // MMA columns
constexpr int TC_GPS = 2;                      // groups per accumulator slot
constexpr int TC_SD = 2, TC_D_COLS = TC_GPS * TC_BN;            // accumulator slots
constexpr int TC_SA = 3, TC_A_COLS = TC_STAGE / 2;              // A slots
constexpr int TC_SMEM_TWO = 112 * 1024;         // shared memory of a CTA that leaves room for a second one
constexpr int TC_SMEM_WHOLE = 224 * 1024;      // of the 227 KB a CTA may opt into
static_assert(TC_SD * TC_D_COLS + TC_SA * TC_A_COLS <= TC_TMEM, "tensor memory");

// the batch (of two tokens or more) rounded up to the tokens a kernel is compiled for
__host__ __device__ constexpr int tc_tokens(int t) { return t <= 2 ? 2 : t <= 4 ? 4 : t <= 8 ? 8 : 16; }

// ... and whether it is compiled: 16-bit activations take the kernel from five tokens on, two fp32 tokens up to five bits
__host__ __device__ constexpr bool tc_compiled(int bits, int ntk, int split) { return split == 1 ? ntk >= 8 : ntk > 2 || bits <= 5; }

struct TcBarriers {
    uint64_t full_a[TC_SA], empty_a[TC_SA];
    uint64_t d_full[TC_SD], d_empty[TC_SD];
    uint64_t red_full[2], red_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};

struct TcPlan {
    int kz, kz_shift;        // CTAs (a cluster) that share a block along K
    int clusters;
    int n_blocks;            // blocks of 128 rows; part i of the layer starts at block first_block[i]
    int first_block[3];
    int first_row[3];        // ... and its rows in y
    int stages;              // K / 128
    int depth;               // stages in flight: 8, 6, 4 or 3
    int off_x, off_xsum, off_red, off_bars;
    int s_align;             // alignment of the scales' and biases' first rows: 16, 4 or 2 bytes
};

// bytes of a row per stage, and its pitch in shared memory: an odd number of 16-byte pieces
template <int BITS> struct TcRow {
    static constexpr int BYTES = TC_STAGE * BITS / 8, PIECES = BYTES / 16;
    static constexpr int PITCH = PIECES % 2 ? BYTES : BYTES + 16;
    static constexpr int WARP_SLOT = 32 * PITCH;
};
__host__ __device__ constexpr int tc_slot_bytes(int bits) { return TC_UNPACKERS * 32 * (TC_STAGE * bits / 8 + (bits % 2 ? 0 : 16)); }

// Register N of a run of 32 codes, holding codes q some places p up, as fp16 numbers (q - 2^(BITS-1)) * 2^p: the code is or'ed
// into the mantissa of 1024 (one instruction with the masking of it).
template <int BITS, int N> constexpr float tc_offset(int half) {
    if constexpr (planned_width<BITS>()) {
        constexpr CodePlan<BITS, 32> P{};
        return 1024.0f + static_cast<float>((1 << (BITS - 1)) << P.shl[half ? P.second[N] : P.first[N]]);
    } else {
        return 1024.0f + static_cast<float>((1 << (BITS - 1)) << (BITS == 4 ? (N & 1) * 4 : BITS == 2 ? (N & 3) * 2 : 0));
    }
}
template <int BITS, int N> __device__ __forceinline__ uint32_t tc_centred(uint32_t v) {
    constexpr float lo = tc_offset<BITS, N>(0), hi = tc_offset<BITS, N>(1);
    const uint32_t u = v | 0x64006400u;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&u), __floats2half2_rn(lo, hi));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// columns [taddr, taddr + N) of the warp's lanes
template <int N> __device__ __forceinline__ void tc_ld_cols(uint32_t taddr, uint32_t* v) {
    if constexpr (N == 2) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(taddr) : "memory");
    } else if constexpr (N == 4) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
    } else {
        static_assert(N % 8 == 0, "columns a load");
#pragma unroll
        for (int c = 0; c < N; c += 8)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(v[c]), "=r"(v[c + 1]), "=r"(v[c + 2]), "=r"(v[c + 3]), "=r"(v[c + 4]), "=r"(v[c + 5]), "=r"(v[c + 6]), "=r"(v[c + 7])
                         : "r"(taddr + c) : "memory");
    }
}

// pairs of fp32 numbers
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_store(uint32_t remote, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory"); }
// (a release at cluster scope: it waits for all that the thread has stored, to y too -- not to be done where nobody waits for it)
__device__ __forceinline__ void cluster_arrive(uint32_t remote_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
// Whole-warp waits by one polling lane (see mbar_wait_warp), whose outcome nothing depends on: when a wait runs out the error
// word and the abort flag are set, every later wait of the CTA returns at once, the loops run to their ends on whatever is
// there, and the host discards the result.
__device__ __forceinline__ void mbar_await_warp(uint64_t* bar, uint32_t parity, int* abort_flag, unsigned* err) {
    if ((threadIdx.x & 31) == 0) mbar_wait(bar, parity, abort_flag, err);
    __syncwarp();
}
// the same for a barrier that other CTAs of the cluster arrive at: acquires at cluster scope
static __device__ __noinline__ void mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* abort_flag, unsigned* err) {
    uint64_t t0 = 0;
    for (uint32_t n = 1;; n++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (ok) return;
        if ((n & 63u) != 0) continue;
        if (*reinterpret_cast<volatile int*>(abort_flag)) return;
        if (t0 == 0) t0 = global_ns();
        if (global_ns() - t0 > WAIT_NS) {
            *reinterpret_cast<volatile int*>(abort_flag) = 1;
            atomicOr(err, ERR_WAIT_TIMEOUT | ERR_GEMM_PIPELINE);
            return;
        }
    }
}
__device__ __forceinline__ void mbar_await_cluster_warp(uint64_t* bar, uint32_t parity, int* abort_flag, unsigned* err) {
    if ((threadIdx.x & 31) == 0) mbar_wait_cluster(bar, parity, abort_flag, err);
    __syncwarp();
}
// (relaxed: it orders no memory, only the CTAs' beginnings and ends; not the .aligned form: lanes may come here from loops of
// different lengths)
__device__ __forceinline__ void tc_cluster_barrier() {
    asm volatile("barrier.cluster.arrive.relaxed;\n\tbarrier.cluster.wait;" ::: "memory");
}

// Eight consecutive activations (k a multiple of eight, inside the slice) of a token into the staged tiles: 64 codes a row of
// 128 bytes, 16-byte pieces permuted by the 128-byte swizzle, in the order in which the unpacking warps lay the codes out.
// Two parts: the fp16 numbers nearest to them, and what those leave.
template <int BITS, int SPLIT>
__device__ __forceinline__ void tc_stage8(uint8_t* xs, int tile_bytes, int part_bytes, int tok, int k, const float (&v)[8]) {
    uint8_t* row = xs + (k >> 6) * tile_bytes + tok * 128;
    const int p = k & 63, sw = tok & 7;
    auto at = [&](int h) -> uint8_t* { return row + ((((h >> 3) ^ sw) << 4) | ((h & 7) * 2)); };
    if constexpr (planned_width<BITS>()) {
        const int u0 = p & 31, run = p & 32;
        plan_static_for<0, 32, 8>([&](auto uc) {
            constexpr int U0 = decltype(uc)::value;
            if (u0 == U0) {
                constexpr CodePlan<BITS, 32> P{};
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float w = v[i] * __int_as_float((127 - P.shl[U0 + i]) << 23);
                    const __half h = __float2half_rn(w);
                    uint8_t* to = at(run + P.pos[U0 + i]);
                    *reinterpret_cast<__half*>(to) = h;
                    if (SPLIT == 2) *reinterpret_cast<__half*>(to + part_bytes) = __float2half_rn(w - __half2float(h));
                }
            }
        });
    } else if constexpr (BITS == 2) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float w = v[i] * __int_as_float((127 - stage_shift<BITS>(i)) << 23);
            const __half h = __float2half_rn(w);
            uint8_t* to = at((p & ~15) + 2 * i + ((p >> 3) & 1));
            *reinterpret_cast<__half*>(to) = h;
            if (SPLIT == 2) *reinterpret_cast<__half*>(to + part_bytes) = __float2half_rn(w - __half2float(h));
        }
    } else {
        // pairs in the order of the A registers: 0,4 | 1,5 | 2,6 | 3,7 at 4 bits, 0,2 | 1,3 | 4,6 | 5,7 at 8
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int a = BITS == 4 ? i : (i >> 1) * 4 + (i & 1), b = BITS == 4 ? i + 4 : a + 2;
            constexpr int UW = MmaUnit<BITS>::UW;
            const float sc = __int_as_float((127 - stage_shift<BITS>(a % UW)) << 23);    // (the same for both of a pair)
            const float wa = v[a] * sc, wb = v[b] * sc;
            const __half2 h = __floats2half2_rn(wa, wb);
            hi[i] = *reinterpret_cast<const uint32_t*>(&h);
            if (SPLIT == 2) {
                const float2 r = __half22float2(h);
                const __half2 l = __floats2half2_rn(wa - r.x, wb - r.y);
                lo[i] = *reinterpret_cast<const uint32_t*>(&l);
            }
        }
        *reinterpret_cast<uint4*>(at(p)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if (SPLIT == 2) *reinterpret_cast<uint4*>(at(p) + part_bytes) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

// NTK: tokens a drain works for (the batch rounded up); SPLIT: fp16 parts per activation.
//
// The code is kept short on purpose: every role's loops are rolled and stand once.  A launch on a small layer works for 4 us, and
// what it runs through only once it waits for, line by line, at the instruction cache.
template <int BITS, int NTK, int SPLIT>
__global__ void __launch_bounds__(TC_THREADS, 2)
qmv_tc_kernel(const __grid_constant__ MmaParams p, const __grid_constant__ TcPlan tp) {
    using R = TcRow<BITS>;
    // 64 codes of the tokens' staged activations: eight or sixteen rows of 128 bytes per part.  (Eight: the MMA's second eight
    // columns are whatever lies behind them, the part or tile that follows, and nobody looks at their sums.)
    constexpr int X_PART = NTK <= 8 ? 1024 : 2048, X_TILE = SPLIT * X_PART;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const QmvParams& q = p.q;
    uint8_t* xs = smem + tp.off_x;
    float* xsum = reinterpret_cast<float*>(smem + tp.off_xsum);          // [group of the slice][2][NTK]: sums, inverse factors
    float* red = reinterpret_cast<float*>(smem + tp.off_red);            // [parity][source CTA][token][row of this CTA's share]
    TcBarriers* bars = reinterpret_cast<TcBarriers*>(smem + tp.off_bars);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, quad = warp & 3;
    const int T = q.T, gs_shift = q.gs_shift;
    const int kz = tp.kz, rank = blockIdx.x & (kz - 1), cid = blockIdx.x >> tp.kz_shift;
    const int s_begin = (tp.stages * rank) >> tp.kz_shift, ns = ((tp.stages * (rank + 1)) >> tp.kz_shift) - s_begin;
    const int k0 = s_begin * TC_STAGE, codes = ns * TC_STAGE;
    const int ng = codes >> gs_shift, g_begin = k0 >> gs_shift, groups = q.K >> gs_shift;
    const int my_blocks = cid < tp.n_blocks ? (tp.n_blocks - 1 - cid) / tp.clusters + 1 : 0;
    auto part_of = [&](int blk) { return q.n_parts > 2 && blk >= tp.first_block[2] ? 2 : q.n_parts > 1 && blk >= tp.first_block[1] ? 1 : 0; };
    uint32_t tmem = 0;
    // the CTA's (and the cluster's) barriers and tensor memory are set up
    auto ready = [&]() {
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (kz > 1) tc_cluster_barrier();
        tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base), 0);
    };

    if (warp >= TC_DRAINERS && warp < TC_ISSUER) {
        // ---- unpacking warps: a lane quadrant's 32 rows of every stage; (block, stage) pairs in order ---------------------
        const int total = my_blocks * ns;
        const size_t row_bytes = static_cast<size_t>(q.K) * BITS / 8;
        const uint32_t ring = smem_u32(smem) + quad * (tp.depth * R::WARP_SLOT), ring_end = ring + tp.depth * R::WARP_SLOT;
        int f_left = total, f_s = ns, f_blk = cid;              // the copies' cursor
        const uint8_t* f_src[R::PIECES];
        uint32_t slot = ring, sa = 0, a_phase = 1, a_base = 0;  // (the first turn of every A slot waits for nothing)
#pragma unroll 1
        for (int it = -tp.depth; it < total; it++) {            // (the first `depth` turns only fetch)
            if (it >= 0) {
                if (it == 0) {
                    ready();
                    a_base = tmem + (static_cast<uint32_t>(quad * 32) << 16) + TC_SD * TC_D_COLS;
                }
                // (the first turns fill the A slots ahead of the previous launch's end; from here on the others are at work or soon will be)
                if (it == TC_SA) asm volatile("griddepcontrol.wait;" ::: "memory");
                if (tp.depth == 8) asm volatile("cp.async.wait_group 7;" ::: "memory");
                else if (tp.depth == 6) asm volatile("cp.async.wait_group 5;" ::: "memory");
                else if (tp.depth == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
                else asm volatile("cp.async.wait_group 2;" ::: "memory");
                __syncwarp();                                   // (a lane's row was copied by several lanes)
                const uint32_t src = slot + lane * R::PITCH;
                constexpr bool BY_RUN = BITS == 8;              // (registers: the whole stage's words at once where they are few)
                uint32_t wd[BY_RUN ? BITS : 4 * R::PIECES];
                auto words = [&](int first, int n) {            // 16-byte pieces
#pragma unroll
                    for (int c = 0; c < n; c++)
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                     : "=r"(wd[4 * c]), "=r"(wd[4 * c + 1]), "=r"(wd[4 * c + 2]), "=r"(wd[4 * c + 3]) : "r"(src + 16 * (first + c)));
                };
                if constexpr (!BY_RUN) words(0, R::PIECES);
                mbar_await_warp(&bars->empty_a[sa], a_phase, &bars->abort_flag, p.err);
                tc_fence_after();
                static_for<0, 4, 1>([&](auto rc) {
                    constexpr int run = decltype(rc)::value;    // 32 codes: BITS words, sixteen registers
                    if constexpr (BY_RUN) words(run * (BITS / 4), BITS / 4);
                    uint32_t v[16];
                    static_for<0, 8, 1>([&](auto jc) {
                        constexpr int j = decltype(jc)::value;
                        a_regs_run<BITS, 32, j>(wd + (BY_RUN ? 0 : run * BITS), v[2 * j], v[2 * j + 1]);
                        v[2 * j] = tc_centred<BITS, 2 * j>(v[2 * j]);
                        v[2 * j + 1] = tc_centred<BITS, 2 * j + 1>(v[2 * j + 1]);
                    });
                    tc_st16(a_base + sa * TC_A_COLS + run * 16, v);
                });
                __syncwarp();                                   // every lane has read the slot
            }
            if (f_left > 0) {
                if (f_s == ns) {                                // the first stage of a block
                    const int pi = part_of(f_blk), row0 = (f_blk - tp.first_block[pi]) * 128 + quad * 32;
                    const uint8_t* w = q.part[pi].w + static_cast<size_t>(s_begin) * R::BYTES;
#pragma unroll
                    for (int m = 0; m < R::PIECES; m++) {
                        const int pc = lane + 32 * m, rr = pc / R::PIECES;      // rows past the end read a valid row; never stored
                        f_src[m] = w + static_cast<size_t>(min(row0 + rr, q.part[pi].rows - 1)) * row_bytes + (pc - rr * R::PIECES) * 16;
                    }
                    f_s = 0;
                    f_blk += tp.clusters;
                }
#pragma unroll
                for (int m = 0; m < R::PIECES; m++) {
                    const int pc = lane + 32 * m, rr = pc / R::PIECES;
                    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(slot + rr * R::PITCH + (pc - rr * R::PIECES) * 16), "l"(f_src[m]) : "memory");
                    f_src[m] += R::BYTES;
                }
                f_left--;
                f_s++;
            }
            cp_commit();
            slot += R::WARP_SLOT;
            if (slot == ring_end) slot = ring;
            if (it >= 0) {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->full_a[sa]);
                if (++sa == TC_SA) { sa = 0; a_phase ^= 1; }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
        if (threadIdx.x == TC_ISSUER * 32) {
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            for (int i = 0; i < TC_SA; i++) { mbar_init(&bars->full_a[i], TC_UNPACKERS); mbar_init(&bars->empty_a[i], 1); }
            for (int i = 0; i < TC_SD; i++) { mbar_init(&bars->d_full[i], 1); mbar_init(&bars->d_empty[i], TC_DRAINERS); }
            // (full: from every CTA the warps with rows of this CTA's share)
            for (int i = 0; i < 2; i++) { mbar_init(&bars->red_full[i], kz > 4 ? kz : 4); mbar_init(&bars->red_empty[i], TC_DRAINERS * kz); }
            bars->abort_flag = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        if (warp == TC_HELPER) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(TC_TMEM) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        // scales and biases, eight groups at a time: 16 bytes where they may be read so, else four or two
        const int vec = (groups & 7) == 0 && (g_begin & 7) == 0 && tp.s_align >= 16 ? 16 : (groups & 1) == 0 && (g_begin & 1) == 0 && tp.s_align >= 4 ? 4 : 2;
        const int n_chunks = (ng + 7) >> 3, trow = quad * 32 + lane;
        int n_blk = cid, n_c = 0;                               // the cursor of these loads
        auto load_pairs = [&](const char* ptr, int left) -> uint4 {
            if (vec == 16) return __ldg(reinterpret_cast<const uint4*>(ptr));
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                w[i] = 0u;
                if (2 * i < left) {
                    if (vec == 4) {
                        w[i] = __ldg(reinterpret_cast<const uint32_t*>(ptr) + i);
                    } else {
                        w[i] = __ldg(reinterpret_cast<const uint16_t*>(ptr) + 2 * i);
                        if (2 * i + 1 < left) w[i] |= static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(ptr) + 2 * i + 1)) << 16;
                    }
                }
            }
            return make_uint4(w[0], w[1], w[2], w[3]);
        };
        uint4 s_next = make_uint4(0, 0, 0, 0), b_next = s_next;
        auto load_next = [&]() {
            const int pi = part_of(n_blk), r = min((n_blk - tp.first_block[pi]) * 128 + trow, q.part[pi].rows - 1);
            const size_t off = (static_cast<size_t>(r) * groups + g_begin + n_c * 8) * 2;
            s_next = load_pairs(static_cast<const char*>(q.part[pi].s) + off, ng - n_c * 8);
            b_next = load_pairs(static_cast<const char*>(q.part[pi].b) + off, ng - n_c * 8);
            if (++n_c == n_chunks) { n_c = 0; n_blk += tp.clusters; }
        };
        if (warp < TC_DRAINERS && my_blocks > 0) load_next();   // (the layer's constants)
        ready();
        // ---- the activations: nothing before this line reads x or writes y --------------------------------------------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        {
            const int sidx = warp < TC_DRAINERS ? threadIdx.x : threadIdx.x - TC_UNPACKERS * 32;
            const int cpr = codes >> 3, cpg = 1 << (gs_shift - 3);               // chunks of eight activations per token and group
            constexpr int U = 2;                                // chunks of a thread in work together, and as many in flight
            int tok[U], c[U], ntok = 0, nc = sidx;              // (token ntok, chunk nc: the thread's next to load)
            uint4 ra[U], rb[U];
            auto load = [&]() {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    while (nc >= cpr && ntok < T) { nc -= cpr; ntok++; }
                    tok[u] = ntok; c[u] = nc;
                    ra[u] = rb[u] = make_uint4(0, 0, 0, 0);
                    if (ntok < T) load8_raw(q.x, q.x_dtype, static_cast<size_t>(ntok) * q.x_stride + k0 + nc * 8, ra[u], rb[u]);
                    nc += TC_STAGERS;
                }
            };
            load();
#pragma unroll 1
            for (int base = 0; base < T * cpr; base += U * TC_STAGERS) {         // whole warps
                float f[U][8], sum[U], top[U];
                int kt[U], kc[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    raw_to_float8(q.x_dtype, ra[u], rb[u], f[u]);
                    kt[u] = tok[u]; kc[u] = c[u];
                }
                load();
#pragma unroll
                for (int u = 0; u < U; u++) {
                    sum[u] = ((f[u][0] + f[u][1]) + (f[u][2] + f[u][3])) + ((f[u][4] + f[u][5]) + (f[u][6] + f[u][7]));
                    top[u] = 0.0f;
#pragma unroll
                    for (int i = 0; i < 8; i++) top[u] = fmaxf(top[u], fabsf(f[u][i]));
                }
                for (int o = 1; o < cpg; o <<= 1)
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        sum[u] += __shfl_xor_sync(0xffffffffu, sum[u], o);
                        top[u] = fmaxf(top[u], __shfl_xor_sync(0xffffffffu, top[u], o));
                    }
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (kt[u] < T) {
                        // a power of two per token and group, which the drain undoes
                        const uint32_t e = token_scale_exponent(top[u]);
                        const float factor = __uint_as_float(e << 23);
                        if ((kc[u] & (cpg - 1)) == 0) {
                            float* g = xsum + ((kc[u] * 8) >> gs_shift) * 2 * NTK + kt[u];
                            g[0] = sum[u];
                            g[NTK] = __uint_as_float((254u - e) << 23);
                        }
#pragma unroll
                        for (int i = 0; i < 8; i++) f[u][i] *= factor;
                        tc_stage8<BITS, SPLIT>(xs, X_TILE, X_PART, kt[u], kc[u] * 8, f[u]);
                    }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // the MMAs read the tiles through the async proxy
            asm volatile("bar.sync 1, %0;" ::"n"(TC_STAGERS) : "memory");
        }

        if (warp == TC_ISSUER) {
            // ---- MMA issuer: the warp's lanes stay together, one is elected for the instructions ---------------------------
            uint32_t slot = 0, d_phase = 1, sa = 0, a_phase = 0;                 // (the first turn of every slot waits for nothing)
            // fp32 accumulate, A and B fp16, both K-major, N = 16, M = 128
            constexpr uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(TC_BN >> 3) << 17) | (8u << 24);
            const uint32_t xa = smem_u32(xs);
            const uint64_t x_desc = static_cast<uint64_t>((xa >> 4) & 0x3FFF) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
            auto issue = [&](auto gc) {
                constexpr int GS = decltype(gc)::value, GPT = TC_STAGE / GS;    // groups per stage
#pragma unroll 1
                for (int b = 0; b < my_blocks; b++)
#pragma unroll 1
                    for (int s = 0; s < ns; s++) {
                        const uint32_t a = tmem + TC_SD * TC_D_COLS + sa * TC_A_COLS;
                        const uint64_t x = x_desc + static_cast<uint64_t>(s * 2 * (X_TILE / 16));
                        static_for<0, GPT, 1>([&](auto ic) {
                            constexpr int gi = decltype(ic)::value;
                            const int g = s * GPT + gi;
                            if (gi == 0 || g % TC_GPS == 0) {
                                if (lane == 0) {
                                    if (g % TC_GPS == 0) mbar_wait(&bars->d_empty[slot], d_phase, &bars->abort_flag, p.err);
                                    if (gi == 0) mbar_wait(&bars->full_a[sa], a_phase, &bars->abort_flag, p.err);
                                }
                                __syncwarp();
                                tc_fence_after();
                            }
                            const uint32_t d = tmem + slot * TC_D_COLS + (g % TC_GPS) * TC_BN;
                            const bool done = g % TC_GPS == TC_GPS - 1 || g == ng - 1;
                            if (elect_one()) {
                                // (the low parts first: a sum is cut off at about 2^-25 of what the accumulator holds, so that they
                                // lose nothing then, and the high parts' sum no more than without them; with the parts by turns the
                                // error was twice as large)
#pragma unroll
                                for (int part = SPLIT - 1; part >= 0; part--)
#pragma unroll
                                    for (int kk = 0; kk < GS / 16; kk++) {
                                        const int at = gi * (GS / 16) + kk;     // K slice of 16 inside the stage
                                        tc_mma_ts(d, a + at * 8, x + static_cast<uint64_t>((at / 4) * (X_TILE / 16) + part * (X_PART / 16) + (at % 4) * 2), idesc,
                                                  part < SPLIT - 1 || kk != 0);
                                    }
                                if (gi == GPT - 1) tc_commit(&bars->empty_a[sa]);
                                if (done) tc_commit(&bars->d_full[slot]);
                            }
                            __syncwarp();
                            if (done && ++slot == TC_SD) { slot = 0; d_phase ^= 1; }
                        });
                        if (++sa == TC_SA) { sa = 0; a_phase ^= 1; }
                    }
            };
            if (gs_shift == 6) issue(std::integral_constant<int, 64>{});
            else if (gs_shift == 5) issue(std::integral_constant<int, 32>{});
            else issue(std::integral_constant<int, 128>{});
        } else if (warp < TC_DRAINERS) {
            // ---- draining warps: a lane quadrant's 32 rows, all tokens ------------------------------------------------------
            const uint32_t base = tmem + (static_cast<uint32_t>(quad * 32) << 16);
            const bool s_f16 = q.s_dtype == DT_F16;
            const int rp_shift = 7 - tp.kz_shift, rp = 128 >> tp.kz_shift;       // rows of a block that this CTA finishes
            const int owner = trow >> rp_shift;
            const int total = my_blocks * n_chunks;
            uint32_t slot = 0, d_phase = 0;
            int j = 0, c = 0;                                   // the block in work (its number here) and its eight groups
            uint64_t acc2[NTK / 2];
#pragma unroll
            for (int t = 0; t < NTK / 2; t++) acc2[t] = 0ull;
#pragma unroll 1
            for (int ci = 0; ci <= total; ci++) {               // (the last turn finishes the last block)
                uint4 sv = s_next, bv = b_next;
                if (ci + 1 < total) load_next();
                int done = ci == total ? my_blocks - 1 : -1;    // the block to finish in this turn
                if (ci < total) {
                    const int g_end = min(ng, c * 8 + 8);
#pragma unroll 1
                    for (int g = c * 8; g < g_end; g += TC_GPS) {
                        mbar_await_warp(&bars->d_full[slot], d_phase, &bars->abort_flag, p.err);
                        tc_fence_after();
                        uint32_t d[TC_GPS][NTK];
#pragma unroll
                        for (int i = 0; i < TC_GPS; i++) tc_ld_cols<NTK>(base + slot * TC_D_COLS + i * TC_BN, d[i]);
                        float sc[2], bi[2];                      // of groups g and g + 1
                        if (s_f16) {
                            const float2 s2 = __half22float2(*reinterpret_cast<const __half2*>(&sv.x)), b2 = __half22float2(*reinterpret_cast<const __half2*>(&bv.x));
                            sc[0] = s2.x; sc[1] = s2.y; bi[0] = b2.x; bi[1] = b2.y;
                        } else {
                            sc[0] = __uint_as_float(sv.x << 16); sc[1] = __uint_as_float(sv.x & 0xFFFF0000u);
                            bi[0] = __uint_as_float(bv.x << 16); bi[1] = __uint_as_float(bv.x & 0xFFFF0000u);
                        }
                        sv.x = sv.y; sv.y = sv.z; sv.z = sv.w;   // on to the next pair
                        bv.x = bv.y; bv.y = bv.z; bv.z = bv.w;
                        const float* xg = xsum + g * 2 * NTK;
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars->d_empty[slot]);
                        if (++slot == TC_SD) { slot = 0; d_phase ^= 1; }
#pragma unroll
                        for (int i = 0; i < TC_GPS; i++, xg += 2 * NTK) {
                            if (i > 0 && g + i >= ng) break;     // (an odd number of groups: the slot's second is not there)
                            const float s1 = sc[i], b1 = fmaf(sc[i], static_cast<float>(1 << (BITS - 1)), bi[i]);
                            const uint64_t s2 = f2_pack(s1, s1), b2 = f2_pack(b1, b1);
#pragma unroll
                            for (int t = 0; t < NTK; t += 4) {
                                // the tokens' sums and inverse factors, four at a time
                                uint64_t x2[2], f2[2];
                                if constexpr (NTK >= 4) {
                                    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xg + t), b = *reinterpret_cast<const ulonglong2*>(xg + NTK + t);
                                    x2[0] = a.x; x2[1] = a.y; f2[0] = b.x; f2[1] = b.y;
                                } else {
                                    x2[0] = *reinterpret_cast<const uint64_t*>(xg); f2[0] = *reinterpret_cast<const uint64_t*>(xg + NTK);
                                }
#pragma unroll
                                for (int h = 0; h < (NTK >= 4 ? 2 : 1); h++) {
                                    const uint64_t v = f2_pack(__uint_as_float(d[i][t + 2 * h]), __uint_as_float(d[i][t + 2 * h + 1]));
                                    acc2[t / 2 + h] = f2_add(acc2[t / 2 + h], f2_fma(b2, x2[h], f2_mul(f2_mul(s2, v), f2[h])));
                                }
                            }
                        }
                    }
                    if (++c == n_chunks) {
                        // ---- the block is drained: its sums to the CTAs that finish the rows ------------------------------
                        c = 0;
                        // (they have read what was stored two blocks ago)
                        if (j >= 2) mbar_await_cluster_warp(&bars->red_empty[j & 1], ((j >> 1) - 1) & 1, &bars->abort_flag, p.err);
                        const uint32_t to = cluster_map(smem_u32(red + static_cast<size_t>(j & 1) * T * 128 + ((rank * T) << rp_shift) + (trow & (rp - 1))), owner);
#pragma unroll
                        for (int t = 0; t < NTK; t += 2) {
                            float v0, v1;
                            f2_unpack(acc2[t / 2], v0, v1);
                            acc2[t / 2] = 0ull;
                            if (t < T) cluster_store(to + ((t << rp_shift) * 4), v0);
                            if (t + 1 < T) cluster_store(to + (((t + 1) << rp_shift) * 4), v1);
                        }
                        __syncwarp();
                        // one arrival per warp and owner: of eight owners a warp's rows have two
                        if (lane == 0 || (kz == 8 && lane == 16)) cluster_arrive(cluster_map(smem_u32(&bars->red_full[j & 1]), owner));
                        __syncwarp();
                        done = j - 1;
                        j++;
                    }
                }
                if (done >= 0) {
                    // ---- the slices' sums of this CTA's rows of block number `done`, in order; row bias, store ---------------
                    mbar_await_cluster_warp(&bars->red_full[done & 1], (done >> 1) & 1, &bars->abort_flag, p.err);
                    const float* from = red + static_cast<size_t>(done & 1) * T * 128;
                    const int blk = cid + done * tp.clusters, pi = part_of(blk);
#pragma unroll 1
                    for (int i = threadIdx.x; i < (T << rp_shift); i += TC_DRAINERS * 32) {
                        float v = 0.0f;
                        for (int z = 0; z < kz; z++) v += from[((z * T) << rp_shift) + i];
                        const int row = (blk - tp.first_block[pi]) * 128 + rank * rp + (i & (rp - 1));
                        if (row < q.part[pi].rows) {
                            if (q.has_bias) v += load_scalar(q.part[pi].bias, q.bias_dtype, row);
                            store_scalar(q.y, q.y_dtype, static_cast<size_t>(i >> rp_shift) * q.y_stride + tp.first_row[pi] + row, v);
                        }
                    }
                    __syncwarp();
                    if (done + 2 < my_blocks && lane < kz) cluster_arrive(cluster_map(smem_u32(&bars->red_empty[done & 1]), lane));
                    __syncwarp();
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == TC_HELPER) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM) : "memory");
    }
    if (kz > 1) tc_cluster_barrier();                           // nobody leaves while others store into its shared memory or arrive there
}

// What a device holds at once: its SMs, and clusters of 1, 2, 4 and 8 CTAs with one CTA an SM and with two.
struct TcRoom {
    int sms;
    int one[4], two[4];
};
const TcRoom& qmv_tc_room(int device, int sms);

// What a call runs on where the kernel does not take it (`general`: the one-token kernel's general plan); `named` is a call that the
// kernel takes whenever it can serve it.
enum class TcInstead { named, token_major, cluster, scaled_cluster, halves, general, other };

// Plans a call; returns the shared memory it needs, 0 when the call is not one the kernel serves, or not one that it is the faster
// for than what the call runs on otherwise.
size_t qmv_tc_plan(int bits, const MmaParams& p, int tokens, TcInstead instead, const TcRoom& room, TcPlan& tp);
cudaError_t launch_qmv_tc(int bits, const MmaParams& p, const TcPlan& tp, size_t smem, int device, cudaStream_t st);

}  // namespace mlxq
