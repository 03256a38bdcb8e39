// Planner and launcher of the tensor-memory decode matvec (qmv_tc.cuh).
#include "qmv_tc.cuh"

#include <mutex>

namespace mlxq {

// (qmv_tc_inst.cu) clusters of `kz` CTAs with `smem` bytes each that the current device holds at once; 0 where it cannot say
int qmv_tc_clusters(int kz, size_t smem);

cudaError_t launch_qmv_tc_b2(const MmaParams&, const TcPlan&, size_t, int, cudaStream_t);
cudaError_t launch_qmv_tc_b3(const MmaParams&, const TcPlan&, size_t, int, cudaStream_t);
cudaError_t launch_qmv_tc_b4(const MmaParams&, const TcPlan&, size_t, int, cudaStream_t);
cudaError_t launch_qmv_tc_b5(const MmaParams&, const TcPlan&, size_t, int, cudaStream_t);
cudaError_t launch_qmv_tc_b6(const MmaParams&, const TcPlan&, size_t, int, cudaStream_t);
cudaError_t launch_qmv_tc_b8(const MmaParams&, const TcPlan&, size_t, int, cudaStream_t);

namespace {

int align_up(int v, int a) { return (v + a - 1) / a * a; }

// Whether the kernel is the faster one for a call that others could serve, and no less exact.  Both sides in us, this kernel's
// first; 4 bits in groups of 64 unless it says otherwise.
bool worth(int bits, int gs, int K, int rows, int tokens, int split) {
    // 6 and 8 bits in groups of 128: long sums of uncentred codes, whose error is above the token-major kernel's (8 bits, fp32
    // tokens 4.4e-7 of the result against 3.4e-7; in groups of 64 3.1e-7 against 3.7e-7)
    if (bits >= 6 && gs == 128) return false;
    // more fp32 tokens than the others take at once: 1024 x 1024, 16 tokens 5.7 : 8.3; 4096 x 4096 12.3 : 24.8; 4096 x 12288
    // 37 : 231; 24576 x 4096 42 : 72; 11008 x 4096 at 3 bits 31 : 361
    if (split == 2 && tokens > 8) return true;
    // short rows: the fixed part of a launch decides (6 fp32 tokens: 4096 x 1024 at 8 bits 5.8 : 5.3, 1024 x 1024 4.5 : 4.1;
    // 2048 x 2048 5.7 : 6.3, 1024 x 3072 at 8 bits 6.1 : 7.9)
    if (K < 2048) return false;
    // the token-major kernel's second eight columns.  6 fp32 tokens: 4096 x 4096 9.3 : 11.8, 4096 x 12288 15.5 : 24.4,
    // 24576 x 4096 25.7 : 33.4, 151936 x 4096 at 6 bits 152 : 158, at 8 bits 140 : 153
    if (split == 2 && tokens > 4) return true;
    // 13 fp16 tokens (sixteen columns drained): 4096 x 4096 12.0 : 13.6, 4096 x 12288 23 : 36, 11008 x 4096 at 3 bits 25.6 : 31.0,
    // but 24576 x 4096 36.8 : 36.8, 14336 x 4096 at 8 bits 27.2 : 26.0, 151936 x 4096 at 8 bits 197 : 164
    if (split == 1 && tokens > 8) return rows <= (bits == 8 ? 8192 : 12288);
    if (bits == 8) return false;                               // 14336 x 4096, 4 fp32 tokens 18.2 : 16.8, 8 fp16 ones 21.3 : 18.6
    // 4 fp32 tokens: 4096 x 4096 8.6 : 9.2, 24576 x 4096 22.3 : 25.8, 40960 x 2048 19.6 : 22.1, 151936 x 4096 at 6 bits 145 : 130
    if (split == 2 && tokens > 2) return rows <= 40960;
    // 8 fp16 tokens: 4096 x 4096 9.8 : 10.4, 4096 x 12288 16.6 : 19.5, 24576 x 4096 26.6 : 27.6, 40960 x 2048 23.9 : 23.2
    if (split == 1 && tokens > 4) return rows <= 24576;
    // 2 fp32 tokens: 4096 x 12288 14.4 : 17.4, but 4096 x 4096 8.4 : 7.7
    return split == 2 && tokens == 2 && K >= 8192 && rows <= 12288;
}

}  // namespace

// Asked for once per device, with that device current.  (B200: 148 SMs, 148, 74, 33 and 15 clusters with one CTA an SM, 296, 148,
// 71 and 33 with two: parts of the chip have an SM count that is no multiple of the cluster's.)
const TcRoom& qmv_tc_room(int device, int sms) {
    static std::mutex mu;
    static TcRoom rooms[64] = {};
    TcRoom& r = rooms[device];
    std::lock_guard<std::mutex> lk(mu);
    if (r.sms == 0) {
        for (int shift = 0; shift <= 3; shift++) {
            r.one[shift] = qmv_tc_clusters(1 << shift, TC_SMEM_WHOLE);
            r.two[shift] = qmv_tc_clusters(1 << shift, TC_SMEM_TWO);
        }
        r.sms = sms;
    }
    return r;
}

size_t qmv_tc_plan(int bits, const MmaParams& p, int tokens, bool always, const TcRoom& room, TcPlan& tp) {
    const QmvParams& q = p.q;
    if (q.K > STAGED_K_MAX || tokens < 2 || tokens > 16 || q.peer.n > 0 || q.x_up != nullptr || q.e != nullptr) return 0;
    if ((q.gs != 32 && q.gs != 64 && q.gs != 128) || (q.s_dtype != DT_F16 && q.s_dtype != DT_BF16) || q.K % TC_STAGE != 0) return 0;
    if (!always && !worth(bits, q.gs, q.K, q.total_rows, tokens, p.split)) return 0;
    tp = TcPlan{};
    uintptr_t at = 16;
    for (int i = 0; i < q.n_parts; i++) {
        if ((reinterpret_cast<uintptr_t>(q.part[i].w) & 15u) != 0) return 0;
        at |= reinterpret_cast<uintptr_t>(q.part[i].s) | reinterpret_cast<uintptr_t>(q.part[i].b);
        tp.first_block[i] = tp.n_blocks;
        tp.first_row[i] = i == 0 ? 0 : tp.first_row[i - 1] + q.part[i - 1].rows;
        tp.n_blocks += (q.part[i].rows + 127) / 128;
    }
    tp.s_align = static_cast<int>(at & (~at + 1));
    tp.stages = q.K / TC_STAGE;
    // The cut of K: the one that is done first by what was measured (6 fp32 tokens, 4 bits): a stage takes 0.8 us where two CTAs
    // share an SM and 0.47 where one has it, the end of a block and its slices' meeting 2 us.  24576 x 4096 in 2, 4 and 8
    // slices: 30.1, 25.7, 31.9 us; 40960 x 2048: 22.3, 26.6, 37.8; 4096 x 4096: 13.9, 10.5, 9.3.  (From the tokens the kernel
    // is compiled for, not the batch's: a token's sums do not change with its company.)
    const int ntk = tc_tokens(tokens), part = ntk <= 8 ? 1024 : 2048, slot = tc_slot_bytes(bits);
    // 16-bit activations at 8 bits, and at 5 and 6 bits in groups of 32: the call stands in for kernels that multiply and add in
    // fp32, whose error grows with the number of groups and codes that one CTA sums up.  Error of the result, this kernel's first
    // (16 bf16 tokens): 8 bits in groups of 32, 48 groups of 12288 codes 1.42e-7 : 1.19e-7 and 28 groups of 8192 codes below
    // theirs; in groups of 64, 3072 codes 1.39e-7 : 1.19e-7, 1792 codes 1.19e-7 : 1.24e-7.
    const bool fp32_stand_in = p.split == 1 && (bits == 8 || (bits >= 5 && q.gs == 32));
    double best = 0.0;
    size_t best_smem = 0;
    for (int shift = 0; shift <= 3; shift++) {
        const int kz = 1 << shift;
        if (kz > tp.stages) continue;
        const int slice = (tp.stages + kz - 1) / kz;
        if (fp32_stand_in && (slice * TC_STAGE > 2048 || slice * TC_STAGE / q.gs > 32)) continue;
        const int x_bytes = slice * 2 * p.split * part, xsum = align_up((slice * TC_STAGE / q.gs) * ntk * 8, 16), redb = 2 * ntk * 128 * 4;
        const int fixed = 1024 + x_bytes + xsum + redb + static_cast<int>(sizeof(TcBarriers));
        const bool two = fixed + 3 * slot <= TC_SMEM_TWO;
        int depth = ((two ? TC_SMEM_TWO : TC_SMEM_WHOLE) - fixed) / slot;
        if (depth < 3) continue;
        depth = depth >= 8 ? 8 : depth >= 6 ? 6 : depth >= 4 ? 4 : 3;
        const int resident = (two ? room.two : room.one)[shift], clusters = tp.n_blocks < resident ? tp.n_blocks : resident;
        if (clusters < 1) continue;
        const int rounds = (tp.n_blocks + clusters - 1) / clusters;
        const double cost = rounds * (slice * (clusters * kz > room.sms ? 0.8 : 0.47) + 2.0);
        if (best_smem != 0 && cost >= best) continue;
        best = cost;
        tp.kz = kz; tp.kz_shift = shift; tp.clusters = clusters; tp.depth = depth;
        tp.off_x = depth * slot;
        tp.off_xsum = tp.off_x + x_bytes;
        tp.off_red = tp.off_xsum + xsum;
        tp.off_bars = tp.off_red + redb;
        best_smem = static_cast<size_t>(fixed) + static_cast<size_t>(depth) * slot;
        if (two && best_smem < 80 * 1024) best_smem = 80 * 1024;            // (never three an SM: they would queue for tensor memory)
    }
    return best_smem;
}

cudaError_t launch_qmv_tc(int bits, const MmaParams& p, const TcPlan& tp, size_t smem, int device, cudaStream_t st) {
    switch (bits) {
        case 2: return launch_qmv_tc_b2(p, tp, smem, device, st);
        case 3: return launch_qmv_tc_b3(p, tp, smem, device, st);
        case 4: return launch_qmv_tc_b4(p, tp, smem, device, st);
        case 5: return launch_qmv_tc_b5(p, tp, smem, device, st);
        case 6: return launch_qmv_tc_b6(p, tp, smem, device, st);
        case 8: return launch_qmv_tc_b8(p, tp, smem, device, st);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace mlxq
