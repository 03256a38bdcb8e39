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

// Whether the kernel is the faster one, by what the call runs on otherwise.  Fitted to 70,000 calls timed on both sides in turn: 6
// widths, groups of 32, 64 and 128, 33 row counts of 512 ... 151936, 26 row lengths of 512 ... 14336, batches of 2 ... 16 tokens of
// each type: of the 24,100 calls that the rules take, 0.7 % are more than 1.5 % slower than before, 9 by more than 10 %, and the
// mean is 2.4 times as fast.  (11008 x 4096, 3 bits, 16 fp32 tokens, in the place of CUDA cores: 361 -> 32 us.)

// In the place of one launch of the token-major kernel on single CTAs.  Each of its CTAs stages all of K of the batch: the KB of
// that decide, fewer of them where there are few rows to share it.  us before : with this kernel, groups of 64: 6 fp32 tokens at
// 4 bits, 4096 x 4096 (96 KB) 12.1 : 10.1, 24576 x 4096 33.5 : 28.7, 24576 x 2048 17.7 : 17.9, 4096 x 1024 5.8 : 6.8; 4 tokens
// 24576 x 4096 25.9 : 27.3; 6 tokens at 6 bits 151936 x 4096 159 : 175; 8 fp16 tokens at 3 bits 11008 x 4096 (64 KB) 22.5 : 20.3.
bool over_token_major(int bits, int gs, int rows, int tokens, int split, int kb) {
    const bool even = bits == 4 || bits == 8, fp32 = split == 2;
    if (gs == 32 && bits == 4 && !fp32) return false;
    if (tokens <= 4) {
        // (few tokens: the other kernel has one set of accumulators and few staged columns)
        if (!fp32) return false;
        if (tokens == 2) return gs == 64 && bits <= 5 && rows <= 6144 && (even || bits == 2 ? kb >= 80 && kb <= 96 : kb >= 60);
        if (rows <= 3072) return kb >= (gs == 128 && !even ? 40 : 80);
        if (gs == 32) return bits >= 6 && kb >= (rows <= 15360 ? 72 : 48);
        if (gs == 128 || bits >= 6) return false;
        if (rows <= 15360) return kb >= 80 && (bits != 2 || rows <= 6144);
        return bits != 2 && kb >= (bits == 4 ? 144 : 112);
    }
    if (gs == 32) {
        if (bits == 6 && !fp32 && rows > 15360 && tokens <= 8) return kb >= 56;
        return kb >= (rows <= 3072 || bits == 4 || !fp32 || (bits == 6 && rows <= 15360) ? 96 : 56);
    }
    if (gs == 128) {
        if (!even) return rows <= 15360 && kb >= (rows <= 3072 ? 32 : rows <= 6144 ? 40 : 64);
        if (rows <= 3072) return kb >= (bits == 4 ? 56 : 40);
        return bits == 8 && fp32 && kb >= (rows <= 6144 ? 40 : 64);
    }
    if (rows <= 3072) return kb >= (fp32 || even ? 48 : rows <= 1536 ? 32 : 40);
    if (rows <= 6144) return kb >= (bits == 8 ? 112 : bits == 4 ? 72 : fp32 ? 64 : 56);
    if (fp32) {
        if (rows <= 15360) return kb >= (bits >= 6 ? 112 : bits == 5 ? 80 : 72);
        return bits <= 5 && kb >= (bits == 2 ? 144 : bits == 3 ? 96 : bits == 5 ? 80 : 72);
    }
    if (tokens <= 8 && bits >= 3 && bits <= 5) return kb >= (bits == 5 ? 72 : bits == 3 && rows <= 15360 ? 64 : 96);
    return rows <= 15360 && !even && kb >= 112;
}

// ... of the token-major kernel with K split over a cluster, `scaled` or not: mostly the taller layers, where its clusters queue
// (8 fp32 tokens, 4 bits, 11008 x 12288 60.9 : 41.0 us; 6 bits 61.4 : 64.2).
bool over_cluster(int bits, int gs, int K, int rows, int tokens, int split, bool scaled) {
    const bool fp32 = split == 2;
    if (tokens <= 4) return false;
    if (gs != 64 && scaled && fp32 && tokens >= 7 && (bits == 4 || (bits == 2 && gs == 128))) return true;
    if (gs == 128) return false;
    if (gs == 32) return fp32 && bits >= 6 && rows > 3072;
    if (!scaled) {
        if (!fp32) return (bits == 4 || bits == 5) && tokens <= 8 && rows > 6144 && K <= 12288;
        return (bits == 4 && rows > (tokens >= 6 ? 3072 : 6144)) || (bits == 5 && rows > 6144) || (bits == 3 && rows > 15360);
    }
    switch (bits) {
        case 2: return rows <= (fp32 ? 15360 : 3072) || (fp32 && tokens >= 7);
        case 3: return rows > 6144 && (fp32 || rows <= 15360);
        case 4: return fp32 || rows <= 15360;
        case 5: return rows > 3072;
        case 8: return fp32 && tokens >= 7 && rows <= 6144 && K <= 12288;
        default: return false;
    }
}

bool worth(TcInstead instead, int bits, int gs, int K, int rows, int tokens, int split) {
    switch (instead) {
        case TcInstead::named: return true;
        case TcInstead::token_major: return over_token_major(bits, gs, rows, tokens, split, tokens * split * (K / 128) / 4);      // (K <= STAGED_K_MAX)
        case TcInstead::cluster: return over_cluster(bits, gs, K, rows, tokens, split, false);
        case TcInstead::scaled_cluster: return over_cluster(bits, gs, K, rows, tokens, split, true);
        case TcInstead::halves:
            // two launches of the token-major kernel, which read the weights twice.  Not where they are near the memory's rate all the
            // same: vocabulary-sized layers, at 8 bits on rows that cut badly (100352 x 2560, 16 fp32 tokens 140 : 205 us), in groups of 128,
            // and at 6 bits on very short rows
            if (rows > 32768 && ((bits == 8 && K > 2048 && K < 4096) || (gs == 128 && K > 3072 && K < 8192))) return false;
            if (rows > 20480 && bits == 6 && K < 1024) return false;
            return true;
        case TcInstead::general: return tokens >= (split == 2 ? 3 : 5);
        default: return tokens >= (split == 2 ? 2 : 5);        // kernels on the CUDA cores, or that read the weights several times
    }
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

size_t qmv_tc_plan(int bits, const MmaParams& p, int tokens, TcInstead instead, const TcRoom& room, TcPlan& tp) {
    const QmvParams& q = p.q;
    if (q.K > STAGED_K_MAX || tokens < 2 || tokens > 16 || q.peer.n > 0 || q.x_up != nullptr || q.e != nullptr) return 0;
    if ((q.gs != 32 && q.gs != 64 && q.gs != 128) || (q.s_dtype != DT_F16 && q.s_dtype != DT_BF16) || q.K % TC_STAGE != 0) return 0;
    if (!tc_compiled(bits, tc_tokens(tokens), p.split) || !worth(instead, bits, q.gs, q.K, q.total_rows, tokens, p.split)) return 0;
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
    // The cut of K: the one that is done first by a cost in units of a stage of 128 codes on a CTA that has its SM alone.  Fitted
    // to the times of all four cuts at 6 widths, 14 row counts, 8 row lengths and 11 batches: the cut it takes is 1.1 % slower
    // than the best one on average, and 4 % at the ninth decile.  What it says: two CTAs an SM hide nearly all of a stage, so that
    // little but the staging of the activations (per stage, token and part; four times the stores at the widths whose codes
    // straddle bytes) and the blocks' ends are left to count.  11008 x 4096, 3 bits, 8 fp16 tokens in 2 and 8 slices: 34.2 and
    // 20.3 us; 24576 x 4096, 4 bits, 16 fp32 tokens in 2 and 8 slices: 55.2 and 45.1.  (From the tokens the kernel is compiled for,
    // not the batch's: a token's sums do not change with its company.)
    const int ntk = tc_tokens(tokens), part = ntk <= 8 ? 1024 : 2048, slot = tc_slot_bytes(bits);
    // 16-bit activations at 8 bits, and at 6 bits in groups of 32: the call stands in for kernels that multiply and add in fp32, and
    // the error here grows with the groups and codes that one CTA sums up.  Error of the result, this kernel's first (16 bf16
    // tokens): 8 bits in groups of 32, 48 groups of 12288 codes 1.42e-7 : 1.19e-7, 32 groups of 8192 codes below theirs; in groups
    // of 64, 3072 codes 1.39e-7 : 1.19e-7, 1792 codes 1.19e-7 : 1.24e-7; 6 bits, 96 groups 1.85e-7 : 1.73e-7, 48 groups
    // 1.41e-7 : 1.65e-7.
    const bool fp32_stand_in = p.split == 1 && (bits == 8 || (bits == 6 && q.gs == 32));
    const int most_codes = bits == 8 ? 2048 : 1536, most_groups = bits == 8 ? 32 : 48;
    double best = 0.0;
    size_t best_smem = 0;
    for (int shift = 0; shift <= 3; shift++) {
        const int kz = 1 << shift;
        if (kz > tp.stages) continue;
        const int slice = (tp.stages + kz - 1) / kz;
        if (fp32_stand_in && (slice * TC_STAGE > most_codes || slice * TC_STAGE / q.gs > most_groups)) continue;
        const int x_bytes = slice * 2 * p.split * part, xsum = align_up((slice * TC_STAGE / q.gs) * ntk * 8, 16), redb = 2 * ntk * 128 * 4;
        const int fixed = 1024 + x_bytes + xsum + redb + static_cast<int>(sizeof(TcBarriers));
        const bool two = fixed + 3 * slot <= TC_SMEM_TWO;
        int depth = ((two ? TC_SMEM_TWO : TC_SMEM_WHOLE) - fixed) / slot;
        if (depth < 3) continue;
        depth = depth >= 8 ? 8 : depth >= 6 ? 6 : depth >= 4 ? 4 : 3;
        const int resident = (two ? room.two : room.one)[shift], clusters = tp.n_blocks < resident ? tp.n_blocks : resident;
        if (clusters < 1) continue;
        const int rounds = (tp.n_blocks + clusters - 1) / clusters;
        const double staging = (bits == 3 || bits == 5 || bits == 6 ? 0.04 : 0.025) * ntk * (p.split + 1);
        const double cost = slice * staging + rounds * (slice * (clusters * kz > room.sms ? 0.07 : 1.0) + 0.25 + 0.3 * shift);
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
