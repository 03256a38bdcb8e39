// Host program of test_decode_plans_cpu.py: runs the planners of the decode kernels on calls given on standard input, one per
// line, and prints what they plan.  It launches nothing and needs no GPU; pointers are made up and never followed.
#include <cstdio>

#include "qmv_pipe.cuh"
#include "qmv_tc.cuh"
#include "qmv_tok.cuh"

using namespace mlxq;

int main(int argc, char** argv) {
    TcRoom room = {148, {148, 74, 33, 15}, {296, 148, 71, 33}};         // a B200
    if (argc > 1) room = TcRoom{20, {20, 10, 5, 0}, {40, 20, 10, 0}};   // a part of one that holds no cluster of eight
    int bits, gs, K, rows, tokens, split, instead;
    while (std::scanf("%d %d %d %d %d %d %d", &bits, &gs, &K, &rows, &tokens, &split, &instead) == 7) {
        MmaParams p = {};
        QmvParams& q = p.q;
        for (QmvPart& part : q.part) {
            part.w = reinterpret_cast<const uint8_t*>(4096);
            part.s = part.b = reinterpret_cast<const void*>(4096);
            part.rows = rows;
        }
        q.n_parts = 1;
        q.total_rows = rows;
        q.K = K;
        q.gs = gs;
        q.T = tokens;
        q.s_dtype = DT_BF16;
        q.x_dtype = split == 2 ? DT_F32 : DT_BF16;
        for (int s = 3; s < 31; s++) if ((1 << s) == gs) q.gs_shift = s;
        p.split = split;
        TcPlan tc = {};
        const size_t tcs = qmv_tc_plan(bits, p, tokens, static_cast<TcInstead>(instead), room, tc);
        std::printf("%zu %d %d %d %d %d %d %d %d %d", tcs, tc.kz, tc.stages, tc.depth, tc.off_x, tc.off_xsum, tc.off_red, tc.off_bars, tc.clusters, tc.n_blocks);
        const bool columns = qmv_mma_plan(bits, K, gs, tokens * split, p);
        for (int clusters = 0; clusters <= 2; clusters++) {
            TokPlan tok = {};
            const size_t s = columns ? qmv_tok_plan(bits, p, tokens, 148, tok, clusters) : 0;
            std::printf(" | %zu %d %d %d %d %d", s, tok.off_parts, tok.off_zero, tok.off_part, tok.off_tab, tok.off_ring);
        }
        PipePlan pipe = {};
        const size_t s = columns ? qmv_pipe_plan(bits, p, tokens, 148, pipe) : 0;
        std::printf(" | %zu %d %d %d %d %d\n", s, pipe.off_xsum, pipe.off_zero, pipe.off_scratch, pipe.off_part, pipe.off_ring);
    }
    return 0;
}
