// cg_flow.cuh — host interface of the dataflow CG (cg_flow.cu): the whole
// solve of a few small systems in one cooperative launch whose blocks pass
// vectors to each other in self-validating words.
#pragma once

#include <vector>

#include "cg_common.cuh"

namespace sfh {

constexpr int kFlowMaxLanes = 16;   // lanes of one system (RHS x parities)

// the blocks that own one system: block b of the team owns the checkerboard
// sites [b n, (b + 1) n) of both parities
struct FlowTeam {
    int sys, blk0, nblk, n;
    int words0;  // the team's first word in FlowArgs::sums
};

struct FlowArgs {
    const FlowTeam* teams;
    const int* blk_team;        // team of every block
    // {double, tag} words per team [2][4 nlanes][nblk], the block fastest, each
    // half followed by the totals' copies [ceil(nblk / 8)][4 nlanes]
    uint4* sums;
    unsigned* flags;            // one per block: barriers passed
    char* const* pub;           // per RHS: published p, then published t
    int* err;                   // set by a wait that gave up
    int polls;                  // bound on each wait
};

// The plan of one launch over all systems of a workspace.
struct FlowPlan {
    std::vector<FlowTeam> teams;   // one per system
    std::vector<int> blk_team;     // team of every block
    std::vector<size_t> pub_at;    // per RHS: its place in the published vectors
    size_t words = 0, pub_bytes = 0;
    int threads = 0;
    int split = 1;                 // threads per site in a hop
    int rounds = 1;                // of the block's threads, for a hop (1 where split is 4)
    size_t dyn = 0;                // dynamic shared memory of a block
};
// false where the per-phase kernels are the better ones (or the systems do
// not fit); host arithmetic only
bool flow_plan(const std::vector<CgSys>& sys, int prec, int num_sms, FlowPlan* plan);
// whether such a plan beats the best of the per-phase kernels' schedules too
bool flow_beats_tuned(const std::vector<CgSys>& sys, const FlowPlan& plan);
// the whole solve (after cg_init) in one cooperative launch
cudaError_t flow_launch(int prec, const CgArgs& a, const FlowArgs& f, const FlowPlan& plan, cudaStream_t stream);

constexpr int kFlowPolls = 1 << 22;  // bound on each wait, about 0.6 us a poll

}  // namespace sfh
