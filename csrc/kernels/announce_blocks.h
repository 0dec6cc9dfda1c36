// How many blocks the transport kernels of the expert-parallel step are launched with. Plain arithmetic: the launchers and the
// threaded host twin (csrc/sched/moe_twin.cc) use the same rule.
#pragma once

namespace fastb {

// `blocks`: what a rank's own rows ask for, 0 when it has none. A kernel that also tells the peers something they wait for (its
// receive buffers may be written; its expert rows are final) is launched all the same: a rank without tokens still owns experts
// that other ranks' tokens went to. One block is enough to say so.
inline int announce_blocks(int blocks, bool announces) { return blocks > 0 ? blocks : announces ? 1 : 0; }

}  // namespace fastb
