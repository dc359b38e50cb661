// team_ring.cuh -- the order of work of teams of threads on a ring of tile
// buffers: tile j is in buffer j mod NB and is transformed by team j mod TEAMS.
// Used by the two-round pass (ntt_pass_duo.cuh); free of CUDA names, so that
// CPU threads can run the same code.
//
// Load j completes phase j / NB of its buffer's `landed` barrier, and a wait
// names the phase's parity only: it also succeeds on a barrier that is one
// phase behind.  The buffer's uses alternate between the teams (NB is odd,
// TEAMS 2), so a team that is through with tile j + 1 can come to wait for tile
// j + NB while tile j, another team's, is still on its way.  It therefore waits
// first until load j + NB has been issued, a phase of the buffer's `issued`
// barrier: that comes after tile j has landed, and the issue before it (load j)
// was the waiting team's own, so neither wait can meet an older phase.  With
// one team every earlier use of the buffer is the team's own.
//
// Ops, called by every thread of a team but for those marked (leader):
//   bool wait_issued(b, parity), wait_landed(b, parity)
//                             bounded waits on buffer b's barriers; false: gave up
//   void gave_up()            raise the error and the abort flag of all teams
//   void landed(b)            (leader) count a load of buffer b that has landed
//   void issue(j)             (leader) start the load of tile j
//   void transform(j, b)      transform tile j in its buffer
//   bool aborted()            the abort flag
//   bool any(x)               barrier of the team; true for all of its threads
//                             if any of them brought x.  (The flag as each
//                             thread reads it can differ between them, as other
//                             teams set it at any time: some would leave and
//                             the rest wait for them.)
//   void store(j, b)          (leader) start the store of tile j
//   void store_read()         (leader) wait until the stores have read their buffers
#pragma once
#include "fields.cuh"

namespace omr {

template <int NB, int TEAMS, class Ops>
OMR_D void team_ring_run(Ops& op, uint32_t team, bool leader, uint32_t njobs) {
  static_assert(2 * NB % TEAMS == 0, "loads j and j + 2 NB are issued by one team");
  uint32_t refill = 0xffffffffu;  // (leader) the load that follows the last store's read
  for (uint32_t j = team; j < njobs; j += TEAMS) {
    const uint32_t b = j % NB, k = j / NB;
    // read here, where the wait covers it, and not at the barrier: on GB300
    // BabyBear 64 x 2^20 289.0 -> 286.5 us, inverse 297.1 -> 294.5
    const bool seen = op.aborted();
    bool ok = true;
    if (TEAMS > 1) ok = op.wait_issued(b, k & 1);
    if (ok) ok = op.wait_landed(b, k & 1);
    if (!ok)
      op.gave_up();
    else if (leader)
      op.landed(b);
    if (leader && refill != 0xffffffffu) {
      op.store_read();  // (long done: it had the wait above)
      op.issue(refill);
      refill = 0xffffffffu;
    }
    op.transform(j, b);
    if (op.any(!ok || seen)) break;
    if (leader) {
      op.store(j, b);
      if (j + NB < njobs) {
        refill = j + NB;
        if (NB == 1) {  // the next tile needs this buffer
          op.store_read();
          op.issue(refill);
          refill = 0xffffffffu;
        }
      }
    }
  }
}

}  // namespace omr
