// Handing out the clusters of a grid that have not started yet (cluster launch control), without anything of the GPU in
// it, so that a host compiler takes it too.
//
// Port is what the protocol talks to:
//   request()       asks for a cluster that has not started; if there is one it will not start, and its work is the asker's
//   wait()          until the answer is there; false: abandoned, the answer may still be on its way
//   wait_through()  the same with a time limit as the only reason to give up (not because some other role has)
//   answer()        first CTA of the cluster, or -1 if none was left
#pragma once

#ifdef __CUDACC__
#define MOE_DRAW_FN __device__ __forceinline__
#else
#define MOE_DRAW_FN inline
#endif

namespace moe {
namespace tc {

// One request at a time, and none after an answer without a cluster.
template <typename Port>
class ClusterDraw {
  Port& port;
  bool pending = false;  // a request whose answer has not been read
  bool empty = false;    // the last answer had no cluster

  MOE_DRAW_FN int read() {
    pending = false;
    const int cta = port.answer();
    empty = cta < 0;
    return cta;
  }

 public:
  enum : int { NONE_LEFT = -1, ABANDONED = -2 };
  MOE_DRAW_FN explicit ClusterDraw(Port& p) : port(p) {}
  MOE_DRAW_FN void ask() { port.request(); pending = true; }
  MOE_DRAW_FN int collect() { return port.wait() ? read() : (int)ABANDONED; }
  // Called when the asker leaves.  After the last answer there is nothing to do.  When it leaves early (some wait of this
  // CTA ran into its limit), the answer on its way to this CTA's shared memory is waited for, and the clusters that have not
  // started are claimed without doing their work: each of them would otherwise start and could run into the same limit,
  // one wave after the other.
  MOE_DRAW_FN void leave() {
    if (pending) {
      if (!port.wait_through()) return;
      read();
    }
    while (!empty) {
      ask();
      if (!port.wait_through()) return;
      read();
    }
  }
};

// Publishes this cluster's own tile `first`, then the tiles of the clusters drawn, then -1.  Ids from `total` on (the grid
// is an upper bound) are passed over.  publish(tile) returns false when its wait was abandoned.
template <int CTAS, typename Port, typename Publish>
MOE_DRAW_FN void hand_out_tiles(Port& port, int total, int first, Publish publish) {
  ClusterDraw<Port> draw(port);
  for (int tile = first;;) {
    if (tile < total && !publish(tile)) break;
    draw.ask();
    const int cta = draw.collect();
    if (cta == ClusterDraw<Port>::ABANDONED) break;
    if (cta < 0) { publish(-1); break; }
    tile = cta / CTAS;
  }
  draw.leave();
}

}  // namespace tc
}  // namespace moe
