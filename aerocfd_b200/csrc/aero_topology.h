// Host-side builders of the device tables that replace the reference's
// per-iteration MPI exchange bookkeeping: the ghost-node gather map of
// UpdateBuffer / UpdateBufferCoordinate, the source/destination lists of
// average1 / average2, and the ordered physical-BC operations of physical_bc.
#pragma once
#include <string>
#include <vector>

#include "aero_kernels.h"

namespace aero {

struct SubRow {
  int f_no, face, is, ie, js, je, ks, ke, blk_t, subface_t, ori;
  Box box() const { return Box{is, ie, js, je, ks, ke}; }
};

struct TopoBlock {
  Box b, b0, b1;
  std::vector<SubRow> subs;
  long at(int i, int j, int k) const {
    return (long)(i - b.is) + (long)b.nx() * ((long)(j - b.js) + (long)b.ny() * (long)(k - b.ks));
  }
};

struct Topology {
  std::vector<HaloEntry> halo;     // ghost <- donor interior, all layers
  std::vector<AvgSrc> avg_src;     // grouped by destination, in reference order
  std::vector<AvgDst> avg_dst;
  std::vector<BcOp> bc_ops;        // per block, bcinfo order
  std::vector<int> bc_start;       // nblock+1 offsets into bc_ops
  std::vector<int> bc_level;       // per op: dependency level within its block (see bc_levels)
};

// Builds all tables (dimension: iflag_dimension, 2 or 3); returns an empty
// string on success or the reason the block/subface description is
// inconsistent.
std::string build_topology(const std::vector<TopoBlock>& blocks, int buffer_length, int solver,
                           int dimension, Topology& out);

// Fills out.bc_level from out.bc_ops and out.bc_start: each op's dependency
// level within its block (build_topology calls it).
void bc_levels(Topology& out);

// Host tables of the pipelined sweeps' order (PipeView) of one updated box cut
// along `dir` into `ce` slabs: the slabs' first planes, every plane's first
// position and node count; pmax the largest plane, lmax the largest message across a cut (nodes), hmax the most planes of a slab.
struct PipeTables {
  int dir = 0, ce = 1, pmax = 0, lmax = 0, hmax = 0;
  std::vector<int> slab;
  std::vector<PipePlane> plane;
};
PipeTables pipe_tables(const Box& b1, int dir, int ce);

// Slabs of a block at most.
constexpr int kPipeSlabs = 16;
// The direction to cut for clusters of ncta CTAs: the one whose slabs have the
// smallest largest plane (a cut of a short direction leaves every slab most of
// the block's planes, so that the CTAs all work most of the time; a cut of a
// long one leaves few and wide ones).
int pipe_direction(const Box& b1, int ncta);

// What a set of blocks asks of the pipelined sweeps on clusters of one size:
// the largest plane P, message L and slab H (planes), the most plane steps of
// both passes and the most slabs of a block.
struct PipeNeed {
  int P = 1, L = 1, H = 1, steps = 1, cuts = 1;
  void add(const Box& b1, int ncta);
};
// Their launch shape, ok false where a plane does not fit: threads and dynamic
// shared memory of a CTA; two: two CTAs per SM.
struct PipeLaunch {
  bool ok = false, two = false;
  PipeShape sh{};
  int threads = 0;
  size_t smem = 0;
};
// The mean flow's, for `ctas` CTAs in all on a device of `sms` SMs, and the SA
// equation's.
PipeLaunch pipe_launch(const PipeNeed& need, long ctas, int sms);
PipeLaunch pipe_sa_launch(const PipeNeed& need);

}  // namespace aero
