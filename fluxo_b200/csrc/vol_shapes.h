// Launch shapes of the Euler / Navier-Stokes volume kernel per N+1:
//   epb   elements per block;
//   lpw   lines per warp in the pair phase (0: lines contiguous in the thread index, needs N+1 | 32);
//         64/(N+1) for N+1 = 4, 6, 8 selects the kernel with two nodes of a line per thread;
//   minb  resident blocks per SM the register allocation must allow (0: 2 up to 512 threads, else 1);
//   ownsm 1: a thread reads its own node's record from shared memory in every round instead of
//         holding it in registers (fewer registers, more shared-memory loads).
// All shapes of one N add the same terms, the one-node ones also in the same order; they agree to roundoff
// and differ in occupancy, idle lanes, register spills and shared-memory traffic.  vol_shape_rule says which
// one a solve runs.
#pragma once

namespace fluxo {

struct VolShapeId {
  int epb, lpw, minb, ownsm;
};

constexpr int kVolShapeMax = 3;

// kVolShapes[NP][i]; an entry with epb 0 ends a list
constexpr VolShapeId kVolShapes[10][kVolShapeMax] = {
    {{0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}},    // NP 0 (unused)
    {{0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}},    // NP 1 (unused)
    {{32, 0, 0, 0}, {16, 0, 0, 0}, {0, 0, 0, 0}},  // NP 2: 256 / 128 threads
    {{8, 10, 0, 0}, {8, 8, 0, 0}, {4, 8, 0, 0}},   // NP 3: 256 / 512 / 256 threads
    {{4, 16, 4, 0}, {1, 16, 16, 0}, {2, 0, 0, 0}},  // NP 4: two nodes per thread, 128 / 32 threads; one, 128
    {{2, 6, 0, 0}, {2, 4, 0, 0}, {1, 4, 0, 0}},    // NP 5: 320 / 448 / 224 threads
    {{1, 10, 4, 0}, {2, 10, 2, 0}, {1, 5, 0, 0}},   // NP 6: two nodes per thread, 128 / 256 threads; one, 256
    {{1, 4, 0, 0}, {1, 4, 1, 0}, {1, 4, 0, 1}},    // NP 7: 416 threads; 1-block registers; own record in smem
    {{1, 8, 2, 0}, {1, 0, 0, 1}, {0, 0, 0, 0}},    // NP 8: two nodes per thread, 256 threads; one, 512
    {{1, 3, 0, 1}, {0, 0, 0, 0}, {0, 0, 0, 0}},    // NP 9: 864 threads
};

constexpr int vol_shape_count(int NP) {
  int c = 0;
  while (NP >= 0 && NP < 10 && c < kVolShapeMax && kVolShapes[NP][c].epb > 0) ++c;
  return c;
}

// The shape that a solve of nElems elements runs: a function of its configuration and size alone, so that its
// results do not depend on what else the process ran, nor on a timing.  A batch keeps solves of different
// shapes in different groups, so an instance runs the shape that it would run alone.
//
// us per step, best of repeated legs of the time loop, EC-KEP flux unless said:
//   N = 1: {16} as fast or faster at every size (40^3 Euler 636, {32} 662);
//   N = 2: {8,10} (27^3 Euler 605; {8,8} 717, {4,8} 730; at 4^3 84, 89, 83);
//   N = 4: {2,6} (16^3 Navier-Stokes 1065; {2,4} 1083, {1,4} 1305; at 4^3 158, 163, 155);
//   N = 6: {1,4} (13^3 Euler 779; {1,4,1} 1097, {1,4,0,1} 784; at 4^3 104, 102, 103);
//   N = 7: two nodes per thread (12^3 Navier-Stokes 1371, one node 1482; at 4^3 217, 210);
//   N = 5: two nodes per thread, {1,10,4} (14^3 Euler 579; {2,10,2} 581, one node 731), but one node, whose
//   chain per thread is shorter, below 4^3 elements (3^3 Euler 96, two nodes 112; at 4^3 98, 113);
//   N = 3: one node per thread, {2}, up to a few waves (8^3 Euler 88, two nodes 104); two nodes, {1,16,16},
//   above 2^20 nodes (40^3 Euler 2617, one node 2695; Kennedy-Gruber 2491, 2750; Navier-Stokes 5743, 5773),
//   and from 2^18 for Euler (20^3 407, 414).  Between, where launches start while the last wave of their
//   predecessor drains (pdl_mode), one node is faster for Navier-Stokes (20^3 858, 870) and for the longer
//   records of standard DG, dealiased metrics and Ducros (20^3 Euler 420, 479).
// On a few dozen elements some shapes are 2 to 10 % faster than the one that is best on many.  They are not
// used there: the small solves of a batch share a launch, and with shapes and groups of their own for up to
// 148 elements at N = 4, 5 and 7 a batch of 64 solves (4^3 to 16^3 elements) took 20.2 instead of 18.7 ms a step.
constexpr int vol_shape_rule(int NP, int VF, bool visc, int nElems) {
  if (NP == 4)
    return nElems > (1 << 14) || (nElems >= (1 << 12) && !visc && VF != 0 && VF != 1 && VF != 3) ? 1 : 2;
  return NP == 2 ? 1 : (NP == 6 && nElems < 64 ? 2 : 0);
}

}  // namespace fluxo
