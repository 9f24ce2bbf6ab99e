// The rings of the fused quantized GEMM, tile by tile: plain constants, so that a program on the host can walk the kernel's waits.
#pragma once

struct TcConfig { int bn, kstep, stages, ncw; };
// the instantiated tile configurations (tl_variant p0..p3)
constexpr TcConfig kTcConfigs[] = {{192, 64, 6, 4}, {192, 64, 6, 8}, {128, 64, 8, 4}, {128, 64, 8, 8},
                                   {64, 128, 6, 8}, {32, 128, 8, 8}, {16, 128, 8, 8},
                                   {128, 128, 4, 8}, {192, 128, 3, 8}, {128, 128, 4, 16}, {192, 128, 3, 16},
                                   {64, 128, 6, 16}, {32, 128, 8, 16}};

struct TcRing {
  int slots;        // operand slots in TMEM: what two accumulators leave, no more than stages
  int groups;       // of converter warps, on k steps in turn
  bool slot_first;  // a converter waits for its slot before it reads the stage, not after
};
// A wait for a stage's load by the parity of its phase also passes while the load `stages` steps earlier is still out, so a converter
// may only ask for a stage once it knows that load to have landed.  One group has converted every step; of two, the one that asks has
// converted the earlier step itself if the ring is even.  On an odd ring the other group did: there the wait for the slot comes
// first.  It says that the products of step - slots have run, hence all loads up to that one, and slots <= stages.
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr TcRing tl_tc_ring(const TcConfig& c) {
  const int free_slots = (512 - 2 * c.bn) / (c.kstep / 2);
  const int groups = c.ncw == 16 ? 2 : 1;
  return TcRing{free_slots < c.stages ? free_slots : c.stages, groups, groups > 1 && c.stages % groups != 0};
}
