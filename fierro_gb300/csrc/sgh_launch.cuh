// Launches of a cycle that begin as the launch before them drains (programmatic
// dependent launch): a cycle of a small mesh is eight to ten kernels of a few
// microseconds each.  Included inside each unit's implementation namespace.
//
// Every kernel launched this way calls previous_launch_done() in every thread,
// before it returns and before it touches anything but the mesh's index lists
// (which no launch of a cycle writes).  It waits until the launch before has ended
// and its stores are visible, so launches take effect in their order as before
// (each one's end implies the end of all before it).  State is read with plain
// loads, never through the read-only path, whose data may not change while a
// kernel is resident.
//
// A cycle at 8^3 39.5 -> 37.3 us, 12^3 41.7 -> 40.6, 32^3 170.3 -> 169.5 (exact; graphs
// of four cycles on both sides).  Letting the next
// launch in any earlier (griddepcontrol.launch_dependents after the wait, or
// before the stores) was slower: blocks placed while the launch before them still
// holds its SMs crowd on few of them (12^3: 103 us, 32^3: 241 against 194).
#pragma once

__device__ __forceinline__ void previous_launch_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
static void launch(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
