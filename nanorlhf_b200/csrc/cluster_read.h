// Reads of the shared memory of another block of the cluster.  Only reads: a block's memory is read behind a cluster barrier at which it has arrived with
// its data written, and in front of another without which it does not leave.
#pragma once
#include "common.cuh"

namespace nrl {

// four floats at the same place in the shared memory of the cluster's block `rank`
NRL_DEVICE float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
  return v;
}

}  // namespace nrl
