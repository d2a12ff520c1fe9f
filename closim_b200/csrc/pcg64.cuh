// The FP64 path's linear solve (pcg64.cu): launch plan and launcher.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "ordered_sum.cuh"
#include "plain.cuh"

namespace cs {

struct HostMesh;

constexpr int kPcg64T = 512;       // threads per CTA: two per vertex
constexpr int kPcg64Stages = 8;    // published stages per segment of an ordered sum
constexpr int kPcg64Rows = 12;     // rows of approximate segment sums

struct Pcg64Plan {
  int G = 0;         // CTAs
  int cluster = 0;   // 1: one thread-block cluster; 0: cooperative grid
  int nv = 0;        // vertices per CTA (contiguous)
  int R = 1;         // segments (ordering warps) per CTA
  int K = 1;         // terms per lane of a segment (odd: conflict-free shared reads)
  int NS = 0;        // G * R segments
  int offSmem = 0, vecSmem = 0, elemSmem = 0;  // whether the CTA's contact-record offsets / vectors / element
                                               // results fit in shared memory
  size_t smem = 0;
  size_t elemStride = 0;          // element results per CTA (doubles)
  const int* slotOff = nullptr;   // G + 1
  const int4* slots = nullptr;    // per CTA: its incident triangles (i0, i1, i2, triangle)
  const uint32_t* inc = nullptr;  // 3m, memRec's order: CTA slot << 2 | corner
  double* elem = nullptr;         // G * elemStride when not in shared memory
  OrdStage* heads = nullptr;      // 4 x NS: the first stage of each segment
  OrdStage* stages = nullptr;     // 4 x NS x kPcg64Stages: lists of more than one
  double* sums = nullptr;         // kPcg64Rows x NS
  double* curv = nullptr;         // barrier curvature per active contact
};

// The plan for `me` on a device with `sms` SMs; clusterMax: largest
// co-schedulable cluster (0: none). Without `lists` only the launch's shape.
struct Pcg64Host {
  Pcg64Plan p;
  std::vector<int> slotOff;
  std::vector<int4> slots;
  std::vector<uint32_t> inc;
};
void build_pcg64_plan(const HostMesh& me, int sms, int clusterMax, bool lists, Pcg64Host& out);
int pcg64_cluster_max();
int launch_pcg64(const Dev& d, const Pcg64Plan& p, int maxIters, double tol, cudaStream_t s);

}  // namespace cs
