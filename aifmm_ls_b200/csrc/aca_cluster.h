// aca_cluster.h -- how many CTAs the ACA gives a job.
#pragma once

constexpr int kAcaMaxCluster = 8;
// Two CTAs a job at least, up to eight while four of them a slot of the device (four CTAs
// on each of 148 SMs) are not reached.  Measured, whole assemblies with all levels at one,
// two, four and eight: depth 3 (128 and 32 jobs) 2.5, 1.16, 1.16, 1.07 ms; depth 4, 8 x 8
// nodes (512 ..) 19.6, 11.6, 10.5, 10.6 ms; depth 5 (2048 ..) 47.5, 31.7, 32.8, 38.3 ms.
// By the jobs of the whole level, not of one launch: the sums of a job's stopping rule run
// in an order that depends on the cluster, and a job must not depend on how many
// of its level's boxes share a launch.
inline int aca_cluster_size(long level_jobs) {
  constexpr long kCtas = 4 * (4 * 148);
  int size = kAcaMaxCluster;
  while (size > 2 && level_jobs * size > kCtas) size /= 2;
  return size;
}
