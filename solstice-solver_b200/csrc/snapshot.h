/*
 * snapshot.h - a scene snapshot resident in device memory, for the
 * renderers (render.cpp). solve.cpp builds it with the same flattening,
 * index validation and device memory cache as a solve.
 */
#ifndef SSOL_B200_SNAPSHOT_H
#define SSOL_B200_SNAPSHOT_H

#include "device_scene.h"
#include "objects.h"

#define SSOL_SHARED_BUILD
#include "../../include/ssol_b200.h"

#include <cuda_runtime_api.h>

struct DeviceSnapshot {
  void* d_scene = nullptr;
  size_t alloc = 0; /* bytes of the device block */
  size_t bytes = 0; /* host -> device bytes */
  int precision = SSOL_B200_FP32;
  int features = 0; /* FEAT_* bits the scene needs */
  ssolb::DScene<float> s32{};
  ssolb::DScene<double> s64{};
};

/* Flatten `scn` in the precision and BVH leaf size of `options` (NULL =>
 * defaults; the launch shape fields are ignored), check it and upload it on
 * the device's stream. Needs the sun, its spectrum and DNI (RES_BAD_ARG),
 * not a sampled instance. `samples`: camera samples that will be traced, which
 * decide where the default builder builds the BVH. The 1080p field view takes
 * 3.8 ms as a draft of 4 samples and 9.5 ms path-traced with 16 on the host's
 * tree, 2.0 and 7.8 ms on the device's, which takes 2 ms less to build and
 * traces 5 % slower: 40 ms of tracing, about 2e8 samples, make up for it. */
res_T ssolb_snapshot_create
  (ssol_scene* scn, const ssol_b200_options* options, uint64_t samples, DeviceSnapshot& out);
void ssolb_snapshot_release(ssol_device* dev, DeviceSnapshot& s);

/* Device blocks through the per-device cache of solve.cpp */
cudaError_t ssolb_dev_alloc(ssol_device* dev, void** p, size_t bytes);
void ssolb_dev_free(ssol_device* dev, void* p, size_t bytes);

#endif /* SSOL_B200_SNAPSHOT_H */
