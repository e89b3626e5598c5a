// das_direct.h -- one-launch delay-and-sum for small real problems (das_direct.cu).
#pragma once
#include "core.h"
#include "das_problem.h"

namespace ffdas {

// Problems of at most this many units (voxels x channels x events x items)
// take the direct kernel when the planner chooses: single frames up to 2^25
// units (measured on B200: 15 us against 18-27 us staged for a 4.2e6-unit
// plane-wave frame, 39 us against 49 us at 2.7e7 units), batches up to 2^22
// (the staged batch tiles share each tap's delay over the items; the direct
// kernel only shares the geometry).
constexpr int64_t kDirectUnits = int64_t(1) << 25;
constexpr int64_t kDirectUnitsBatched = int64_t(1) << 22;

// Frames among them that are staged without a schedule: 2^24 units on 2^16 voxels
// fill the staged tiles.  Not two events, whose passes of four are half empty; and
// five or more only past the voxels that get eight threads each in the direct
// kernel's two waves (148 SMs x 2048 threads): with four its chains double.  Direct
// and staged, us per call: 400 x 256 pixels, 64 channels, 4 events 57 and 38; 96, 3:
// 71 and 52; 192, 1: 58 and 42; 48, 6: 64 and 46; 256 x 256, 128, 3: 51 and 42;
// 300 x 250, 48, 5: 33 and 46; 40, 6: 33 and 42; 63, 5: 41 and 53; two events, 300 x
// 250, 192 channels: 58 and 123 (windows that overflow); 400 x 256, 90: 49 and 52.
constexpr int64_t kFrameUnits = int64_t(1) << 24, kFrameVoxels = int64_t(1) << 16;
constexpr int64_t kEightThreadVoxels = int64_t(2) * 148 * 2048 / 8;
inline bool staged_frame(int64_t V, int S, int64_t units) {
    return units >= kFrameUnits && V >= kFrameVoxels && S != 2 && (S <= 4 || V > kEightThreadVoxels);
}

// Real channel data (f32, f16, bf16) into f32 output, dense.
bool direct_supported(const das_problem &pb, ffdas_datatype_t xt, ffdas_datatype_t ot, int kind);

ffdas_error_t launch_direct(ffdas_context &h, const das_problem &pb, ffdas_datatype_t xt, const void *x,
                            const float *srcpos, const float *srcdir, const float *dstpos, const float *offsets,
                            const float *weights, float *out, double beta, int beta_zero, int batch_tile,
                            int split_req);

}  // namespace ffdas
