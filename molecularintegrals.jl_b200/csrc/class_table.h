// Generated by gen_eri.py from data/class_table_b200.json.  Do not edit.
// Default MOLINTS_METHOD_AUTO table of contexts on the device named below:
// autotune.tune_class_methods on B200 (bench.py): 8 molecules of the 256-molecule batch and 4 serving requests, each class pair's HGP and Rys kernels (FP64 and MIXED) timed alone; the d and f class pairs timed again with the column-per-thread Rys kernels on an 8-molecule FP64 batch, 16 serving requests and molecules of 8 and 11 atoms (us, HGP / Rys: (dd|dp) 314 / 46, (dd|pp) 185 / 56, (dd|ds) 139 / 46, (dp|pp) 245 / 107, (dp|ds) 144 / 109, (dd|ps) 74 / 78 and 41 / 22 on the 8-atom molecule).
// Entries: 1 HGP, 2 Rys, | 4 (MOLINTS_CLASS_NO_FP32) where MIXED runs the FP64 kernel.
#pragma once
#include <stdint.h>
namespace molints {
constexpr const char *kTunedDevice = "NVIDIA B200";
static const int32_t kTunedClassMethods[11][11] = {
    {5, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {5, 5, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {5, 5, 5, 0, 0, 0, 0, 0, 0, 0, 0},
    {5, 5, 5, 5, 0, 0, 0, 0, 0, 0, 0},
    {5, 5, 6, 6, 6, 0, 0, 0, 0, 0, 0},
    {5, 5, 5, 5, 6, 6, 0, 0, 0, 0, 0},
    {5, 6, 6, 6, 6, 6, 6, 0, 0, 0, 0},
    {5, 5, 6, 6, 6, 6, 6, 6, 0, 0, 0},
    {6, 6, 6, 6, 2, 6, 6, 6, 6, 0, 0},
    {5, 6, 6, 6, 6, 6, 6, 6, 6, 6, 0},
    {5, 2, 6, 6, 6, 6, 6, 6, 6, 6, 6},
};
// 1 where an AUTO plan's Rys kernel follows the Boys mode as the HGP kernel of the class pair does
// (RysTab::xmax = 30 in the reference mode): (dp|dp), (fp|pp) and (dd|dd) evaluate the exact function
// in either mode, and so do the class pairs without an HGP kernel.  For nine polarised atoms with f
// shells the two forms differ by up to 7.4e-12 in (dd|pp), 1.3e-12 in (dd|ps).
static const unsigned char kRysFollowsBoys[11][11] = {
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {0, 0, 1, 1, 0, 0, 0, 0, 0, 0, 0},
    {0, 0, 0, 0, 1, 1, 0, 0, 0, 0, 0},
    {0, 1, 1, 1, 1, 0, 0, 0, 0, 0, 0},
    {0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0},
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {0, 1, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
};
// work-queue schedule: lane_cost, hgp_widen, rys_chunks, rys_max_width, gather_blocks (autotune.tune_schedule on B200 (bench.py): a batch plan over 8 molecules of the 256-molecule batch, 54.8 ms with lane_cost 320 and 5 gather blocks per SM, 53.0 ms with this one)
static const double kTunedSchedule[5] = {640.0, 1.0, 4096.0, 8.0, 4.0};
}  // namespace molints
