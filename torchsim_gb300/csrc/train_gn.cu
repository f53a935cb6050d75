// Instantiations of the recorded-train sweep (epg_train.cuh).
#include "epg_train.cuh"

namespace tsg {
const SweepEntry kTrainGN[] = {
    TSG_TRAIN_GN_ENTRY(2, 5, 1),
    TSG_TRAIN_GN_ENTRY(2, 10, 1),
    TSG_TRAIN_GN_ENTRY(2, 16, 1),
    TSG_TRAIN_GN_ENTRY(4, 5, 1),
    TSG_TRAIN_GN_ENTRY(4, 4, 1),
    TSG_TRAIN_GN_ENTRY(4, 10, 1),
    TSG_TRAIN_GN_ENTRY(4, 8, 1),
    TSG_TRAIN_GN_ENTRY(8, 8, 1),
    TSG_TRAIN_GN_ENTRY(4, 16, 1),
    TSG_TRAIN_GN_ENTRY(4, 32, 1),
    TSG_TRAIN_GN_ENTRY(10, 1, 1),
    TSG_TRAIN_GN_ENTRY(10, 2, 1),
};
const int kTrainGNCount = sizeof(kTrainGN) / sizeof(kTrainGN[0]);
}  // namespace tsg
