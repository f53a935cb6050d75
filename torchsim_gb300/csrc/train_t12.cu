// Instantiations of the recorded-train sweep (epg_train.cuh).
#include "epg_train.cuh"

namespace tsg {
const SweepEntry kTrainT12[] = {
    TSG_TRAIN_ENTRY(MODE_T12, 2, 5, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 2, 10, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 2, 16, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 4, 5, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 4, 4, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 4, 10, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 8, 4, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 4, 8, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 8, 8, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 4, 16, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 4, 32, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 10, 1, 3, 1),
    TSG_TRAIN_ENTRY(MODE_T12, 16, 1, 3, 1),
};
const int kTrainT12Count = sizeof(kTrainT12) / sizeof(kTrainT12[0]);
}  // namespace tsg
