// Instantiations of the recorded-train sweep (epg_train.cuh).
#include "epg_train.cuh"

namespace tsg {
const SweepEntry kTrainT12B[] = {
    TSG_TRAIN_ENTRY(MODE_T12B, 2, 5, 7, 1),
    TSG_TRAIN_ENTRY(MODE_T12B, 2, 10, 7, 1),
    TSG_TRAIN_ENTRY(MODE_T12B, 2, 16, 7, 1),
    TSG_TRAIN_ENTRY(MODE_T12B, 4, 5, 7, 4),
    TSG_TRAIN_ENTRY(MODE_T12B, 4, 4, 7, 4),
    TSG_TRAIN_ENTRY(MODE_T12B, 4, 10, 7, 4),
    TSG_TRAIN_ENTRY(MODE_T12B, 4, 8, 7, 4),
    TSG_TRAIN_ENTRY(MODE_T12B, 4, 16, 7, 4),
    TSG_TRAIN_ENTRY(MODE_T12B, 4, 32, 7, 4),
    TSG_TRAIN_ENTRY(MODE_T12B, 10, 1, 7, 1),
};
const int kTrainT12BCount = sizeof(kTrainT12B) / sizeof(kTrainT12B[0]);
}  // namespace tsg
