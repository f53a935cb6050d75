// Instantiations of the recorded-train sweep (epg_train.cuh).
#include "epg_train.cuh"

namespace tsg {
const SweepEntry kTrainT12BI[] = {
    TSG_TRAIN_ENTRY(MODE_T12BI, 2, 5, 15, 1),
    TSG_TRAIN_ENTRY(MODE_T12BI, 2, 10, 15, 1),
    TSG_TRAIN_ENTRY(MODE_T12BI, 2, 16, 15, 1),
    TSG_TRAIN_ENTRY(MODE_T12BI, 4, 5, 15, 1),
    TSG_TRAIN_ENTRY(MODE_T12BI, 4, 4, 15, 1),
    TSG_TRAIN_ENTRY(MODE_T12BI, 4, 10, 15, 1),
    TSG_TRAIN_ENTRY(MODE_T12BI, 4, 8, 15, 1),
    TSG_TRAIN_ENTRY(MODE_T12BI, 4, 16, 15, 1),
    TSG_TRAIN_ENTRY(MODE_T12BI, 4, 32, 15, 1),
};
const int kTrainT12BICount = sizeof(kTrainT12BI) / sizeof(kTrainT12BI[0]);
}  // namespace tsg
