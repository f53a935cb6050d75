// Instantiations of the recorded-train sweep (epg_train.cuh).
#include "epg_train.cuh"

namespace tsg {
const SweepEntry kTrainForward[] = {
    TSG_TRAIN_ENTRY(MODE_FORWARD, 2, 5, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 2, 10, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 2, 16, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 4, 5, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 4, 4, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 4, 10, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 8, 4, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 4, 8, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 8, 8, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 4, 16, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 4, 32, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 10, 1, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 16, 1, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 20, 1, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 32, 1, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 10, 2, 0, 1),
    TSG_TRAIN_ENTRY(MODE_FORWARD, 20, 2, 0, 1),
};
const int kTrainForwardCount = sizeof(kTrainForward) / sizeof(kTrainForward[0]);
}  // namespace tsg
