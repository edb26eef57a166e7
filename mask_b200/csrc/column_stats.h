// Column features of a packed matrix: the device part, which a caller can let run while it does something
// else, and the host part.
#pragma once

#include "mem.h"
#include "plan.h"

namespace mask {

class ColumnStatsJob {
public:
    // Enqueues the kernels and the copy of their results to the host.
    int enqueue(const int32_t* d_val_soff, const int32_t* d_val_sidx, int32_t M, int32_t K, int64_t T, int32_t N, cudaStream_t st);
    // On the device, after the kernels: 1 if plan->local will be set.
    const int32_t* device_local() const { return d_local_; }
    // After the stream has been synchronised.
    void finish(mask_column_features* out) const;

private:
    DevScratch buf_;
    HostStage host_;
    int32_t K_ = 0, N_ = 0, local_rows_ = 0, l2_ = 0;
    int64_t T_ = 0;
    const int32_t* d_local_ = nullptr;
};

// The plan table: sets the plan's kernel parameters from the features.
void choose_plan_parameters(mask_plan* plan, const mask_column_features& f);

}  // namespace mask
