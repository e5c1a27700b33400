// Page-locked staging of state transfers.
//
// A state that is read or written is two or three arrays.  Copied one by one
// from and to pageable memory each costs a transpose, a copy that the driver
// stages, and for a read a wait.  Here kernels move all arrays between the
// device's layout and page-locked memory that they address directly, half a
// block at a time, and the host copies the other half meanwhile.
// Measured array by array and staged:
//   a cloth's x, v and dv        write (us)      read (us)
//     8^2                         32 /   20       62 /   20
//    64^2      (144 KB)          100 /   31      101 /   35
//   128^2      (576 KB)           72 /   57      195 /   66
//   180^2      (1.1 MB)           90 /  102      319 /  110
//   383^2      (5.0 MB)          329 /  400      997 /  561
//   700^2      (17 MB)           955 / 1354    2,520 / 1,756
//  1024^2      (36 MB)         1,985 / 3,487   5,017 / 5,183
// A large write is bound by the host's copy, which the driver does faster; a
// large read by the new pages it touches.  So writes up to 768 KiB and reads up
// to 24 MiB come this way.
// The blocks are a pool of the process: a call takes one and gives it back
// before it returns, at most kKept lie idle, and the last object that may use
// the pool frees them.  So a new cloth's first transfer costs what a repeated
// one does (page-locked memory of its own: 17 ms for 12 MB).
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace b3g {

constexpr int kStageArrays = 3;

// One array: `words` 32-bit words on the host, and on the device the same words
// in order (planes = 0) or as three planes of `planes` = words / 3 (xyz triples).
struct StageArray {
    float* dev;
    void* host;
    uint32_t words;
    uint32_t planes;
};

// A member of every object that calls host_stage_copy.
struct HostStageUse {
    HostStageUse();
    ~HostStageUse();
    HostStageUse(const HostStageUse&) = delete;
    HostStageUse& operator=(const HostStageUse&) = delete;
};

// Moves the arrays (those whose host pointer is not null) to the host or to the
// current device, which `st` belongs to, and waits.  *taken is false, and nothing
// is done, where the stage is not for this call: too large, a host pointer the
// CUDA runtime knows (page-locked, managed or device memory, which a plain copy
// treats by its kind), or no page-locked memory to be had.
cudaError_t host_stage_copy(const StageArray (&arrays)[kStageArrays], bool to_host, cudaStream_t st, bool* taken);

}  // namespace b3g
