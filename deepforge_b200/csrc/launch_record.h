// Launches written down for repetition. While a recorder is open on a thread, every kernel that thread's launchers send
// off is also copied (kernel, grid, argument bytes); a record can then be sent again on any stream without walking the
// launchers. An argument block is a function of the params and the pointers alone, so a record stands for exactly the
// call it was made from. Between the kernel library and the host library, which are built together; not part of the C ABI.
#pragma once

#include <cstddef>
#include <cstdint>
#include <memory>
#include <vector>

namespace dfgpu {

struct RecordedLaunch {
    const void* function;
    unsigned grid[3], block[3];
    unsigned cluster;                     // CTAs per cluster along x (0: none)
    std::size_t shared_bytes;
    std::vector<std::size_t> offsets;     // of the arguments in `arguments`
    std::unique_ptr<unsigned char[]> arguments;
};

struct LaunchRecord {
    int device = -1;
    std::vector<RecordedLaunch> launches;
};

int current_device();                        // the thread's CUDA device, -1 when there is none
void open_recorder(LaunchRecord* record);    // launches of this thread are written down from here on
void close_recorder();
int replay(const LaunchRecord& record, void* stream);   // 0 or a Status code, like the launchers

}  // namespace dfgpu
