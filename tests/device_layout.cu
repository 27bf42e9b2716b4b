// Compile-time checks of device data that kernels read in wide words.
#include "svdag_device.cuh"

// item_ptr answers a bad handle with this item, which the edit phases read in 16-byte words.
static_assert(__alignof__(svdag::kZeroItem) >= 16, "read as uint4");
static_assert(sizeof(svdag::kZeroItem) >= 48, "three uint4 of an item");
