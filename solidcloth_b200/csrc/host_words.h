// host_words.h — status words in this library's own host memory, one per device.
#pragma once

namespace sc {

// A kernel on device d writes its word, the call that launched it reads the same
// word: calls on different devices may overlap, so no two devices share one. A
// page of its own (it is registered with the driver as a whole), 64 bytes a word.
struct HostWords
{
    static constexpr int DEVICES = 64, STRIDE = 16;
    alignas(4096) int word[DEVICES * STRIDE];
    static bool has(int dev) { return dev >= 0 && dev < DEVICES; }
    int* of(int dev) { return word + dev * STRIDE; }
};

} // namespace sc
