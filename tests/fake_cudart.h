// fake_cudart.h -- controls of tests/fake_cudart.cpp, a stand-in for the CUDA
// runtime that keeps "device" memory on the host and runs no kernel.  The
// library's own objects, linked with it, show on a machine without a GPU what
// their host side asks of the runtime and what it makes of a failed call.
#pragma once

#include <cstddef>
#include <string>
#include <vector>

namespace fake {

struct Launch {
    std::string kernel;      // its mangled name
    unsigned grid, block;    // along x
    std::vector<void *> args;
};
struct Fill {
    void *ptr;
    size_t bytes;
};

void reset();                              // empties the records, disarms failures
long calls();                              // calls that can fail, since reset()
void fail_call(long k);                    // the k-th of them fails (from 0)
void fail_launch(const char *kernel);      // the next launch of a kernel whose name holds this fails
bool failed();                             // whether the armed failure has happened
const std::vector<Launch> &launches();
const std::vector<Fill> &fills();          // memsets
int captures();                            // stream captures begun
void meet(int threads, int ms);            // a synchronisation waits until so many threads have come to one, or ms have passed

}  // namespace fake
