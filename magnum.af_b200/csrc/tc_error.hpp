// What a tensor-core kernel does when one of its bounded waits gives up (umma.cu,
// conv.cu): its CTA leaves without storing, so its outputs keep their former values,
// and raises a flag of the device.  The flag is two words: one in device memory, which
// later kernels of the stream can look at, and one in mapped host memory, which the host
// reads after any synchronisation of the stream without a copy.
#pragma once
#include "common.cuh"

namespace mafb {

struct TcFlag {
    int up;      // the word in device memory
    int* host;   // device address of the host word
};

// (not inlined: in the kernels' last branch it cost k_conv<64> 1.5 %)
static __device__ __noinline__ void tc_raise(TcFlag* f) {
    atomicExch(&f->up, 1);
    *static_cast<volatile int*>(f->host) = 1;
    __threadfence_system();
}

// The current device's flag (in device memory), made on first use and kept for the process.
TcFlag* tc_flag();

// Throws MAF_ERR_TIMEOUT and lowers the flag if it is up.  Waits for the stream's work first
// when `wait` is set; else the caller has, or asks about earlier work only.
void tc_check(cudaStream_t st, bool wait);

}  // namespace mafb
