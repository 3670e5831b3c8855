// output.hpp -- the output pass's and the enstrophy's launches without their
// scratch and host sums (output.cu, enstrophy.cu), for callers that keep the
// partial sums' buffer and copy them together with the fields.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace vfb
{
// partial sums: 5 doubles per output block, 2 per enstrophy block
unsigned outputBlocks(unsigned long long N);
unsigned enstrophyBlocks(unsigned long long N);

int outputLaunch(int storage, const void* dist, unsigned long long N, const uint32_t* geo, const uint32_t* nX,
                 const uint32_t* nY, const uint32_t* nZ, const uint8_t* mask, int even, void* rho, void* vx, void* vy,
                 void* vz, double* partial, cudaStream_t s);
int enstrophyLaunch(int precision, const void* rho, const void* vx, const void* vy, const void* vz,
                    unsigned long long N, const uint32_t* geo, const uint32_t* nX, const uint32_t* nY,
                    const uint32_t* nZ, const uint32_t* neighborInverse, double* partial, cudaStream_t s);

// the sums of vfb_output_pass and the mean and count of vfb_enstrophy from host copies of the partial sums
void outputSums(const double* partial, unsigned blocks, double* out5);
void enstrophyMean(const double* partial, unsigned blocks, double* out2);
} // namespace vfb
