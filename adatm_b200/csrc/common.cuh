// common.cuh -- shared definitions for the B200 AdaTM library.
//
// Device layout conventions used throughout:
//  * tensor indices are uint32 on the device (dims and nnz must stay below
//    2^32 - 1; the C-ABI rejects larger inputs with SPLATT_ERROR_BADINPUT);
//  * dense row matrices (factors, MTTKRP outputs, memo rows) are row-major
//    with a padded leading dimension ldr = round_up(R, 4) floats, so every
//    lane of a row group moves one 16-byte float4 (or 8-byte bf16x4);
//  * CSF levels follow the reference layout (include/splatt.h:235-287):
//    fptr[l] has nfibs[l]+1 entries and points into level l+1 (into the
//    nonzeros for l = N-2); fids[l] holds the index of every node, with
//    fids[0] kept explicitly (root ids) on the device.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "check.hpp"
#include "devmem.hpp"

namespace adatm {

constexpr int kMaxModes = 8;  // device kernels support orders 3..8

// SMs of a B200. Written out where work is split into chunks: the split, and
// with it the last bits of the sums, does not depend on what a device reports.
constexpr uint32_t kSms = 148;

inline int ldr_of(uint64_t R) { return (int)((R + 3) / 4 * 4); }

// (not volatile: a pure function of the lane, so the compiler may reuse it)
__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Exclusive device-wide prefix sum of n uint32 values (scan.cu). `tmp` must
// hold scan_tmp_words(n) uint32 of scratch. Values are summed in uint32.
size_t scan_tmp_words(size_t n);
void exclusive_scan_u32(const uint32_t *in, uint32_t *out, size_t n, uint32_t *tmp,
                        cudaStream_t stream);

}  // namespace adatm
