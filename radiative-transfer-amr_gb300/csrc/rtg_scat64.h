// FP64 scattering product on the tensor cores (rtg_scat64.cu).
#pragma once

#include "rtg_internal.h"

namespace rtg {

struct Scat64;   // digits of W, thresholds and CTAs of one handle

// whether the column's product can run on the tensor cores (its FP32 sums stay exact)
bool scat64_fits(const ColDev& C);
// For the columns flagged in cols (each one fits): scls and thr are the
// drop-rule classes and thresholds per spatial node, d_thr their device copy,
// which must outlive the result.  nullptr when the digits cannot hold a W or
// there is no device memory for the tables.
Scat64* build_scat64(const rtg_handle* h, const std::vector<char>& cols, const uint8_t* scls, const uint64_t* thr,
                     const uint64_t* d_thr);
void free_scat64(Scat64* p);
// y += the off-diagonal scattering terms of the columns (nodes of classes 1 and 2)
void launch_scat64(const Scat64* p, const OpView<double>& v, uint32_t flags, const double* x,
                   double* y, cudaStream_t s);
// device flag: RTG_ERR_TIMEOUT once a wait of the kernel gave up
int* scat64_status(const Scat64* p);

}  // namespace rtg
