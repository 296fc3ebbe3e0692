// Band-wise dedispersion (dedisperse_band.cu): host interface used by
// dedisperse.cu.
#pragma once
#include "vfrb_common.cuh"

namespace vfrb {

struct BandTables;

// Tables of the band kernel for the delay table h_off [ndm][nchan]; *out stays
// NULL when the kernel does not apply to it (too few trials, or trials that
// are not close to equally spaced).  VFRB_ERR_NOMEM when device memory runs out.
int band_create(BandTables** out, const int32_t* h_off, int ndm, int nchan);
void band_destroy(BandTables* t);
int band_launches(const BandTables* t);  // of a call

// The dedispersed series of one call (njobs == 0) or of the jobs of a batched
// launch (grid z = job; the fields of `a` that DdJob holds are ignored).
// *launched = 0 when the call's layout does not suit the kernel: nothing has
// been launched then.  give_up (FP32): waits for staged rows give up at once, and the
// call is flagged.
int band_launch(const BandTables* t, const vfrb_dd_args& a, const DdJob* jobs, int njobs, bool give_up,
                cudaStream_t s, int* launched);

}  // namespace vfrb
