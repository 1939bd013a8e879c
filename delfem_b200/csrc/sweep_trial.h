// What the sweep autotuner makes of its candidates' trials (host only).
#pragma once
#include "dfm_b200.h"

namespace dfm {

struct SweepTrials {
  int err = DFM_OK;    // the tuning failed: an expired wait, ...
  float best = 1e30f;  // ms of the fastest candidate
  // Takes a trial's status and time; true if it is the fastest so far.  A candidate that cannot be launched is one
  // that cannot be had, not an error of the call that is being tuned for.
  bool note(int rc, float ms) {
    if (rc == DFM_ERR_UNSUPPORTED || rc == DFM_ERR_CUDA) return false;
    if (rc != DFM_OK) {
      if (err == DFM_OK) err = rc;
      return false;
    }
    if (!(ms < best)) return false;
    best = ms;
    return true;
  }
};

}  // namespace dfm
