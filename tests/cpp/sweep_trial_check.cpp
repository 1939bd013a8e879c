// The sweep autotuner's rule for its candidates' trials (delfem_b200/csrc/sweep_trial.h).
#include <cstdio>

#include "sweep_trial.h"

#define CHECK(c)                                                    \
  do {                                                              \
    if (!(c)) {                                                     \
      std::printf("line %d: %s\n", __LINE__, #c);                   \
      return 1;                                                     \
    }                                                               \
  } while (0)

int main() {
  dfm::SweepTrials t;
  CHECK(!t.note(DFM_ERR_CUDA, 0.1f) && t.err == DFM_OK);         // a launch that fails: the next candidate
  CHECK(!t.note(DFM_ERR_UNSUPPORTED, 0.1f) && t.err == DFM_OK);
  CHECK(t.note(DFM_OK, 2.0f) && t.best == 2.0f);
  CHECK(!t.note(DFM_OK, 3.0f) && t.best == 2.0f);
  CHECK(!t.note(DFM_ERR_CUDA, 1.0f) && t.best == 2.0f && t.err == DFM_OK);
  CHECK(t.note(DFM_OK, 1.5f) && t.best == 1.5f);
  CHECK(!t.note(DFM_WAIT_TIMEOUT, 1.0f) && t.err == DFM_WAIT_TIMEOUT);  // the tuning itself has failed
  CHECK(!t.note(DFM_ERR_NOMEM, 1.0f) && t.err == DFM_WAIT_TIMEOUT);     // the first error stays
  return 0;
}
