"""The likelihood setup's folded coefficients are written by every lane of a set's group into the one record in
shared memory, and lanes need not run in step.  Host threads stand in for the lanes: whatever order they run in,
the record has to be the one that a single lane leaves."""
import ctypes

import numpy as np

from hostcc import compile_host

CODE = r"""
#include "qcbc_device.cuh"
#include <atomic>
#include <thread>
using qcbc::PhdRec;
extern "C" int rec_bytes() { return (int)sizeof(PhdRec); }
// runs of two threads on one record that ended other than one lane's
extern "C" int differing(const void* start, double rdm, int runs) {
  PhdRec one, two;
  memcpy(&one, start, sizeof(one));
  qcbc::mix_phase(one, rdm, 1e-16, 1e-17, 0.3);
  std::atomic<int> turn{0}, ready{0}, done{0};
  int bad = 0;
  auto lane = [&](bool lead) {
    for (int k = 1; k <= runs; k++) {
      if (lead) {
        memcpy(&two, start, sizeof(two));
        ready = 0;
        done = 0;
        turn = k;
      }
      while (turn < k) std::this_thread::yield();
      ready++;
      while (ready < 2) std::this_thread::yield();
      qcbc::mix_phase(two, rdm, 1e-16, 1e-17, 0.3);
      done++;
      if (lead) {
        while (done < 2) std::this_thread::yield();
        bad += memcmp(&one, &two, sizeof(one)) != 0;
      }
    }
  };
  std::thread other(lane, false);
  lane(true);
  other.join();
  return bad;
}
"""


def test_lanes_out_of_step_leave_one_lanes_record(tmp_path):
    L = compile_host(str(tmp_path), CODE, "-O0", "-pthread")
    rec = np.random.default_rng(4).uniform(0.1, 3.0, size=L.rec_bytes() // 8)
    assert L.differing(rec.ctypes.data_as(ctypes.c_void_p), ctypes.c_double(1.7), 20000) == 0
