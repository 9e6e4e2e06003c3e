"""A cooperative launch that the device refuses as too large is made again with fewer blocks, down to one (host
build with the launch and the error state faked)."""
from hostcc import compile_host

CODE = r"""
#define cudaGetLastError fake_last_error
#include <cuda_runtime.h>
#undef cudaGetLastError
static int cleared;
static cudaError_t cudaGetLastError() { cleared++; return cudaSuccess; }
#include "qcbc_coop.h"
// room: blocks that fit; other: an error of another kind at once.  Returns error | blocks << 16 | clears << 32
extern "C" long long run(int most, int room, int other) {
  cleared = 0;
  int tries = 0, ran = 0;
  const cudaError_t e = qcbc::launch_coop(most, [&](int blocks) -> cudaError_t {
    if (++tries > 64) return cudaErrorUnknown;
    if (other) return cudaErrorInvalidValue;
    if (blocks > room) return cudaErrorCooperativeLaunchTooLarge;
    ran = blocks;
    return cudaSuccess;
  });
  return (long long)e | (long long)ran << 16 | (long long)(tries - cleared) << 32;
}
extern "C" int too_large() { return (int)cudaErrorCooperativeLaunchTooLarge; }
extern "C" int invalid() { return (int)cudaErrorInvalidValue; }
"""


def test_shrinks_until_it_fits(tmp_path):
    L = compile_host(str(tmp_path), CODE)
    import ctypes
    L.run.restype = ctypes.c_longlong

    def run(most, room, other=0):
        r = L.run(most, room, other)
        return r & 0xffff, r >> 16 & 0xffff, r >> 32
    assert run(148, 148) == (0, 148, 1)
    assert run(148, 1000) == (0, 148, 1)
    assert run(148, 74) == (0, 74, 1)          # every refused try's error was cleared, the last try has none
    assert run(148, 20) == (0, 19, 1)
    assert run(148, 1) == (0, 1, 1)
    assert run(1, 1) == (0, 1, 1)
    assert run(148, 0) == (L.too_large(), 0, 1)     # nothing fits: the error is the caller's
    assert run(148, 0, 1) == (L.invalid(), 0, 1)
