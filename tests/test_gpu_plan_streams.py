"""cuFFT plans that cannot be moved to another stream (an error code from a stand-in for
cufftSetStream, preloaded into a process of its own): no transform runs on a stream
other than the context's.  The call that needs the plan reports the error or does
without the move, and every call that returns has waited for the work queued before
it on its stream and gives what a fresh context gives, bit for bit."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int calls, fail_from, fail_to;
void shim_fail(int from, int to) { calls = 0; fail_from = from; fail_to = to; }
int cufftSetStream(int plan, void* stream) {
  static int (*real)(int, void*);
  if (!real) real = (int (*)(int, void*))dlsym(dlopen("libcufft.so.11", RTLD_LAZY | RTLD_NOLOAD),
                                               "cufftSetStream");
  calls++;
  if (calls >= fail_from && calls < fail_to) return 5; /* CUFFT_INTERNAL_ERROR */
  return real(plan, stream);
}
int shim_calls(void) { return calls; }
"""

CHILD = r"""
import ctypes, sys
import torch
from gse_b200 import workloads as W
from gse_b200.gse import Context, GseError
shim = ctypes.CDLL(sys.argv[1])
n, L, M = 300, 20.0, 20
x0 = torch.from_numpy(W.triplets(n, L, 3)).double().cuda()

def context():
    return Context(M, M, M, 2.0, 0.4, 3.0, 3.0, L, L, L, precision="fp64")

def moved(k):
    y = x0.clone()
    y[:, 0] += 0.25 * k
    return y

def forward(ctx, x, f, e):
    ctx.forward(n, x, f[0], f[1], f[2], energy_out=e)
    return torch.cat([e, f.reshape(-1)])

def buffers():
    return (torch.zeros(3, n, dtype=torch.float64, device="cuda"),
            torch.zeros(1, dtype=torch.float64, device="cuda"))

want = [forward(context(), moved(k), *buffers()) for k in range(10)]
# from the first, second, ... move on, for one, two or all further moves; the capture on
# the default stream makes two and the next direct call two
for explicit in (False, True):
    side = torch.cuda.Stream()
    for start in range(1, 5):
        for count in (1, 2, 100):
            ctx, x, (f, e) = context(), moved(0), buffers()
            torch.cuda.synchronize()
            errors = 0
            for k in range(10):
                if k == 2:
                    shim.shim_fail(start, start + count)
                    if explicit:
                        try:
                            ctx.set_stream(side.cuda_stream)
                        except GseError:
                            errors += 1
                if k == 6:
                    assert shim.shim_calls() > 0 or not explicit
                    shim.shim_fail(0, 0)
                with torch.cuda.stream(side if explicit and k >= 2 else torch.cuda.default_stream()):
                    torch.cuda._sleep(20000000)  # about 10 ms before the new positions are there
                    x.copy_(moved(k))
                    f.zero_()
                    try:
                        got = forward(ctx, x, f, e)
                    except GseError as err:
                        assert err.status == 3, err
                        errors += 1
                        continue
                    finally:
                        torch.cuda.synchronize()
                    assert torch.equal(got, want[k]), (explicit, start, count, k)
            shim.shim_fail(0, 0)
            assert count == 100 or errors <= 2, errors
            assert torch.equal(got, want[9])
print("plans ok")
"""


def test_plans_never_run_on_another_stream(tmp_path):
    c, so = tmp_path / "shim.c", tmp_path / "shim.so"
    c.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(c), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD, str(so)], cwd=root, text=True,
                       env=dict(os.environ, LD_PRELOAD=str(so)), capture_output=True, timeout=300)
    assert r.returncode == 0 and "plans ok" in r.stdout, r.stdout + r.stderr
