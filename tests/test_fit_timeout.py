"""A fit vector whose evaluation ran into a bounded device wait never yields a likelihood:
fitparam.cpp built for the host against a fake of the batched evaluation that returns a
status for each vector.
"""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from qlens_gb300 import abi

CSRC = os.path.join(abi.package_dir(), "csrc")
FAKE = r"""
#include "fitparam.cpp"
#include <string>
static int g_status[16], g_rc;
static std::string g_err;
namespace qlpix {
void set_error(const char*, const char* a, int) { g_err = a; }
int n_params_of(int) { return 7; }
int ctx_eval_batch(qlp_ctx*, const double*, const double*, const qlp_instance*, int n, qlp_result* out)
{
    for (int i = 0; i < n; i++) {
        memset(&out[i], 0, sizeof(out[i]));
        out[i].status = g_status[i];
        out[i].m2logev = 100.0 + i;
    }
    return g_rc;
}
}
extern "C" int fake_fit(const int* status, int rc, int n, double* ll, qlp_result* out)
{
    qlp_ctx c;
    c.lenses.resize(1);
    qlp_fit_param f;
    memset(&f, 0, sizeof(f));
    f.use_penalty_limits = 1;
    f.penalty_lo = 0;
    f.penalty_hi = 1;
    c.fit.assign(1, f);
    memcpy(g_status, status, sizeof(int) * n);
    g_rc = rc;
    std::vector<double> x(n, 0.5);
    return qlpix::fit_loglike_batch(&c, x.data(), n, ll, out);
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not shutil.which("g++") or not os.path.isdir(os.path.join(cuda, "include")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("fake")
    src, lib = str(d / "fake.cpp"), str(d / "fake.so")
    with open(src, "w") as f:
        f.write(FAKE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, "-I", os.path.join(cuda, "include"),
                           src, "-o", lib])
    return C.CDLL(lib)


def _run(fake, status, rc=0):
    n = len(status)
    ll, out = np.zeros(n), (abi.qlp_result * n)()
    r = fake.fake_fit((C.c_int * n)(*status), rc, n, ll.ctypes.data_as(C.POINTER(C.c_double)), out)
    return r, ll, [o.status for o in out]


def test_timed_out_vector_is_an_error_and_penalised(fake):
    r, ll, st = _run(fake, [0, 8, 0])
    assert r == 8 and st == [0, 8, 0]
    assert ll.tolist() == [50.0, 1e30, 51.0]


def test_other_statuses_as_before(fake):
    # not SPD, no source pixels: the evaluation's value; a rejected lens: the penalty
    r, ll, st = _run(fake, [0, 3, 4, 1], rc=1)
    assert r == 0 and st == [0, 3, 4, 1]
    assert ll.tolist() == [50.0, 50.5, 51.0, 1e30]
    assert _run(fake, [0, 0], rc=2)[0] == 2
