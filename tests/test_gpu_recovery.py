"""After a kernel gave up a wait: the error is reported once, and whatever it may have left in the library's scratch is gone before the
next launch reads it.  The error word and the leftovers are put there from the host; no kernel gives anything up here.  And a launch
whose CTAs do not all start at once needs no such end."""
import ctypes as C
import os
import subprocess
import time

import numpy as np
import pytest

import tl_b200 as tl
from test_launch_plans_cpu import matvec_slices
from tl_b200 import _lib, build, synth

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PEEK = r"""
#include "tlb_internal.h"
extern "C" int *error_word() { return tlb::ctx()->err_flag; }
extern "C" unsigned long long slices(unsigned long long *bytes) { *bytes = tlb::ctx()->mv_part1_floats * 4; return (unsigned long long)tlb::ctx()->mv_part1; }
extern "C" unsigned long long counts(unsigned long long *bytes) { *bytes = tlb::ctx()->mv_cnt_n * 4; return (unsigned long long)tlb::ctx()->mv_cnt; }
"""

HOLD = r"""
__global__ void hold(unsigned long long ns)
{
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do { __nanosleep(10000); asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)); } while (t - t0 < ns);
}
static cudaStream_t stream;
extern "C" int hold_all_but(int free_sms, int ms)      // one CTA an SM, by its shared memory
{
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
    if (!stream) cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
    cudaFuncSetAttribute(hold, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 << 10);
    hold<<<sms - free_sms, 32, 200 << 10, stream>>>(1000000ull * ms);
    return (int)cudaGetLastError();
}
extern "C" int let_go() { return (int)cudaStreamSynchronize(stream); }
"""


@pytest.fixture(scope="module")
def hold(tmp_path_factory):
    tl.init()
    d = tmp_path_factory.mktemp("hold")
    (d / "hold.cu").write_text(HOLD)
    subprocess.check_call([build.NVCC, *build.FLAGS, "-shared", "-o", str(d / "hold.so"), str(d / "hold.cu")])
    return C.CDLL(str(d / "hold.so"))


@pytest.mark.parametrize("t,n,k,m,sms", [(synth.Q4_K, 250, 2560, 16, 6), (synth.Q8_0, 250, 2560, 5, 6), (synth.Q6_K, 250, 4096, 11, 6), (synth.Q4_0, 250, 8192, 8, 6),
                                         (synth.Q4_K, 2048, 2048, 1, 40), (synth.Q8_0, 2040, 5632, 1, 6), (synth.Q6_K, 4096, 4096, 1, 3), (synth.Q4_0, 4096, 14336, 1, 100),
                                         (synth.Q4_K, 2048, 4096, 3, 6), (synth.Q8_0, 2048, 2048, 100, 12)])
def test_beside_a_kernel_that_holds_the_sms(hold, t, n, k, m, sms):
    """On a few SMs the CTAs that are there cannot wait for the others, which start when they have ended: 5 to 16 rows with one group of
    tiles in 10 to 32 pieces, one row in K slices, the forms for other rows.  The kernel beside them holds the other SMs for longer
    than any wait of the library."""
    assert m != 1 or matvec_slices(t, n, k, 1) > 1
    rng = np.random.default_rng(60 + t)
    q = tl.QTensor.from_gguf_bytes(t, n, k, synth.random_quant(t, n, k, rng))
    x = tl.Tensor.from_numpy(rng.standard_normal((m, k), dtype=np.float32))
    want = x.matmul_quantized(q).numpy()
    assert hold.hold_all_but(sms, 1500) == 0
    time.sleep(0.02)
    began = time.monotonic()
    got = [x.matmul_quantized(q) for _ in range(3)]
    tl.sync()
    took = time.monotonic() - began
    assert hold.let_go() == 0
    for g in got:
        np.testing.assert_array_equal(g.numpy().view(np.uint32), want.view(np.uint32))
    assert took < 1.0


@pytest.fixture(scope="module")
def peek(tmp_path_factory):
    tl.init()
    d = tmp_path_factory.mktemp("peek")
    (d / "peek.cpp").write_text(PEEK)
    so = str(d / "peek.so")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "tl_b200", "csrc"), "-I", cuda, "-o", so, str(d / "peek.cpp"), _lib.SO_PATH])
    L = C.CDLL(so)
    L.error_word.restype = C.POINTER(C.c_int)
    L.slices.restype = L.counts.restype = C.c_uint64
    return L


@pytest.mark.parametrize("m", [1, 3, 8, 40])
def test_leftovers_of_an_abandoned_launch(peek, m):
    """2048 x 4096 Q8_0: one row folds slices that rest at a sentinel, three rows and eight count theirs, forty take the tensor cores."""
    drv = C.CDLL("libcuda.so.1")
    rng = np.random.default_rng(40 + m)
    q = tl.QTensor.from_gguf_bytes(synth.Q8_0, 2048, 4096, synth.random_quant(synth.Q8_0, 2048, 4096, rng))
    x = tl.Tensor.from_numpy(rng.standard_normal((m, 4096), dtype=np.float32))
    want = x.matmul_quantized(q).numpy()
    for _ in range(3):
        tl.sync()
        for area, value in ((peek.slices, 0x3F800000), (peek.counts, 1)):
            size = C.c_uint64()
            at = area(C.byref(size))
            assert drv.cuMemsetD32_v2(C.c_uint64(at), C.c_uint(value), C.c_size_t(size.value // 4)) == 0
        assert drv.cuCtxSynchronize() == 0
        peek.error_word()[0] = 2
        with pytest.raises(tl.TlbError, match="code 2"):
            tl.sync()
        got = [x.matmul_quantized(q) for _ in range(4)]
        tl.sync()
        for g in got:
            np.testing.assert_array_equal(g.numpy().view(np.uint32), want.view(np.uint32))
