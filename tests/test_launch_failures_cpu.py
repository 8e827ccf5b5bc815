"""A launch that fails gives back what its function took.  A shim in front of the library stands in for its context and its
allocator (host memory, counted); there is no device for the process, so that every launch returns an error of its own accord."""
import os
import subprocess
import sys

import pytest

from tl_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include <cstdlib>
#include <dlfcn.h>
#include "layered_kernels.h"
static int live = 0;
namespace tlb {
static Context fake;
Context *ctx() { fake.sm_count = 148; fake.smem_optin = 227 << 10; return &fake; }
Storage *storage_alloc(size_t bytes) { Storage *s = new Storage(); s->ptr = malloc(256); s->bytes = bytes; live++; return s; }
void storage_release(Storage *s) { free(s->ptr); delete s; live--; }
tlb_status launch_prefill_attention_tc(const float *, const void *, const void *, float *, int, int, int, int, int, float);
}
using namespace tlb;
template <typename F> static F symbol(const char *name) { return (F)dlsym(dlopen(getenv("TLB_SO"), RTLD_NOW | RTLD_NOLOAD), name); }
// status of the call (0: it ran, which it must not), or minus the blocks it kept
extern "C" int run(const char *what)
{
    static float x[4096];
    tlb_status st = TLB_OK;
    live = 0;
    if (!strcmp(what, "prompt")) {
        auto f = symbol<decltype(&launch_prefill_attention_tc)>("_ZN3tlb27launch_prefill_attention_tcEPKfPKvS3_Pfiiiiif");
        st = f(x, x, x, x, 64, 4, 2, 128, 0, 0.1f);
    } else if (!strncmp(what, "latent", 6)) {
        MixLatent m = {};
        m.H = 2; m.D = 96; m.RD = 32; m.DV = 128; m.R = 128; m.ld = 160; m.max_seq = 256; m.window = 256; m.scale = 0.1f; m.eps = 1e-5f;
        m.cache = x; m.q = x; m.ldq = 256;
        auto f = symbol<decltype(&launch_latent_prompt)>("_ZN3tlb20launch_latent_promptERKNS_9MixLatentEiiiiiPvib");
        st = f(m, 0, what[6] == 's' ? 40 : 128, 0, 0, 1, x, 256, what[6] == 'f');
    }
    return live ? -live : (int)st;
}
"""
RUN = "import ctypes, os, sys\nL = ctypes.CDLL(os.environ['TLB_SO'])\nprint('kept', ctypes.CDLL(sys.argv[1]).run(sys.argv[2].encode()))"


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-O1", "-I", os.path.join(ROOT, "tl_b200", "csrc"), "-I", cuda, "-o", so, str(d / "shim.cpp"), "-ldl"])
    return so


@pytest.mark.parametrize("what", ["prompt", "latent", "latents", "latentf"])
def test_failed_launches_keep_nothing(shim, what):
    """The prompt attention of heads of 128; the expanded latent attention for tcgen05, for mma.sync (40 tokens) and in f32."""
    env = dict(os.environ, LD_PRELOAD=shim, TLB_SO=_lib.SO_PATH, CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, "-c", RUN, shim, what], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("kept "), r.stdout + r.stderr
    assert int(r.stdout.split()[1]) > 0, "blocks kept, or no error: " + r.stdout
