"""The row buffers of prompt passes over several chunks: where the memory is not to be had prompts go chunk by chunk with the same bits, and the buffers give way
to whatever else the library has to allocate.  A stand-in for cudaMalloc plays a GPU whose memory is used up, and counts kernel launches."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

_FAKE = r"""
#include <dlfcn.h>
#include <map>
#include <mutex>
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
static std::map<void*, size_t> live;
static std::mutex mu;
static size_t used = 0, budget = ~(size_t)0, largest = 0;
static long launches = 0;
extern "C" {
int cudaMalloc(void** p, size_t n) {
    static auto f = (int (*)(void**, size_t))real("cudaMalloc");
    std::lock_guard<std::mutex> l(mu);
    if (used + n > budget) { f(p, (size_t)1 << 60); return 2; }   // the runtime records the error as it does for a GPU that is full
    const int rc = f(p, n);
    if (rc == 0) { live[*p] = n; used += n; if (n > largest) largest = n; }
    return rc;
}
int cudaFree(void* p) {
    static auto f = (int (*)(void*))real("cudaFree");
    { std::lock_guard<std::mutex> l(mu); auto i = live.find(p); if (i != live.end()) { used -= i->second; live.erase(i); } }
    return f(p);
}
int cudaLaunchKernelExC(const void* c, const void* k, void** a) {
    static auto f = (int (*)(const void*, const void*, void**))real("cudaLaunchKernelExC");
    launches++;
    return f(c, k, a);
}
size_t fake_used(void) { return used; }
size_t fake_largest(void) { const size_t n = largest; largest = 0; return n; }
void fake_budget(size_t b) { budget = b; }
long fake_launches(void) { const long n = launches; launches = 0; return n; }
}
"""

_SCRIPT = r"""
import ctypes as C
import sys
import numpy as np
import pyre_b200 as pb
from pyre_b200 import synth
from helpers import small_cfg
fake = C.CDLL(sys.argv[1])
for f in (fake.fake_used, fake.fake_largest): f.restype = C.c_size_t
fake.fake_launches.restype = C.c_long
fake.fake_budget.argtypes = [C.c_size_t]
NO = 2 ** 64 - 1
ctx = pb.Ctx(0)
cfg = small_cfg(pb, max_ctx=1400, kv_bits=4)
ids = np.random.default_rng(0).integers(0, cfg.vocab, 1024).astype(np.uint32)

def model():
    return synth.build_model(ctx, cfg, synth.model_spec(cfg, 12), 12)

def prompt(st):
    st.reset(); fake.fake_launches()
    return st.forward(ids), fake.fake_launches()

m = model()
fake.fake_largest()
st = m.new_state(1)
ws = fake.fake_largest()                     # the row buffers: by far the largest allocation of a state
shared, few = prompt(st)
assert fake.fake_largest() == 0              # a prompt allocates nothing
# switched off: a pass per chunk, same bits, memory back; on again: as before
u = fake.fake_used(); m.prompt_passes(False); assert fake.fake_used() == u - ws
by_chunk, many = prompt(st)
st.reset(); st.forward(ids)                  # (chunks are captured in graphs by now)
assert np.array_equal(shared.view(np.uint32), by_chunk.view(np.uint32)) and few < many, (few, many)
m.prompt_passes(True)
again, n = prompt(st)
assert fake.fake_used() == u and n == few and np.array_equal(again.view(np.uint32), shared.view(np.uint32)), (n, few)
# what needs memory gets the idle buffers': a state, a matrix; the prompt then goes by chunk, and passes are shared again once there is room
for need in (lambda: m.new_state(2).destroy(), lambda: pb.QMat.synth(ctx, pb.Q4_K, 4096, 2048, 0, 1).free()):
    fake.fake_budget(fake.fake_used() + (64 << 10))
    u = fake.fake_used()
    need()
    assert fake.fake_used() == u - ws
    fake.fake_budget(fake.fake_used() + (64 << 10))
    lg, _ = prompt(st)
    assert fake.fake_used() == u - ws and np.array_equal(lg.view(np.uint32), shared.view(np.uint32))
    fake.fake_budget(NO)
    lg, n = prompt(st)
    assert fake.fake_used() == u and n == few and np.array_equal(lg.view(np.uint32), shared.view(np.uint32)), (n, few)
# more than there is: refused as ever, and the next call finds no trace of the refusal
fake.fake_budget(fake.fake_used() + (64 << 10))
try:
    m.new_state(64); assert False
except pb.PyreError as e:
    assert e.status == pb.PB_ERR_OOM
lg, _ = prompt(st)
assert np.array_equal(lg.view(np.uint32), shared.view(np.uint32))
# a state made while there is no room for them works without, and with them later
m.prompt_passes(False); m.prompt_passes(True)
st.destroy(); m.destroy()
fake.fake_budget(NO)
m = model()
st = m.new_state(1); need = fake.fake_used()
st.destroy(); m.prompt_passes(False); m.prompt_passes(True); m.destroy()
m = model()
fake.fake_budget(need - ws // 2)
st = m.new_state(1)
assert fake.fake_used() < need - ws // 2
lg, _ = prompt(st)
assert np.array_equal(lg.view(np.uint32), shared.view(np.uint32))
fake.fake_budget(NO)
lg, n = prompt(st)
assert fake.fake_used() == need and n == few and np.array_equal(lg.view(np.uint32), shared.view(np.uint32))
assert ctx.device_status() == 0
st.destroy(); m.destroy(); ctx.close()
print("ok")
"""


def test_row_buffers_give_way(tmp_path):
    root = Path(__file__).resolve().parent
    (tmp_path / "fake.cpp").write_text(_FAKE)
    so = tmp_path / "fake.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(tmp_path / "fake.cpp"), "-ldl"], check=True)
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([str(root.parent), str(root), os.environ.get("PYTHONPATH", "")]), LD_PRELOAD=str(so))
    p = subprocess.run([sys.executable, "-c", _SCRIPT, str(so)], env=env, timeout=300, capture_output=True, text=True)
    assert p.returncode == 0 and p.stdout.strip().endswith("ok"), p.stderr[-2000:]
