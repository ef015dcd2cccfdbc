"""Host side of the decode chain (CPU): which graphs a call queues, and that it goes on where a graph of several tokens cannot be had.

The library's calls of the CUDA runtime go to a stand-in, preloaded into a child process, that counts the kernels of each graph and each graph
that is launched, and refuses to instantiate a graph of more than ``limit`` kernels.  No GPU is involved."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
STAND_IN = r"""
#include <stdlib.h>
static int capturing, kernels, limit, n_log, n_refused, record[4096];
void fake_limit(int n) { limit = n; }
int fake_refused(void) { int n = n_refused; n_refused = 0; return n; }
int fake_log(int* out) { int n = n_log; for (int i = 0; i < n; ++i) out[i] = record[i]; n_log = 0; return n; }
static int tensor_map(void) { return 0; }
int cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long flags, int* found) { *f = (void*)tensor_map; if (found) *found = 0; return 0; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int a, int d) { *v = 148; return 0; }
int cudaFuncSetAttribute(const void* f, int a, int v) { return 0; }
int cudaGetLastError(void) { return 0; }
const char* cudaGetErrorName(int e) { return "fake"; }
const char* cudaGetErrorString(int e) { return "fake"; }
int cudaEventCreateWithFlags(void** e, unsigned f) { *e = malloc(1); return 0; }
int cudaEventDestroy(void* e) { free(e); return 0; }
int cudaEventRecord(void* e, void* s) { return 0; }
int cudaEventSynchronize(void* e) { return 0; }
int cudaStreamCreateWithFlags(void** s, unsigned f) { *s = malloc(1); return 0; }
int cudaStreamDestroy(void* s) { free(s); return 0; }
int cudaStreamWaitEvent(void* s, void* e, unsigned f) { return 0; }
int cudaStreamIsCapturing(void* s, int* st) { *st = 0; return 0; }
int cudaStreamBeginCapture(void* s, int mode) { capturing = 1; kernels = 0; return 0; }
int cudaStreamEndCapture(void* s, void** g) { capturing = 0; *g = malloc(sizeof(int)); *(int*)*g = kernels; return 0; }
int cudaLaunchKernelExC(const void* cfg, const void* f, void** args) { if (capturing) ++kernels; return 0; }
int cudaLaunchKernel(void) { if (capturing) ++kernels; return 0; }
int cudaGraphInstantiate(void** x, void* g, unsigned long long flags) {
    if (*(int*)g > limit) { ++n_refused; return 2; }
    *x = malloc(sizeof(int)); *(int*)*x = *(int*)g;
    return 0;
}
int cudaGraphDestroy(void* g) { free(g); return 0; }
int cudaGraphExecDestroy(void* x) { free(x); return 0; }
int cudaGraphLaunch(void* x, void* s) { if (n_log < 4096) record[n_log++] = *(int*)x; return 0; }
"""
# calls: [limit of kernels a graph, steps].  Prints for each [return code, kernels of the graphs launched, graphs refused].
CHILD = r"""
import ctypes as C, importlib.util, json, sys
spec = importlib.util.spec_from_file_location("binding", sys.argv[1])
B = importlib.util.module_from_spec(spec); spec.loader.exec_module(B)
lib, fake = B.lib(), C.CDLL(None)
plan = C.c_void_p()
assert lib.ittai_qwen3_chain_create(C.byref(plan)) == 0
p = B.Qwen3Decode()
p.n_layers, p.vocab, p.kv_cap, p.batch, p.eps, p.write_logits = 1, 512, 8192, 1, 1e-6, 1
for i, (name, kind) in enumerate(B.Qwen3Decode._fields_):
    if kind is C.c_void_p and name not in ("forced", "step_ns", "phase_clk"):
        setattr(p, name, 4096 * (i + 1))
out, log = [], (C.c_int * 4096)()
for limit, steps in json.loads(sys.argv[2]):
    p.n_steps = steps
    fake.fake_limit(limit)
    rc = lib.ittai_qwen3_chain_run(plan, C.byref(p), 60, None)
    out.append([rc, log[:fake.fake_log(log)], fake.fake_refused()])
assert lib.ittai_qwen3_chain_destroy(plan) == 0
print(json.dumps(out))
"""
TOKEN = 7                       # kernels of a token: five of the one layer, head, finish
ANY, ONE, NONE = 1000, TOKEN, 0


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("stand_in")
    (d / "fake.c").write_text(STAND_IN)
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-o", str(d / "fake.so"), str(d / "fake.c")], check=True)

    def f(calls):
        r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "ittai_b200", "_C.py"), json.dumps(calls)], capture_output=True, text=True, timeout=120,
                           env={**os.environ, "LD_PRELOAD": str(d / "fake.so")})
        assert r.returncode == 0, r.stderr
        return [tuple(x) for x in json.loads(r.stdout)]
    return f


def test_a_long_call_takes_graphs_of_four_from_its_17th_token_on(run):
    assert run([(ANY, 26)]) == [(0, [TOKEN] * 16 + [4 * TOKEN] * 2 + [TOKEN] * 2, 0)]


def test_a_graph_of_four_that_cannot_be_had_is_no_error_of_the_call(run):
    """Not in the middle of a long call, which tries once, and not behind a call; the next long call tries again."""
    first, second, third = run([(ONE, 40), (ONE, 24), (ANY, 24)])
    assert first == (0, [TOKEN] * 40, 1) and second == (0, [TOKEN] * 24, 1)
    assert third == (0, [TOKEN] * 16 + [4 * TOKEN] * 2, 0)
    assert run([(NONE, 4)])[0][0] != 0                                  # the graph of one token has to be had


def test_short_calls_get_the_graph_behind_one_of_them(run):
    """From 64 tokens of a kind on, behind a call of eight or more; refused there, it is tried again 64 tokens later."""
    assert run([(ANY, 8)] * 9) == [(0, [TOKEN] * 8, 0)] * 8 + [(0, [4 * TOKEN] * 2, 0)]
    got = run([(ONE, 8)] * 8 + [(ANY, 8)] * 9)
    assert got[:7] == [(0, [TOKEN] * 8, 0)] * 7 and got[7] == (0, [TOKEN] * 8, 1)
    assert got[8:16] == [(0, [TOKEN] * 8, 0)] * 8 and got[16] == (0, [4 * TOKEN] * 2, 0)
    assert run([(ANY, 4)] * 20 + [(ANY, 8)] * 2) == [(0, [TOKEN] * 4, 0)] * 20 + [(0, [TOKEN] * 8, 0), (0, [4 * TOKEN] * 2, 0)]
