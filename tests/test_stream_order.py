"""Work of one handle on several streams: the ordering classes against a fake
of the CUDA calls that fails each of them in turn (on the CPU), and one handle
used from two streams (on the GPU)."""
import os
import subprocess

import numpy as np
import pytest

from cm_gb300 import FiniteElasticityEquationsSet
from cm_gb300 import mesh as M

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "cm_gb300", "csrc")

FAKE = r"""
#pragma once
#include <set>
enum cudaError_t { cudaSuccess, cudaErrorInvalidValue, cudaErrorUnknown };
enum { cudaEventDisableTiming = 2 };
typedef std::set<int> Work;
struct Stream { Work seen; };  // the work that a stream's next item comes after, its own included
struct Event { Work seen; };
typedef Stream* cudaStream_t;
typedef Event* cudaEvent_t;
inline int fail_at = -1, calls = 0;
inline Work done;  // what the host has waited for
inline cudaError_t call() { return calls++ == fail_at ? cudaErrorUnknown : cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) {
  if (cudaError_t r = call()) return r;
  *e = new Event;
  return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  if (cudaError_t r = call()) return r;
  e->seen = s->seen;
  return cudaSuccess;
}
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, int) {
  if (cudaError_t r = call()) return r;
  s->seen.insert(e->seen.begin(), e->seen.end());
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  done.insert(s->seen.begin(), s->seen.end());
  return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
"""

PROGRAM = r"""
#include <cstdio>
#include "fe_order.h"
static int items = 0;
static Work queued;
// an item of a use must come after every item of the uses before it
static bool queue(cudaStream_t s, const Work& before) {
  for (int w : before)
    if (!s->seen.count(w) && !done.count(w)) return false;
  s->seen.insert(items);
  queued.insert(items++);
  return true;
}
static cudaEvent_t order = nullptr;
// one use of the buffers: three parts on side streams, the last on st
static bool use(cudaStream_t st, cudaStream_t* side, cudaEvent_t* ev) {
  const Work before = queued;
  cmfe::HandleOrder o(st);
  if (o.begin(&order)) return true;
  cmfe::Fork fork(st);
  if (cudaEventRecord(ev[0], st)) return true;
  for (int c = 0; c < 3; ++c) {
    if (fork.add(side[c], ev[0], ev[c + 1])) return true;
    if (!queue(side[c], before)) return false;
  }
  return queue(st, before);
}
int main() {
  for (int n = -1;; ++n) {
    Stream a, b, s[3];
    Event e[4];
    cudaStream_t side[3] = {&s[0], &s[1], &s[2]};
    cudaEvent_t ev[4] = {&e[0], &e[1], &e[2], &e[3]};
    order = nullptr;
    queued.clear();
    done.clear();
    fail_at = n;
    calls = 0;
    if (!use(&a, side, ev) || !use(&b, side, ev) || !use(&a, side, ev) || !use(&b, side, ev)) {
      std::printf("out of order when call %d fails\n", n);
      return 1;
    }
    // what is left after the last use: everything is behind the streams the caller knows, or waited for
    for (int w : queued)
      if (!a.seen.count(w) && !b.seen.count(w) && !done.count(w)) {
        std::printf("work left behind when call %d fails\n", n);
        return 1;
      }
    if (n >= calls) return 0;
  }
}
"""


def test_order_survives_every_failing_call(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "t.cpp"), "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("nxi,dims,load", [(2, (4, 4, 4), False), (3, (9, 7, 8), True), (3, (12, 12, 12), False)])
def test_one_handle_on_two_streams(nxi, dims, load):
    """FP64 Jacobians and residuals of one handle queued on two streams in
    turn, without a wait between them, have the bits of calls made alone."""
    import torch
    m = M.regular_box(*dims, nxi_u=nxi, pressure="node" if nxi == 3 else "element", law=M.MR, materials=(2.0, 6.0))
    es = FiniteElasticityEquationsSet(m)
    if load:
        p = np.zeros((3, m.nu))
        p[2, m.node_ijk()[2] == 0] = 0.7
        es.set_surface_pressure(p)
    xs = [torch.from_numpy(M.deformed_state(m, stretch=1.05, noise=0.02, seed=k)).cuda() for k in (1, 2)]
    new = lambda n: torch.empty(n, dtype=torch.float64, device="cuda")  # noqa: E731
    out = [[new(es.nnz), new(es.ndofs), new(es.ndofs)] for _ in xs]

    def call(x, v, r, r2):
        es.jacobian_evaluate(x, v, r)
        es.residual_evaluate(x, r2)

    refs = []
    for x, o in zip(xs, out):
        call(x, *o)
        torch.cuda.synchronize()
        refs.append([t.clone() for t in o])
    streams = [torch.cuda.Stream() for _ in xs]
    for o in out:
        for t in o:
            t.fill_(float("nan"))
    torch.cuda.synchronize()
    for _ in range(10):
        for s, x, o in zip(streams, xs, out):
            with torch.cuda.stream(s):
                call(x, *o)
    torch.cuda.synchronize()
    for o, ref in zip(out, refs):
        assert all(torch.equal(a, b) for a, b in zip(o, ref))
