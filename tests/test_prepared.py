"""csrc/prepared.h, what an operator makes on first use, compiled with the host
compiler and given failures by hand: a shortage is tried again, an unsupported
variant is not, nothing is thrown through it, and threads that come together
prepare once."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cassert>
#include <new>
#include <thread>
#include <vector>
#include "prepared.h"
using hb::Prepared;
int main() {
  int calls = 0, cleared = 0;
  auto clear = [&]() { ++cleared; };
  auto gives = [&](hb_status st) { return [&calls, st]() { ++calls; return st; }; };
  Prepared p;
  // a shortage: refused this time, the pending error cleared, tried again
  assert(!p.ready(0, gives(HB_ERR_CUDA), clear) && calls == 1 && cleared == 1 && !p.has(0));
  assert(!p.ready(0, [&]() -> hb_status { ++calls; throw std::bad_alloc(); }, clear));
  assert(calls == 2 && cleared == 2 && !p.has(0));
  assert(p.ready(0, gives(HB_OK), clear) && calls == 3 && cleared == 2 && p.has(0));
  assert(p.ready(0, gives(HB_ERR_CUDA), clear) && calls == 3);
  // another variant: not built, once and for all; the first is untouched
  assert(!p.has(1) && !p.ready(1, gives(HB_ERR_UNSUPPORTED), clear) && calls == 4 && cleared == 3);
  assert(!p.ready(1, gives(HB_OK), clear) && calls == 4 && p.has(0) && !p.has(1));
  // threads
  for (int round = 0; round < 50; ++round) {
    Prepared q;
    std::atomic<int> made{0}, ok{0};
    std::vector<std::thread> t;
    for (int k = 0; k < 8; ++k)
      t.emplace_back([&]() {
        ok += q.ready(2, [&]() { ++made; return HB_OK; }, []() {});
      });
    for (auto& x : t) x.join();
    assert(made == 1 && ok == 8);
  }
  return 0;
}
"""


def test_prepared_once_or_tried_again(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread",
                           "-I", os.path.join(ROOT, "hedge_b200", "csrc"), str(src), "-o", str(exe)])
    subprocess.check_call([str(exe)], timeout=60)


@pytest.mark.gpu
@pytest.mark.parametrize("want_c", [False, True])
def test_first_adjoint_under_capture(cuda_device, want_c):
    """An operator's first adjoint call, captured: it cannot prepare (that
    allocates), so the CUDA-core kernels are recorded, and the fused stage is
    refused; the replay equals the prepared adjoint."""
    import numpy as np
    import torch
    import hedge_b200 as hb
    from hedge_b200 import _native
    m = hb.make_regular_rect_mesh((-1, -1), (1, 1), (7, 6), jitter=0.03, seed=1)
    d = hb.Discretization(m, order=4)
    comp = hb.VariableVelocityStrongWaveOperator(1.0 + 0.2 * d.nodes[:, 0] ** 2, 2).bind(d).compiled
    rng = np.random.default_rng(3)
    q, lam = (d.to_device(rng.uniform(-1, 1, (3, len(d)))) for _ in range(2))
    comp._adjoint_work()
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    other = lam.clone()
    with torch.cuda.graph(graph, stream=stream):
        got = comp.adjoint(lam, q=q, want_c=want_c)
        st = comp._lib.hb_adjoint_stage(
            comp._handle, 0.1, 0.2, 0.3, q.data_ptr(), lam.data_ptr(), other.data_ptr(), None,
            comp._coeff.data_ptr(), comp._adj_work.data_ptr(), stream.cuda_stream)
    assert st == _native.HB_ERR_UNSUPPORTED
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, comp.adjoint(lam, q=q, want_c=want_c)):
        if a is not None:
            assert float((a - b).norm()) <= 1e-13 * float(b.norm())
    comp.check()
