"""Memory of an FP64 operator's cached digits (csrc/digit_budget.h): the rule on its own, built with
the host compiler, and what changes of precision leave behind on the device."""
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "mpskit.jl_gb300", "csrc")

PROGRAM = r"""
#include "digit_budget.h"
using gb::digits_affordable;
int main() {
  const uint64_t G = 1ull << 30;
  // small sets are kept whatever is left
  if (!digits_affordable(gb::DIGITS_SMALL, 100 * G, 0, 0)) return 1;
  // what the solves need stays free, and as much again as the digits take
  if (!digits_affordable(4 * G, 16 * G, 24 * G, 0)) return 2;
  if (digits_affordable(4 * G, 16 * G, 24 * G - 1, 0)) return 3;
  if (digits_affordable(4 * G, 16 * G, 19 * G, 0)) return 4;
  if (digits_affordable(4 * G, 0, 3 * G, 0)) return 5;  // they do not even fit
  // the unused part of the pool counts for the digits, not for the solves
  if (!digits_affordable(4 * G, 16 * G, 20 * G, 4 * G)) return 6;
  if (digits_affordable(4 * G, 16 * G, 19 * G, 40 * G)) return 7;
  if (!digits_affordable(4 * G, 16 * G, 22 * G, 2 * G)) return 8;
  return 0;
}
"""


def test_rule(tmp_path):
    src, exe = tmp_path / "budget.cpp", tmp_path / "budget"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


@pytest.mark.gpu
def test_changes_of_precision_do_not_pile_up_digits():
    """FP64 to bf16x3 and back ten times: the planes of the constants stay with the operator (4
    bytes an entry and change), digits (14) must not."""
    import torch

    import mpsgb
    ctx = mpsgb.Context(0)
    D = 1024
    rng = np.random.default_rng(0)
    H = mpsgb.heisenberg_XXX(6, dtype=np.float64)
    n = np.asarray(H.W[2]).shape[0]
    G = rng.standard_normal((D, n, D))
    G[:, 0, :] = G[:, -1, :] = np.eye(D)
    dev = lambda k, a: mpsgb.DeviceTensor.from_numpy(ctx, k, a)
    x = dev("mps", rng.standard_normal((D, 2, D)))
    op = mpsgb.DerivativeOperator(ctx, mpsgb._lib.GB_HEFF_AC, dev("gl", G), H.device(ctx)[2], None,
                                  dev("gr", G), mpsgb.GB300Backend("fp64"))
    ref = op(x).numpy()

    def cycle():
        for p in ("bf16x3", "fp64"):
            op.set_precision(p)
            y = op(x)
        ctx.synchronize()
        return y

    cycle()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(10):
        y = cycle()
    entries = 2 * 2 * D * D  # both environments, two physical states
    assert before - torch.cuda.mem_get_info()[0] <= 10 * 8 * entries + (64 << 20)
    assert np.array_equal(y.numpy(), ref)
