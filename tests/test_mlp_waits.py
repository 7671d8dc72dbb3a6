"""After a tensor-core wait that ran out the network's forward kernel, which goes on through its tiles
(its warpgroups share no barrier to leave them by), issues no more products: they would read operand
tiles that are being overwritten and write tensor memory that is about to be given back.  The gradient
kernel ends with the tile, at the check all its threads make.  (A wait does not run out on a working
GPU, so the rule is checked in the source.)"""
import os
import re

CUH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "akuaengine_gb300",
                   "csrc", "mlp.cuh")


def test_products_are_issued_only_while_no_wait_has_run_out():
    with open(CUH) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    forward, gradient = (text[text.index("k_mlp_forward("):text.index("struct GradSmem")],
                         text[text.index("k_mlp_grad("):])
    guards = [m for m in re.finditer(r"if \(t == 0([^(){};]*)\)\s*(\{[^}]*\}|[^;{]*;)", forward)
              if "tc::mma_" in m.group(2)]
    assert len(guards) == 2 == forward.count("tc::mma_commit(")
    assert all(m.group(1).strip() == "&& ok" for m in guards)
    assert re.search(r"ok = __syncthreads_and\(ok\);\s*if \(!ok\) break;", gradient)
