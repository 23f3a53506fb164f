"""The build: what the compiler made of the kernels, from the resource lines it printed when the objects were built, and the ABI
that the host module is tied to."""

import os
import re

import pytest

from linquant_b200 import build


def registers(src, kernel):
    path = os.path.join(build.OBJ, src + ".ptxas")
    if not os.path.exists(path):
        pytest.skip(f"{path} not there: the objects were built elsewhere")
    used, name = {}, None
    for line in open(path):
        if m := re.search(r"Function properties for (\S+)", line):
            name = m.group(1)
        elif (m := re.search(r"Used (\d+) registers", line)) and name:
            used[name] = int(m.group(1))
    return [r for n, r in used.items() if kernel in n]


@pytest.mark.parametrize("src,kernel,threads,ctas", [("lq_ssd", "ssd_state_passing_kernel", 256, 6)])
def test_ctas_per_sm(src, kernel, threads, ctas):
    """The kernel's time rests on this many CTAs on an SM (65 536 registers, dealt to warps in units of 8 per thread)."""
    regs = registers(src, kernel)
    assert regs and all(ctas * threads * ((r + 7) // 8 * 8) <= 65536 for r in regs), regs


def test_host_module_is_tied_to_its_torch(monkeypatch):
    import torch

    from linquant_b200 import _cabi

    build.build()
    obj = os.path.join(build.OBJ, "lq_host.o")
    assert not build._host_stale(obj) and _cabi.host().built_for == build.host_key()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".post1")
    assert build._host_stale(obj)  # the next build compiles it again, whatever the file times say
    monkeypatch.setattr(_cabi, "_host", None)
    with pytest.raises(_cabi.LinQuantError, match="build it with"):
        _cabi.host()
