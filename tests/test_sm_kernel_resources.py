"""Resources of the rounds' kernels that fill an SM with one block, from
ptxas's report (no GPU): all registers and shared memory of one SM at most,
and nothing spilled."""
import re

from test_kernel_resources import _ptxas_report


def test_one_block_fills_an_sm_without_spills():
    kernels = {n: k for n, k in _ptxas_report().items() if "search_sm_kernel" in n}
    assert len(kernels) == 4
    for name, k in kernels.items():
        w, pdb = (int(x) for x in re.search(r"search_sm_kernelILi(\d)ELb(\d)E", name).groups())
        threads = 768 if w == 5 and pdb else 1024
        assert threads * k["regs"] <= 65536, (name, k)
        assert k["smem"] + 1024 <= (164 if pdb else 228) * 1024, (name, k)
        assert k["spill"] == 0, (name, k)
