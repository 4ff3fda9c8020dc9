"""The blocks per SM that the search kernels are laid out for, from ptxas's
report (no GPU): 15-puzzle rounds with tables hold 1024 threads per SM in blocks
of 128 or 256, all others 768, with table searches leaving 64 KB of the SM's
256 to L1."""
from test_kernel_resources import _args, _ptxas_report


def test_registers_and_shared_memory_of_the_planned_blocks():
    seen = 0
    for name, k in _ptxas_report().items():
        a = _args(name) if "search_round_kernel" in name else None
        if a is None:
            continue
        w, pdb, block, multi = a
        threads = 1024 if w == 4 and pdb and not multi else 768
        seen += 1
        assert threads * k["regs"] <= 65536, (a, k)
        assert threads // block * (k["smem"] + 1024) <= (192 if pdb else 228) * 1024, (a, k)
    assert seen == 16
