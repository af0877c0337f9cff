"""Kernels that start before the kernel ahead of them has ended (launch_after) read with __ldg only what no kernel
writes: offset tables, items, permutations.  The operands of contractions and assembles may still be under way."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'ccq_b200', 'csrc')
EARLY = {'gett_multi_kernel', 'gett_multi64_kernel', 'assemble_kernel', 'assemble_group_kernel'}
TABLES = {'multi.cu': {'it.am', 'it.ak', 'it.bn', 'it.bk', 'it.cm', 'it.cn'},
          'gett_tile.cuh': {'offk', 'offA_m', 'offB_n'},
          'kernels.cu': {'P'}}


def _read(name):
    return re.sub(r'//[^\n]*', '', open(os.path.join(CSRC, name)).read())


def test_which_kernels_start_early():
    seen = set()
    for name in os.listdir(CSRC):
        if not name.endswith('.cu'):
            continue
        text = _read(name)
        seen |= set(re.findall(r'launch_after\([^,]*, (\w+)', text)) - {'kernel'}
        if 'launch_after' in text and name == 'kernels.cu':   # through the lambdas of launch_assemble
            seen |= set(re.findall(r'(\w+_kernel)<', ' '.join(re.findall(r'go\(([^;]*)\);', text))))
    assert seen == EARLY


def test_only_tables_are_read_with_ldg():
    for name, tables in TABLES.items():
        text = _read(name)
        if name == 'kernels.cu':   # the assemble kernels
            text = text[text.index('void canonical_element('):text.index('int assemble_lanes(')]
        args = set(re.findall(r'__ldg\(\s*([\w.]+)', text))
        assert args and args <= tables, (name, args - tables)
