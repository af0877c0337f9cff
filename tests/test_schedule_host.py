"""The scheduled runs' host code on the CPU: the runtime's own source on host memory (schedule_host.cpp).

Contexts, offset tables and launches are built as on a GPU for systems whose intermediates no longer all fit the
accumulation buffers (so contractions that overwrite share launches too) and for small ones, checked element by
element.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
UNITS = ('kernels', 'dress', 'multi', 'split', 'crcc', 'ccsdt_layout')


@pytest.fixture(scope='module')
def ask(tmp_path_factory):
    from ccq_b200 import build
    objs = [os.path.join(build.HERE, '_build', u + '.cu.o') for u in UNITS]
    build.build(force=not all(map(os.path.exists, objs)))
    exe = str(tmp_path_factory.mktemp('schedule_host') / 'schedule_host')
    cuda = os.path.dirname(os.path.dirname(build.NVCC))
    subprocess.check_call(['g++', '-std=c++17', '-O1', '-w', '-I', os.path.join(cuda, 'include'),
                           os.path.join(HERE, 'schedule_host.cpp')] + objs + ['-o', exe, '-lpthread'])

    def run(line):
        r = subprocess.run([exe], input=line + '\n', capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr
        return r.stdout.strip()
    return run


def _sched(method, froz, occ_a, occ_b, orbs, rhf, active, deep):
    return f'sched {method} {froz} {occ_a} {occ_b} {orbs} {int(rhf)} {active[0]} {active[1]} {int(deep)}'


ALL = (-1, -1)


# systems at which an overwriting contraction with 128 < K <= 256 shares a launch (their counterparts on a GPU:
# test_gpu_schedule.py), and others around the limits: nothing overwrites, K just inside one half range
@pytest.mark.parametrize('method,froz,occ_a,occ_b,orbs,rhf,active', [
    ('CCSDt', 0, 5, 5, 20, False, (4, 7)),
    ('CCSDt', 0, 5, 5, 20, False, (3, 8)),
    ('CCSDT', 0, 6, 5, 21, False, ALL),
    ('CCSDT', 0, 7, 6, 19, False, ALL),
    ('CCSDT', 1, 7, 6, 22, False, ALL),
    ('CCSDTQ', 0, 5, 5, 15, False, ALL),
    ('CR-CC(2,3)', 0, 7, 7, 38, True, ALL),
    ('CR-CC(2,3)', 0, 12, 11, 33, False, ALL),
    ('CCSD', 0, 9, 9, 48, True, ALL),
    ('CCSDT', 0, 5, 5, 24, False, ALL),
])
def test_items_of_shared_launches(ask, method, froz, occ_a, occ_b, orbs, rhf, active):
    assert ask(_sched(method, froz, occ_a, occ_b, orbs, rhf, active, False)).startswith('ok')


@pytest.mark.parametrize('method,froz,occ_a,occ_b,orbs,rhf,active', [
    ('CCSD', 0, 2, 1, 4, False, ALL),
    ('CCSD', 1, 4, 3, 9, False, ALL),
    ('CCSD', 0, 3, 3, 33, False, ALL),      # dressing in two passes
    ('CCSDT', 0, 3, 2, 8, False, ALL),
    ('CCSDT', 0, 3, 3, 8, True, ALL),
    ('CCSDt', 0, 4, 3, 9, False, (2, 6)),   # pieces of one contraction share an output
    ('CCSDTQ', 0, 4, 3, 7, False, ALL),
    ('CR-CC(2,3)', 0, 3, 2, 7, False, ALL),
    ('CR-CC(2,3)', 1, 3, 3, 8, True, ALL),
])
def test_every_element_is_ordered(ask, method, froz, occ_a, occ_b, orbs, rhf, active):
    assert ask(_sched(method, froz, occ_a, occ_b, orbs, rhf, active, True)).startswith('ok')


def test_two_threads_read_one_context(ask):
    """Large pageable blocks go through pinned slots of the context: one copy at a time."""
    assert ask('copies') == 'ok'
