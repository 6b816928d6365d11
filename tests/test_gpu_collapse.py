"""collapseKernel, which makes the library's wide nodes, against the host form of
the same rules (rt_collapse.cuh) that the CPU tests check. Needs a GPU.

Storage order differs between the two (and between runs), so the trees are
walked together from their roots: every node's grid, slots and planes and every
packed triangle have to be the same bytes."""
import ctypes as c
import subprocess

import numpy as np
import pytest

import scenes
from conftest import ROOT
from test_oracle_golden import GEOMETRY

pytestmark = pytest.mark.gpu

HERE = ROOT / 'tests' / 'hostcheck'
LIB = HERE / '_build' / 'libgpucollapse.so'
CSRC = ROOT / 'custom-ray-tracing-shader_b200' / 'csrc'


@pytest.fixture(scope='module')
def gc():
    sources = [HERE / 'gpu_collapse.cu', CSRC / 'rt_build.cu', CSRC / 'rt_memory.cu', *CSRC.glob('*.cuh')]
    if not LIB.exists() or any(p.stat().st_mtime > LIB.stat().st_mtime for p in sources):
        LIB.parent.mkdir(exist_ok=True)
        subprocess.run(['nvcc', '-O2', '--fmad=false', '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a',
                        '--shared', '-Xcompiler=-fPIC', str(HERE / 'gpu_collapse.cu'), '-o', str(LIB)], check=True)
    lib = c.CDLL(str(LIB))
    lib.gc_collapse.argtypes = [c.c_void_p, c.c_int, c.c_int, c.c_int, c.c_int] + [c.c_void_p] * 5
    return lib


def walk(wide, packed):
    """(node without its storage indices, its groups' triangles) in breadth-first order."""
    out, level = [], [0]
    while level:
        below = []
        for index in level:
            node = wide[index].copy()
            child, tri = int(node[4]), int(node[5])
            node[4:6] = 0
            meta = node[6:8].view(np.uint8)
            imask = int(node[3] >> 24)
            count = sum(bin(m >> 5).count('1') for m in map(int, meta) if m and m & 0x18 != 0x18)
            out.append(node.tobytes() + packed[tri:tri + count].tobytes())
            below += range(child, child + bin(imask).count('1'))
        level = below
    return out


@pytest.mark.parametrize('leaf', (1, 2, 4, 8))
@pytest.mark.parametrize('width,pieces', ((8, 1), (4, 1), (8, 3), (4, 8)))
def test_nodes_are_the_host_forms(gc, oracle, width, pieces, leaf):
    slivers = scenes.cornell_sphere()[0][:1500].copy()
    for axis, k in zip('xyz', (0.9, 0.8, 0.7)):
        slivers['edge1'][axis][::7] = k  # long diagonal edges: boxes that are mostly empty
    sphere = scenes.cornell_sphere()[0]
    sets = [GEOMETRY['overlap'], GEOMETRY['exponential'], GEOMETRY['scatter'], slivers]
    sets += [sphere[:n] for n in (1, 5, 33, 600)] + [sphere]
    split = 0
    for tris in sets:
        n = len(tris)
        linear = oracle.scene(tris).linear_triangles()
        wide = [np.zeros(((2 * pieces * n + 8), 20), np.uint32) for _ in range(2)]
        packed = [np.zeros((pieces * n, 12), np.uint32) for _ in range(2)]
        res = np.zeros(4, np.int32)
        assert gc.gc_collapse(linear.ctypes.data, n, width, pieces, leaf, wide[0].ctypes.data, packed[0].ctypes.data,
                              wide[1].ctypes.data, packed[1].ctypes.data, res.ctypes.data) == 0
        assert res[0] == res[2] and res[1] == res[3]
        assert walk(wide[0], packed[0]) == walk(wide[1], packed[1])
        split += int(res[1] > n)
    assert split > 0 or pieces == 1
