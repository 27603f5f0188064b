"""The wave kernels' host code and the rules that both sides share, without a
GPU: programs compiled against wave_internal.h."""
import os
import subprocess

import pytest

from adds_b200 import build as B

CSRC = B.CSRC


def program(tmp_path, text, link=False):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(text)
    cmd = ["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(B.ROOT, "include"),
           "-I", os.path.join(B.CUDA_HOME, "include"), str(src), "-o", str(exe)]
    if link:
        cmd += ["-L", B.LIBDIR, "-ladds", "-Wl,-rpath," + B.LIBDIR]
    subprocess.run(cmd, check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return [int(x) for x in r.stdout.split()]


@pytest.mark.parametrize("tag_a,tag_b", [(0, 0), (8, 16), (0xFFFFFFF8, 8)])
def test_states_of_two_notes(tmp_path, tag_a, tag_b):
    """Error codes are numbers, not bits: two at once give the larger, and
    never a third."""
    got = program(tmp_path, '#include "wave_internal.h"\n#include <stdio.h>\n'
                  'static_assert(WV_ERR_OVERFLOW < WV_SETTLED && WV_ERR_TIMEOUT < WV_SETTLED &&\n'
                  '              WV_ERR_INPUT < WV_SETTLED && (2u * WV_SETTLED) == 1u << WV_NOTE_BITS, "");\n'
                  'int main() { for (unsigned a = 0; a < 8u; ++a) for (unsigned b = 0; b < 8u; ++b)\n'
                  f'  printf("%u\\n", wv_worse(a | {tag_a}u, b | {tag_b}u)); }}\n')
    want = [max(a & 3, b & 3) | ((a | b) & 4) for a in range(8) for b in range(8)]
    assert got == want


@pytest.mark.parametrize("shape", [0, 1, 2, 3])
def test_failed_layout_leaves_no_engine(tmp_path, shape):
    """A device that is not there: an engine that keeps its variant and number
    of queries without its memory would be taken for a whole one."""
    rc, nq, shape_left, queries, pointers, size = program(
        tmp_path, '#include "wave_internal.h"\n#include <stdio.h>\n'
        'int main() { WvEngine E; std::vector<WvQuery> q(1, WvQuery()); q[0].n = 10; q[0].m = 20;\n'
        f'  const int rc = wv_engine_alloc(E, -1, false, {shape}, 0, q, 0);\n'
        '  const int held = (E.qs != 0) + (E.order != 0) + (E.area != 0) + (E.ws != 0) +\n'
        '                   (E.st != 0) + (E.grp != 0) + (E.st_host != 0);\n'
        '  printf("%d %u %d %zu %d %zu\\n", rc, E.nq, E.shape, E.qs_host.size(), held, E.bytes); }\n',
        link=True)
    assert rc == -5
    assert (nq, shape_left, queries, pointers, size) == (0, -1, 0, 0, 0)
