"""The rule that picks a volume launch's kernel and shape (csrc/dsem_shapes.h), compiled for the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dsem_b200", "csrc")
WIDE, GEN, GEN_WIDE, POINT = 5, 6, 7, -1


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    """shape([(G, diag, nel, ev, variant), ...]) -> the shapes."""
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("shapes")
    src, exe = d / "shapes.cpp", d / "shapes"
    src.write_text('#include <cstdio>\n#include "dsem_shapes.h"\nint main() {\n  int g, d, n, e, v;\n'
                   '  while (std::scanf("%d%d%d%d%d", &g, &d, &n, &e, &v) == 5)\n'
                   '    std::printf("%d\\n", dsem::vol_shape(g, d != 0, n, e != 0, v));\n}\n')
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(rows):
        text = "\n".join(" ".join(str(int(x)) for x in row) for row in rows)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, timeout=60)
        return [int(x) for x in out.stdout.split()]
    return run


@pytest.mark.parametrize("p", range(1, 9))
def test_explicit_shapes(shape, p):
    """Shapes 1..4 reach runs without a model and with Smagorinsky's at p = 4, 6, 8; entropy
    viscosity, general metrics and the other orders take the default for any variant."""
    G = p + 1
    for nel in (1, 200, 5000):
        for v in range(1, 5):
            plain, default = shape([(G, 1, nel, 0, v), (G, 1, nel, 0, 0)])
            assert plain == (v if p in (4, 6, 8) else default)
            ev, evd = shape([(G, 1, nel, 1, v), (G, 1, nel, 1, 0)])
            assert ev == evd
            gen, gend = shape([(G, 0, nel, 0, v), (G, 0, nel, 0, 0)])
            assert gen == gend


@pytest.mark.parametrize("ev", [0, 1])
def test_default_shape_at_p4(shape, ev):
    """p = 4, with a model as without: wide up to 2 elements per SM, four warps up to 4, two above."""
    rows = [(5, 1, n, ev, 0) for n in (1, 296, 297, 592, 593)]
    assert shape(rows) == [WIDE, WIDE, 3, 3, 0]


@pytest.mark.parametrize("p,limits", [(3, (0, 444)), (4, (148, 444)), (5, (296, 444)), (6, (0, 148))])
def test_shapes_of_full_metrics(shape, p, limits):
    """Small launches at p = 4, 5 run the kernel with a thread per point, then the wide shape."""
    point, wide = limits
    rows = [(p + 1, 0, n, ev, 0) for ev in (0, 1) for n in (max(point, 1), point + 1, wide, wide + 1)]
    assert shape(rows) == 2 * [POINT if point else GEN_WIDE, GEN_WIDE, GEN_WIDE, GEN]
