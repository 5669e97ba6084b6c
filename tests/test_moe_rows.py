"""Box heights of a prepared layer's weight maps (csrc/moe_rows.h, plain C++): each kernel's own choice, against a search here."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NSM = 148
Rs = range(32, 129, 8)


def heights(tmp_path, shapes):
    src, exe = tmp_path / 'rows.cpp', tmp_path / 'rows'
    src.write_text('#include "moe_rows.h"\n#include <cstdio>\n#include <cstdlib>\nint main(int n, char** a) {\n'
                   '  for (int i = 1; i + 4 < n; i += 5) { auto v = [&](int k) { return atoi(a[i + k]); };\n'
                   '    auto r = b200::moe_rows(v(0), v(1) != 0, v(2), v(3), v(4), %d);\n'
                   '    printf("%%d %%d %%d %%d\\n", r.stream_gu, r.stream_d, r.chunk_gu, r.chunk_d); }\n}\n' % NSM)
    subprocess.check_call(['g++', '-std=c++17', '-I', os.path.join(ROOT, 'glm-5.3-flash-cuda-server_b200', 'csrc'), str(src), '-o', str(exe)])
    out = subprocess.run([str(exe)] + [str(v) for s in shapes for v in s], capture_output=True, text=True, check=True).stdout
    return [tuple(map(int, line.split())) for line in out.split('\n') if line]


def cost(R, jobs, N, boxes):
    return -(-jobs * -(-N // (boxes * R)) // NSM) * (R + 40)


def stages(R, K):
    """Stages of packed weights that fit beside the digits of 8 rows and the scale rows of a box (gemv_umma.cu)."""
    return min(5, K // 256, (221 * 1024 - K // 256 * 8192 - R * (K // 16)) // (-(-R * 128 // 1024) * 1024))


def test_each_kernel_gets_the_heights_of_its_own_items(tmp_path):
    shapes = [(topk, sh, E, H, I) for topk in (1, 2, 4, 8, 16) for sh in (0, 1) for E in (16, 100, 144) for H in (256, 1024, 2048, 4096, 6144)
              for I in (256, 1024, 1536, 2048, 4096)]
    for (topk, sh, E, H, I), (sg, sd, cg, cd) in zip(shapes, heights(tmp_path, shapes)):
        ns, jobs = topk + sh, round(E * (1 - (1 - topk / E) ** 12)) + 2 * sh
        assert cost(sg, ns, I, 1) == min(cost(R, ns, I, 1) for R in Rs)
        assert cost(sd, ns, H, 2) == min(cost(R, ns, H, 2) for R in Rs)
        for R, n, N, K in ((cg, 2 * jobs, I, H), (cd, jobs, H, I)):
            deepest = max(stages(r, K) for r in Rs)
            assert stages(R, K) == deepest                       # no height at the price of a stage
            top = max(r for r in Rs if stages(r, K) == deepest)
            assert R <= top and cost(R, n, N, 1) == min(cost(r, n, N, 1) for r in Rs if r <= top)


def test_chunks_of_eight_rows_take_tall_boxes(tmp_path):
    """Where the persistent kernel's boxes are half as high as the chunks want them."""
    got = heights(tmp_path, [(8, 1, 144, 2048, 1536), (4, 1, 100, 3072, 1536), (8, 1, 144, 4096, 1024), (1, 0, 2, 4096, 1536)])
    assert [g[2:] for g in got[:3]] == [(128, 128), (128, 128), (104, 128)]
    assert (got[0][1], got[1][0], got[2][0]) == (64, 56, 64)
    assert got[3][2] < 104 and got[3][3] < 128                   # two experts: lower boxes, so that more SMs have one
