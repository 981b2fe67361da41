"""Sizes at which the kernels' 32-bit indexes end, on the CPU: the rules that keep larger grids away from
them are compiled from the engine's headers and compared with the indexes written out in Python."""
import os
import re
import subprocess


from totem_b200 import build

INT_MAX = 2 ** 31 - 1


def _run(tmp_path, body, lines, head=""):
    src, exe = tmp_path / "m.cpp", tmp_path / "m"
    src.write_text('#include <cstdio>\n#include "common.cuh"\n' + head + 'using namespace totem;\nint main() {\n' + body + "\n}\n")
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-I", build.INCLUDE, "-I",
                    os.path.join(build.CUDA_HOME, "include"), str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], input="\n".join(lines), capture_output=True, text=True, check=True).stdout.split()


def test_gridding_takes_only_grids_its_kernels_can_index(tmp_path):
    shapes = [(n, w, half) for n in (64, 400, 2048, 4096) for half in (0, 1)
              for w in (2, 30, 64, 4096, 2 ** 18 - 32, 2 ** 18 - 2, 2 ** 18, 2 ** 19 - 34, 2 ** 19, 2 ** 24 - 2, 2 ** 24,
                        2 ** 25, 2 ** 30, INT_MAX - 1)]
    out = _run(tmp_path, 'int n, w, half; while (std::scanf("%d %d %d", &n, &w, &half) == 3)'
                         ' std::printf("%lld %d\\n", grid_pitch(w, half), (int)grid_indexes_fit(n, w, half));',
               [f"{n} {w} {half}" for n, w, half in shapes])
    for (n, w, half), pitch, fits in zip(shapes, out[::2], out[1::2]):
        cols = w // 2 + 1 if half else w
        assert int(pitch) >= cols and int(pitch) % 16 == 0 and int(pitch) < cols + 16
        # the last fine row and the row past S's last, offset by a whole row
        largest = max((2 * n - 1) * int(pitch), n * int(pitch)) + int(pitch) - 1
        assert (fits == "1") == (largest < INT_MAX), (n, w, half)


def test_gridding_rule_is_asked_before_the_builder_is_planned():
    src = open(os.path.join(build.CSRC, "engine.cu")).read()
    plan = src[src.index("Status totem_session::plan_gridding"):]
    assert plan.index("grid_indexes_fit") < plan.index("grid_ok = true")


def test_element_loops_of_the_cufft_path_stay_within_an_item(tmp_path):
    # the loop headers of the element-wise kernels, run on the CPU for the last thread of the grid that
    # item_grid gives: every element it visits is its own, in order, below vol
    src = open(os.path.join(build.CSRC, "plain.cu")).read()
    heads = re.findall(r"for \(\w+ e = [^;]+;[^;]+; e \+= gridDim\.x \* blockDim\.x\)", src)
    grid = re.search(r"inline dim3 item_grid\(int vol, int items\) \{.*?\n\}", src, re.S).group(0)
    assert len(heads) == 2
    body = "int vol; while (std::scanf(\"%d\", &vol) == 1) {\n  const dim3 gridDim = item_grid(vol, 1);\n"
    for head in heads:
        body += ("  { const int w = 1; (void)w; const struct { unsigned x; } blockIdx{gridDim.x - 1}, blockDim{256}, "
                 "threadIdx{255};\n    long long at = (long long)blockIdx.x * 256 + 255, n = 0; bool ok = true;\n    "
                 + head + " { ok = ok && (long long)e == at && at < vol; at += 256LL * gridDim.x; if (++n > 8) break; }\n"
                 "    std::printf(\"%d\\n\", ok && n <= 4); }\n")
    text = body + "}"
    main = tmp_path / "head.h"
    main.write_text("#include <algorithm>\n#include <cuda_runtime.h>\n" + grid + "\n")
    sizes = [1, 2, 255, 1024, 1025, 304 * 304, 41472 ** 2, 46340 ** 2, INT_MAX - 1, INT_MAX]
    out = _run(tmp_path, text, [str(v) for v in sizes], '#include "head.h"\n')
    assert out == ["1"] * (2 * len(sizes)), list(zip(sizes, out[::2], out[1::2]))
