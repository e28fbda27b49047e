"""The option refill_idle: a value is the threshold of every kernel, all of
1..32 differ, and 0 leaves each kind of kernel its own (which the header
lisa_gb.h states)."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_one_value_is_every_kernels_threshold(tmp_path):
    src = tmp_path / "refill.cc"
    src.write_text('#include <cstdio>\n#include <initializer_list>\n#include "refill.h"\nusing namespace lisa;\nint main() {\n'
                   "  for (uint32_t k = 0; k <= 40; ++k)\n"
                   "    for (uint32_t own : {REFILL_TRACE, REFILL_NEE, REFILL_PATHS})\n"
                   '      std::printf("%u\\n", refill_idle_lanes(k, own));\n}\n')
    exe = str(tmp_path / "refill")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "lisa_gb300", "csrc"), str(src), "-o", exe], check=True)
    out = [int(x) for x in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()]
    rows = [tuple(out[i:i + 3]) for i in range(0, len(out), 3)]
    for k in range(1, 41):
        assert rows[k] == (min(k, 32),) * 3
    text = open(os.path.join(ROOT, "include", "lisa_gb.h")).read()
    doc = re.search(r"in every kernel; 0 = (\d+) in the\s+closest-hit kernel, (\d+) in the emitter search,\s+(\d+)", text)
    assert rows[0] == tuple(map(int, doc.groups()))
    # and the kernels' buffers are made by this rule alone
    wf = open(os.path.join(ROOT, "lisa_gb300", "csrc", "wavefront.cu")).read()
    assert re.findall(r"refill_busy_max = (.*);", wf) == ["32u - refill_idle_lanes(r.opts.refill_idle, own)"]
