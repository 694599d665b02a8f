"""The tensor-memory instructions of the .sync.aligned forms need a converged warp, which a
branch just before them does not promise: in every function that issues one, a __syncwarp()
comes first."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tensor_memory_instructions_follow_a_syncwarp():
    functions = 0
    for path in glob.glob(os.path.join(ROOT, "aether-core-engine_b200", "csrc", "*.cu*")):
        text = open(path).read()
        for m in re.finditer(r"^(?:template <[^\n]*>\n)?__device__[^{;]*\{.*?^\}", text,
                             re.M | re.S):
            at = re.search(r'"[^"]*tcgen05\.\w[^"]*\.sync\.aligned', m.group())
            if at is None:
                continue
            functions += 1
            assert "__syncwarp();" in m.group()[:at.start()], (path, m.group().split("(")[0])
    assert functions >= 10
