"""Instructions that a whole warp has to reach at once (.aligned cluster barriers, giving TMEM back) stand behind __syncwarp() and in no
other place than their helpers."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "csrc"
ALIGNED = r"barrier\.cluster\.arrive|tcgen05\.dealloc"


def test_the_warp_meets_first():
    seen = 0
    for path in sorted([*CSRC.glob("**/*.cu"), *CSRC.glob("**/*.cuh"), *CSRC.glob("**/*.h")]):
        code = re.sub(r"//[^\n]*", "", path.read_text())
        assert "cluster.sync()" not in code, path        # (not said to be safe in a warp whose lanes arrive apart)
        for m in re.finditer(ALIGNED, code):
            body = code[code.rindex("{", 0, code.rindex("asm volatile", 0, m.start())):m.start()]
            assert "__syncwarp();" in body, (path, body)
            seen += 1
    assert seen == 3
