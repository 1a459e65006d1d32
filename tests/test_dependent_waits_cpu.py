"""The limit of a wait in a kernel that starts beside the one ahead does not count that one's time: who waits for what arrives only then
waits for that kernel first."""
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "csrc"


def test_issuers_wait_for_the_kernel_ahead():
    seen = 0
    for name in ("gemm_skinny.cu", "gemm_f32_tc.cu"):
        parts = (CSRC / name).read_text().split("- MMA issuer")
        for before, role in zip(parts, parts[1:]):
            kernel, role = before[before.rindex("__global__"):], role[:role.index("mbar_wait(")]
            assert "pdl_wait();" in role or "warp == kTcThreads / 32) {\n    pdl_wait();" in kernel, name
            seen += 1
    assert seen == 3
