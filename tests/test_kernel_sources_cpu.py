"""Rules that the kernels' sources have to keep and no run can show."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "dscuda_b200" / "csrc"


def test_dependent_kernels_read_with_plain_loads():
    """ld.global.nc (__ldg, or const __restrict__ parameters) wants memory that nothing writes while the kernel lives.  A dependent
    launch lives from before the end of the kernel in front of it, whose results it reads."""
    for path in sorted(CSRC.glob("attention/*.cu*")):
        code = re.sub(r"//.*", "", path.read_text())
        assert not re.search(r"__ldg|ld\.global\.nc|__restrict__", code), path.name
