"""Page-locked host memory of a context: the small uploads' buffers and one for the
largest block on its way to a file, however often either is used."""
import re

import pytest

import scarl_b200 as S

pytestmark = pytest.mark.gpu


def locked_mb():
    """The driver's page-locked allocations are shared mappings of the process."""
    with open("/proc/self/status") as f:
        m = re.search(r"RssShmem:\s+(\d+) kB", f.read())
    if not m:
        pytest.skip("no RssShmem in /proc/self/status")
    return int(m[1]) / 1024


def test_file_writes_between_small_calls(tmp_path):
    import torch
    s = S.make_sample((0, 0, 0), (255, 255, 255), (4, 4, 4), (1, 1, 1), (5, 5, 5))
    lay = S.sample_layout(s)
    assert list(lay["L"]) == [256, 256, 256]
    f = torch.zeros(256 ** 3, dtype=torch.float32, device="cuda")  # 64 MB
    small = S.make_sample((0, 0, 0), (20, 20, 20), (4, 4, 4), (1, 1, 1), (5, 5, 5))
    torch.cuda.synchronize()
    with S.Context(0) as c:
        before = locked_mb()
        for _ in range(10):
            S.write_sample_h5(c, tmp_path, "f", f, s, lay)
            S.generate_sample(c, small, generator=S.GEN_DCT, dtype=S.F64, nb_procs=2, topo=(1, 1, 2))
        assert locked_mb() - before < 64 + 8 + 8
