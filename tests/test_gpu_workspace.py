"""The binning's stage is sized for the classes that a frame runs, not for all that there are."""
import pytest

import scenes as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_first_frame_takes_what_its_classes_need(pf):
    torch = pytest.importorskip("torch")
    sc = S.plain_small(seed=1, n_paths=240, side=1024)

    def taken():
        with pf.Renderer() as r:
            r.upload(sc)
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            r.render()
            torch.cuda.synchronize()
            return before - torch.cuda.mem_get_info()[0]

    taken()  # the kernels' own memory, loaded with their first launch
    # 240 paths, each a CTA of the largest class: 240 * 12,288 visits of 12 bytes and a quarter more
    # (42 MB); lines, tiles and fills of this scene stay under 8 MB, and blocks are rounded up to 2 MB
    assert taken() <= 42 * MB + 8 * MB + 30 * 2 * MB // 3
