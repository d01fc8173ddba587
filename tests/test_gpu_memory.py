"""Device memory of an FP64 handle.  The domains that fit are part of what the
library accepts, so the arrays of the contracting FP64 step stay within what a
step needs: 60 words a point, counted over the state and both advected-field
sets (26), diagnostics and water totals (6), s, deltaw and the two divergences
(4), the column solve's sweep (2), the advection's intermediate fields (10),
and the static metric terms (12).  One word more is 1.7 %; the plane fields,
the handle's small tables and what an allocation rounds up to are 0.6 % here."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,word", [("fp64", 8), ("fp64_exact", 8)])
def test_words_a_point(gpu_lib, mode, word):
    torch = pytest.importorskip("torch")
    jx, iy, kz = 256, 256, 60
    torch.cuda.synchronize()
    warm = gpu_lib.Moloch(8, 8, 4, mode=mode)  # the context's own memory
    free0 = torch.cuda.mem_get_info()[0]
    g = gpu_lib.Moloch(jx, iy, kz, mode=mode)
    used = free0 - torch.cuda.mem_get_info()[0]
    words = used / word / (jx * iy * kz)
    print(f"{mode}: {words:.2f} words a point")
    assert words <= 60 * 1.016
    g.close()
    warm.close()
