"""The tuner times the match search's haplotypes per CTA only for the search that
reads them (with set-maximal errors)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_search_knob_is_timed_where_it_is_read():
    import torch
    from eimp_b200 import synth
    from eimp_b200.autotune import KNOBS, get, set_shape, tune_group
    from eimp_b200.batch import DensityGroup
    from eimp_b200.engine import PhaseParams
    panel, groups = synth.generate("cfg1")
    tg = groups[0]
    dev = torch.device("cuda", 0)
    hm, sm, cm = synth.typed_views(panel, tg.typed)
    g = DensityGroup(0, torch.from_numpy(panel.sitemajor.view(np.int64)).to(dev),
                     torch.from_numpy(panel.af.astype(np.float32)).to(dev), panel.nhaps, tg.typed, hm, sm, cm, tg.gt[:8],
                     PhaseParams(K=256, beamwidth=32), batch_targets=8)
    set_shape(g, "smm_warps", 4)
    assert tune_group(g, reps=1, knobs=("smm_warps",)) == {"smm_warps": {"chosen": 4, "ms": {}}}
    assert get(g, "smm_warps") == 4
    r = tune_group(g, reps=1, knobs=("smm_warps",), setmaxerrors=1)["smm_warps"]
    assert len(r["ms"]) == 3 and get(g, "smm_warps") == r["chosen"] and r["chosen"] in KNOBS["smm_warps"][1]
    g.close()
