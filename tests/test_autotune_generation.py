"""A launch shape that was timed on an earlier build of the column kernel is not taken from the cache
file; one of this build is (no GPU: a trial is a call of the stub's ``to``)."""
import types

import numpy as np
import pytest

from lica_boiling1d_b200 import autotune


class Trial(Exception):
    pass


def _batch():
    n = np.array([64, 128, 200], np.int32)

    def to(dev):
        raise Trial

    return types.SimpleNamespace(n=n, ncol=len(n), arrays={"w": types.SimpleNamespace(device="gpu")}, to=to)


@pytest.mark.parametrize("earlier", [True, False])
def test_entry_of_an_earlier_kernel(tmp_path, monkeypatch, earlier):
    monkeypatch.setenv("LICA_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(autotune, "_gpu_name", lambda dev: "GPU")
    monkeypatch.setattr(autotune, "_memo", {})
    b = _batch()
    key = f"GPU|{autotune.batch_key(b)}" if earlier else autotune.cache_key("GPU", b)
    autotune._store({key: {"threads": 256, "tri_cap": -1, "ms_per_step": {}}})
    if earlier:
        with pytest.raises(Trial):
            autotune.tune(b)
    else:
        assert autotune.tune(b) == ((256, -1), None)
