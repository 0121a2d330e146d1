"""Host side of the frame batches: the sub-samples' listing on CPU tensors."""
import types

import numpy as np
import pytest
import torch

from solarsystemsimulator_b200 import nbody_kernel as nk


@pytest.mark.parametrize("n_ast", [1, 37, 500])
@pytest.mark.parametrize("k", [1, 5, 16])
@pytest.mark.parametrize("samples", [0, 1, 3, 100])
def test_sub_samples_are_listed_within_the_bound(monkeypatch, n_ast, k, samples):
    """The complete sub-samples of every sample, sample by sample, whatever the
    number of samples a pass takes; a pass copies at most SUB_GATHER_BYTES (or
    one sample)."""
    rng = np.random.default_rng(n_ast + k)
    ms, d, pad = 4, 3, 3
    subn = rng.integers(ms - 1, ms + 1, (16, n_ast + pad)).astype(np.uint8)
    subn[k // 2] = 0                                            # a sample without any
    subpos = rng.normal(size=(16, ms, d, n_ast + pad)).astype(np.float32)
    idx = rng.permutation(10 * n_ast)[:n_ast].astype(np.int64)
    st = {"n_ast": n_ast, "dim": d, "subn": torch.from_numpy(subn), "subpos": torch.from_numpy(subpos), "a_idx_h": idx}
    per_sample = n_ast * (4 * ms * d + 17)
    bound = samples * per_sample + 5
    monkeypatch.setattr(nk, "SUB_GATHER_BYTES", bound)
    seen, nonzero = [], torch.nonzero

    def counted(x, **kw):
        seen.append(x.numel() // n_ast * per_sample)
        return nonzero(x, **kw)

    monkeypatch.setattr(torch, "nonzero", counted)
    got = nk.NBodyCuda._collect_sub(types.SimpleNamespace(m_sub=ms), st, k)
    assert len(got) == k and max(seen) <= max(bound, per_sample)
    for ks, (who, pos) in enumerate(got):
        sel = np.flatnonzero(subn[ks, :n_ast] == ms)
        assert np.array_equal(who, idx[sel]) and np.array_equal(pos, subpos[ks][:, :, sel])
        assert pos.dtype == np.float32 and who.dtype == np.int64 and pos.flags.c_contiguous
