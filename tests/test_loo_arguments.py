"""The route of a leave-one-out call's variogram: the kernels read nine numbers of M
and one each of sill and nugget from device memory, so tensors of other sizes must
not go there. The library is a recorder; nothing runs on a GPU."""
from types import SimpleNamespace

import pytest
import torch

from geo_bsd import hpgl_wrap as W
from geo_bsd import loo as L


@pytest.fixture
def calls(monkeypatch):
    made = []

    class Recorder:
        def __getattr__(self, name):
            return lambda *a: made.append(name) or 0

    monkeypatch.setattr(W, "_hpgl_so", Recorder())
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda self, stream: None)
    return made


def _call(M, sill, nugget):
    ints = torch.zeros(3, dtype=torch.int32)
    geom = SimpleNamespace(pts_xyz=ints, targets=ints, nb_idx=ints, nb_cnt=ints, k=1, cov_type=0)
    L._loo_call("hpgl_b200_loo_ok", geom, M, 1.0, sill, nugget, torch.zeros(1, dtype=torch.float64),
                SimpleNamespace(cuda_stream=0), ())


F64 = torch.float64


def test_a_whole_variogram_stays_on_the_device(calls):
    _call(torch.eye(3, dtype=F64), torch.tensor(1.0, dtype=F64), torch.tensor([0.1], dtype=F64))
    assert calls == ["hpgl_b200_loo_ok_device"]


@pytest.mark.parametrize("M", [torch.eye(2, dtype=F64), torch.zeros(0, dtype=F64), torch.ones(3, dtype=F64)])
def test_a_short_transform_is_not_read_on_the_device(calls, M):
    _call(M, torch.tensor(1.0, dtype=F64), torch.tensor(0.1, dtype=F64))
    assert calls == ["hpgl_b200_loo_ok"]


@pytest.mark.parametrize("sill,nugget", [(torch.ones(2, dtype=F64), torch.tensor(0.1, dtype=F64)),
                                         (torch.tensor(1.0, dtype=F64), torch.zeros(0, dtype=F64)),
                                         (torch.tensor(1.0, dtype=F64), torch.ones(3, dtype=F64))])
def test_a_sill_or_nugget_of_several_numbers_is_refused(calls, sill, nugget):
    with pytest.raises((TypeError, ValueError, RuntimeError)):
        _call(torch.eye(3, dtype=F64), sill, nugget)
    assert calls == []


def test_a_transform_of_more_than_nine_numbers_is_refused(calls):
    with pytest.raises(IndexError):
        _call(torch.ones(10, dtype=F64), torch.tensor(1.0, dtype=F64), torch.tensor(0.1, dtype=F64))
    assert calls == []
