"""The autotuner times only what a kernel reads, and applies no table measured on other kernels (no GPU)."""
import json

import pytest

torch = pytest.importorskip("torch")

from wbgpu import autotune  # noqa: E402


@pytest.fixture(autouse=True)
def _reset_table():
    yield
    autotune.reset()


@pytest.mark.parametrize("nw,mode,names", [
    (8, 1, {'eigh_tridiag_group', 'eigh_ql_block', 'eigh_vectors_group'}),
    (32, 3, {'eigh_tridiag_group', 'eigh_ql_block', 'eigh_vectors_group'}),
    (33, 1, {'eigh_ql_block'}),  # above 32 a matrix has a block of its own in the other two kernels
    (96, 3 | autotune.PRECISE_VECTORS, {'eigh_ql_block'}),
])
def test_eigensolver_groups(monkeypatch, nw, mode, names):
    monkeypatch.setattr(autotune, '_eigh_runner', lambda *a: None)
    monkeypatch.setattr(autotune, '_time_ms', lambda *a: 1.0)
    entry, timings = autotune.tune_eigh(nw, mode)
    assert set(entry) == set(timings) == names


@pytest.mark.parametrize("nw", [4, 16, 32, 64])
def test_fp64_rotation_has_nothing_to_tune(nw):
    assert autotune.tune_rotate(nw, 1) == ({}, {})  # (a launch would need a GPU)


def test_tables_of_other_kernels_are_measured_again(monkeypatch, tmp_path):
    path = str(tmp_path / 'tune.json')
    monkeypatch.setattr(torch.cuda, 'get_device_name', lambda d: 'GB300')
    calls = []
    monkeypatch.setattr(autotune, 'tune_eigh', lambda *a, **k: (calls.append(1), ({'eigh_ql_block': 64}, {}))[1])
    monkeypatch.setattr(autotune, 'tune_rotate', lambda *a, **k: ({}, {}))
    # what a library with the same ABI and earlier kernels has left
    with open(path, 'w') as f:
        json.dump({'GB300|abi1|nw8|fp64': {'eigh_ql_block': 256, 'eigh_tridiag_group': 1}}, f)
    assert autotune.ensure(8, 'fp64', path=path) == {'eigh_ql_block': 64} and len(calls) == 1
    assert autotune.ensure(8, 'fp64', path=path) == {'eigh_ql_block': 64} and len(calls) == 1  # its own, from the file
    monkeypatch.setattr(autotune, 'KERNELS', autotune.KERNELS + 1)
    autotune.ensure(8, 'fp64', path=path)
    assert len(calls) == 2
