"""The ensemble tuners on the CPU, the library's calls recorded and the times
made up: they start from the contraction the ensemble runs with (0x3c in FP64,
0x30 in mixed precision), leave orders that are not present as they are, and
report and cache the mask that is applied."""
from types import SimpleNamespace

import pytest

import exahype_b200 as E
from exahype_b200 import autotune, ensemble


@pytest.fixture
def make(monkeypatch):
    def fake_call(name, *args):
        applied.append((name, args))

    applied = []
    monkeypatch.setattr(ensemble, 'call', fake_call)

    def build(precision, orders, times=lambda mask: 1.0):
        monkeypatch.setattr(autotune, '_time_ensemble', lambda ens, steps: times(masks(applied, precision)[-1]))
        e = ensemble.Ensemble(8, 1 << 20, precision=precision)
        e.cfgs = {i: SimpleNamespace(order=n) for i, n in enumerate(orders)}
        return e, applied

    return build


def masks(applied, precision):
    """the contraction masks in force, the library's default first"""
    default = 0x30 if precision == E.PREC_MIXED else 0x3c
    return [default] + [a[-1] for n, a in applied if n == 'exa_ensemble_tune_contraction']


@pytest.mark.parametrize('precision,default', [(E.PREC_FP64, 0x3c), (E.PREC_MIXED, 0x30)])
def test_schedule_alone_keeps_and_caches_the_contraction(make, tmp_path, precision, default):
    cache = str(tmp_path / 'tuned.json')
    e, applied = make(precision, (2, 3))
    best, _ = autotune.tune_ensemble(e, contraction=False, cache=cache, key='k')
    assert best[3] == masks(applied, precision)[-1] == default
    e, applied = make(precision, (2, 3))
    got, _ = autotune.tune_ensemble(e, contraction=False, cache=cache, key='k')
    assert got == best and masks(applied, precision)[-1] == default


@pytest.mark.parametrize('precision,default', [(E.PREC_FP64, 0x3c), (E.PREC_MIXED, 0x30)])
def test_descent_starts_from_the_default(make, precision, default):
    e, applied = make(precision, (4, 5))
    mask, table = autotune.tune_contraction(e)
    assert table[0]['lines_mask'] == default
    assert mask == masks(applied, precision)[-1] == default
    e, applied = make(precision, ())
    assert autotune.tune_contraction(e)[0] == default


def test_descent_flips_what_is_faster_and_keeps_absent_orders(make):
    e, applied = make(E.PREC_FP64, (4,), times=lambda mask: 2.0 if mask & 0x10 else 1.0)
    best, table = autotune.tune_ensemble(e)
    assert best[3] == masks(applied, E.PREC_FP64)[-1] == 0x2c
    assert e.lines_mask == 0x2c
    assert autotune.tune_contraction(e)[1][0]['lines_mask'] == 0x2c
    assert autotune.tune_contraction(e, mask=0x30)[1][0]['lines_mask'] == 0x30


def test_mask_follows_an_accepted_call_only(make, monkeypatch):
    e, _ = make(E.PREC_FP64, (2,))
    e.tune_contraction(0x0c)
    assert e.lines_mask == 0x0c

    def refuse(*a):
        raise E.ExaError(1, 'tune_contraction')

    monkeypatch.setattr(ensemble, 'call', refuse)
    with pytest.raises(E.ExaError):
        e.tune_contraction(0x40)
    assert e.lines_mask == 0x0c
    monkeypatch.setattr(ensemble, 'call', lambda *a: None)
