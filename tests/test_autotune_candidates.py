"""The autotuner times no launch twice: its candidates differ in the launch they give a bucket's form and size, so that
none is kept for the noise between two runs of one launch."""
import pytest

from wavebit_gb300 import autotune as AT


class Lib:
    def __init__(self):
        self.values = {}

    def wb_set_tuning(self, key, value):
        self.values[key] = value
        return 0

    def wb_get_tuning(self, key):
        return self.values.get(key, 0)


def _launch(form, n, qr, hrd):
    """The CTAs a pair of settings launches (0: the library's choice)"""
    most = {'double': 256, 'mixed': 512}.get(form, 768)
    sweep = min(max(qr, 128), most) if qr else 0
    return sweep, 0 if form == 'double' and 33 <= n <= 512 else hrd


@pytest.mark.parametrize('orders,form', [((5, 5), 'double'), ((7, 7), 'mixed'), ((12, 12), 'double'), ((3, 3), 'mixed_df64'),
                                         ((3, 0), 'double')])
def test_no_launch_is_timed_twice(orders, form):
    lib = Lib()
    n = 2 * (2 * orders[0] + 1) * (2 * orders[1] + 1)
    tuner = AT.Autotuner(lib=lib, timer=lambda run: 1.0)
    key = AT.bucket_key(orders, 2, 16, form)
    tuner.tune(key, lambda: None)
    launches = [_launch(form, n, t['settings']['qr_threads'], t['settings']['hrd_threads']) for t in tuner.table[key]['trials']]
    assert len(set(launches)) == len(launches), launches


def test_a_key_of_another_kind_keeps_every_candidate():
    assert AT.candidates('qr_threads', 'k') == AT.KNOBS['qr_threads'][1]
    assert AT.candidates('hrd_threads', 'k') == AT.KNOBS['hrd_threads'][1]
