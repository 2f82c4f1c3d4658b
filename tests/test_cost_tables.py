"""The planner's cost tables describe the kernels there are: one system per lane,
one lane per bubble, padded to 16 and exact, two lanes per bubble padded to 32
and exact.  The values are a B200's, measured outside the tables (uniform
systems, 200 attempts with the GPU full, 1,500 alone); the tables come from other
systems, so they may differ from these by a quarter, while the forms differ from
one another and from what they replaced by more."""
import numpy as np
import pytest

from cbc_b200.ensemble import alone_latency, cost_weight, make_work_list, with_latency_lane

FULL_NS = {1: 0.163, 4: 1.99, 5: 4.04, 7: 6.81, 8: 6.62, 11: 35.8, 16: 25.1, 17: 122.0, 20: 123.0, 24: 125.0,
           31: 132.0, 32: 118.0}
ALONE_US = {1: 5.3, 4: 14.4, 5: 18.0, 7: 19.2, 8: 20.2, 11: 58.5, 16: 38.7, 17: 56.7, 20: 57.2, 24: 57.0, 31: 58.6,
            32: 46.8}


@pytest.mark.parametrize("K", sorted(FULL_NS))
def test_tables_near_the_measured_attempts(K):
    assert 0.75 < cost_weight(K)[0] / FULL_NS[K] < 1.33
    assert 0.75 < alone_latency(K)[0] / ALONE_US[K] < 1.33


def test_padded_forms_cost_more_than_the_exact_ones():
    assert np.all(cost_weight([11, 13, 15]) > cost_weight(16)) and np.all(alone_latency([9, 12, 15]) > alone_latency(16))
    assert np.all(cost_weight([17, 24, 31]) > cost_weight(32)) and np.all(alone_latency([17, 24]) > alone_latency(32))


def test_lanes_take_the_longest_serial_time():
    """Equal predicted steps: the padded count has the longer attempts."""
    K = np.repeat([16, 13, 8], 40)
    work = np.full(K.size, 100.0)
    wl = with_latency_lane(make_work_list(K, work), K, work, fraction=0.05, max_sms=4)
    lanes = [b for b in range(wl.bucket_K.size) if wl.exclusive[b] > 0]
    assert [int(wl.bucket_K[b]) for b in lanes] == [13]
