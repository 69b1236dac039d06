"""Which decode steps run as one kernel: host logic, no GPU needed."""
import pytest

from rocml_b200.parts.decode_layers import pays


def step(lens, hidden, room=None):
    n = 1
    while n < len(lens):
        n *= 2
    return pays(n, hidden, max(lens), sum(lens), room or -(-max(lens) // 256) * 256)


@pytest.mark.parametrize("hidden", [1024, 2560, 4096])
def test_few_sequences(hidden):
    assert step([32000], hidden) and step([8000, 60], hidden) and step([32000, 60], hidden)
    assert step([2000, 60, 61, 62], hidden) and not step([3000, 60, 61], hidden) and step([3000, 2000, 1600], hidden)
    assert step([6000, 60, 61, 62], hidden) and step([8000, 7000, 6000, 5000], hidden) and not step([9000, 60, 61, 62], hidden)
    assert step([16000] * 3, hidden) and not step([17000] * 3, hidden) and step([32000] * 4, hidden)
    assert not step([30000, 8000, 1000, 17], hidden)


@pytest.mark.parametrize("hidden", [1024, 2560, 4096])
def test_five_to_eight(hidden):
    narrow = hidden < 4096
    assert step([150, 140, 40, 99, 17], hidden) and step([255] * 8, hidden)
    assert step([700, 780, 860, 950, 1050, 1150, 1250, 1385], hidden) == narrow
    assert step([1000] * 8, hidden) == narrow and step([4000] * 8, hidden) == narrow
    assert step([500] + [60] * 7, hidden) == narrow
    assert step([8000] * 6, hidden) and step([32000] * 8, hidden) and step([4600] * 7, hidden)
    for lens in ([700] + [60] * 7, [2000, 1900, 1800, 1700, 1600], [8000] + [60] * 7, [8000] * 5, [9000] * 6, [9000] * 7, [17000] * 4 + [15000] * 4):
        assert not step(lens, hidden)
