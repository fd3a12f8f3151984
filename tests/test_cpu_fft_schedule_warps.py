"""The ring FFT pass schedule for the smaller ring CTAs (4 and 8 warps): the
checks of test_cpu_fft_schedule.py with their warp count and buffer."""
import pytest

from . import test_cpu_fft_schedule as schedule


@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("order", ["dif", "dit"])
def test_schedule_of_smaller_ctas(monkeypatch, warps, order):
    monkeypatch.setattr(schedule, "WARPS", warps)
    monkeypatch.setattr(schedule, "THREADS", 32 * warps)
    monkeypatch.setattr(schedule, "BUFFER", 512 * warps)
    schedule.test_every_butterfly_once_and_warp_local_reads_own_writes(order)
