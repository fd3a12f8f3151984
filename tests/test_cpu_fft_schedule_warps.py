"""The ring FFT pass schedule for the smaller ring CTAs (4 and 8 warps), and
for the radix-4 passes of the shortest rings (4 warps): the checks of
test_cpu_fft_schedule.py with their warp count, buffer and radix."""
import pytest

from . import test_cpu_fft_schedule as schedule


@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("order", ["dif", "dit"])
def test_schedule_of_smaller_ctas(monkeypatch, warps, order):
    monkeypatch.setattr(schedule, "WARPS", warps)
    monkeypatch.setattr(schedule, "THREADS", 32 * warps)
    monkeypatch.setattr(schedule, "BUFFER", 512 * warps)
    schedule.test_every_butterfly_once_and_warp_local_reads_own_writes(order)


@pytest.mark.parametrize("order", ["dif", "dit"])
def test_schedule_of_radix_4_passes(monkeypatch, order):
    def radices(M):
        lgM = M.bit_length() - 1
        r0, n = lgM % 2, (lgM + 1) // 2
        r = [2 if (r0 and p == n - 1) else 4 for p in range(n)]
        lgl = [lgM - 2 * p for p in range(n)]
        return n, r, lgl, [lgl[1] if 1 <= p < n else 0 for p in range(n)]

    monkeypatch.setattr(schedule, "radices", radices)
    monkeypatch.setattr(schedule, "WARPS", 4)
    monkeypatch.setattr(schedule, "THREADS", 128)
    monkeypatch.setattr(schedule, "BUFFER", 2048)
    schedule.test_every_butterfly_once_and_warp_local_reads_own_writes(order)
