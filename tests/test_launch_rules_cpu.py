"""Rules of the launches that depend on how many SMs a call has, compiled for the host and run without a GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_rules(tmp_path, body):
    source = tmp_path / "rules.cu"
    source.write_text('#include <cstdio>\n#include "%s/caffecontroll_b200/csrc/cct_internal.h"\nint main() {\n%s\n}\n' % (ROOT, body))
    exe = str(tmp_path / "rules")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-std=c++17", "-o", exe, str(source)], check=True)
    return [tuple(map(int, line.split())) for line in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]


def test_two_jobs_share_the_slots(tmp_path):
    """148 SMs and fewer, as while a reduction keeps some; layers with a slot for every tile, with up to two tiles a slot, and with more: no job
    without blocks, no more blocks than slots, blocks in proportion to the tiles, at most three rounds of them."""
    rows = run_rules(tmp_path, """
  for (int sms : {148, 140, 132, 16, 2})
    for (long long a : {1, 7, 40, 98, 196, 250, 500})
      for (long long b : {1, 16, 84, 98, 98 * 2, 300})
        std::printf("%d %lld %lld %d\\n", 2 * sms, a, b, share_slots(2 * sms, a, b));""")
    assert len(rows) == 5 * 7 * 6
    for slots, a, b, mine in rows:
        if a + b > 2 * slots:
            assert mine == 0
        elif a + b <= slots:
            assert mine == a
        else:
            theirs = min(b, slots - mine)
            assert 1 <= mine <= a and theirs >= 1 and mine + theirs <= slots
            rounds = max(-(-a // mine), -(-b // theirs))
            assert rounds <= 3 and abs(mine - slots * a / (a + b)) <= 1
    assert (280, 196, 98, 186) in rows and (296, 196, 98, 196) in rows
