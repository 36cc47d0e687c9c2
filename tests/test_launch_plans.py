"""The host arithmetic that cuts and schedules launches; no GPU."""
import os
import subprocess
import sys

import pytest

import plans

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_device_of_one_sm_has_a_plan():
    """In a process of its own: half a device of one SM has no pair, and a plan for none would divide by zero."""
    code = "import plans; print([plans.lm_head(R, 2048, 8192, sms)['pairs'] for R in (16, 300) for sms in (0, 1)], plans.product(300, 768, 768, 1)['pair_width'])"
    res = subprocess.run([sys.executable, "-c", code], cwd=os.path.join(ROOT, "tests"), capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.split() == ["[0,", "0,", "0,", "0]", "0"], (res.returncode, res.stdout, res.stderr)


def _every_cut(R, V, rows, workers, most):
    """The cheapest of all split counts and widths; of several, the widest tiles and then the fewest splits."""
    limit = max(16, 160 // -(-R // 128))
    rbs, best = -(-R // rows), None
    for width in range(256, 127, -16):
        tiles = -(-V // width)
        for want in range(1, min(limit, tiles, most) + 1):
            tps = -(-tiles // want)
            sp = -(-tiles // tps)
            cost = float(-(-rbs * sp // workers)) * (tps * (width + 8) + 128) * (1.0 + 0.35 * (256 - width) / 256 if R > 128 else 1.0)
            if best is None or cost < best[0] - 1e-9:
                best = cost, dict(row_blocks=rbs, width=width, splits=sp, tiles_per_split=tps, pairs=int(rows == 256))
    return best


def test_lm_head_cut_is_the_cheapest_of_all():
    for R in (1, 16, 128, 129, 200, 256, 257, 300, 500, 1030, 3000, 8191, 20000, 37889, 600000):
        for V in (1, 128, 257, 777, 2064, 8192, 30000, 65536, 131071):
            for C, sms, most in ((2048, 148, plans.ALL), (768, 148, 16), (4096, 132, 7), (1088, 160, 1), (2048, 16, 40), (2048, 3, plans.ALL)):
                cost, cut = _every_cut(R, V, 128, sms, most)
                if R > 128:
                    pair_cost, pair_cut = _every_cut(R, V, 256, sms // 2, most)
                    if pair_cost * (0.92 + 80.0 / C) < cost:
                        cut = pair_cut
                assert plans.lm_head(R, C, V, sms, most) == cut, (R, C, V, sms, most)


@pytest.mark.parametrize("R,V", [(16, 65536), (128, 65536), (200, 65536), (16, 8192), (8191, 65536), (100000, 65536)])
def test_lm_head_cut_takes_no_time(R, V):
    """A call of few rows against a shard of the vocabulary is 10 us of GPU work: walking every split count took up to 33 us of host time."""
    assert plans.lm_head_ns(R, 2048, V) < 3000


# chains: {chunks: (us in sequence, us on SM partitions)}, 148 SMs
MEASURED = {
    2: {384: (268, 289), 1024: (686, 722), 4096: (2702, 2738)},
    3: {384: (275, 291), 1024: (703, 741), 2048: (1392, 1423), 4096: (2774, 2782)},
    4: {192: (148, 164), 384: (285, 298), 512: (369, 389), 1024: (721, 746), 2048: (1430, 1430), 4096: (2844, 2816)},
    5: {384: (287, 302), 768: (558, 573), 1536: (1102, 1097), 2048: (1465, 1449), 4096: (2918, 2844)},
    6: {384: (294, 307), 768: (573, 579), 1024: (756, 759), 1536: (1129, 1112), 4096: (3002, 2858)},
    7: {384: (300, 311), 512: (395, 403), 768: (585, 585), 1024: (775, 768), 2048: (1538, 1474)},
    8: {384: (307, 314), 512: (404, 405), 768: (598, 590), 1024: (795, 776), 4096: (3142, 2889)},
    10: {384: (320, 322), 512: (421, 415), 768: (627, 600), 2048: (1646, 1495)},
    12: {256: (228, 238), 320: (280, 286), 384: (334, 330), 512: (439, 423), 1024: (864, 799)},
    16: {192: (189, 192), 256: (247, 246), 320: (303, 296), 512: (476, 443)},
    24: {192: (217, 208), 1024: (1098, 867)},
    40: {192: (269, 261), 320: (436, 394)},
    56: {192: (324, 368), 256: (425, 471), 320: (527, 576)},
}


def test_scans_run_beside_operators_where_that_was_measured_to_pay():
    """The rule takes the faster schedule of each measured call, within the 0.6 % that two runs differ by."""
    for chains, row in MEASURED.items():
        for nchunks, (sequence, partitions) in row.items():
            taken = partitions if plans.overlap(chains, nchunks) else sequence
            assert taken <= 1.006 * min(sequence, partitions), (chains, nchunks)
