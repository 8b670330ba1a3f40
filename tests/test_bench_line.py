"""bench.py's stdout line: one JSON line that the last 3000 characters of a log hold whole, whatever the other blocks
hold; its numbers are the full line's."""
import json

import pytest


def full_line(bench, args):
    big = {'%d dB' % i: {'value': 1.23456789e6 + i, 'text': 'x' * 200} for i in range(40)}
    return {
        'metric': bench.METRIC, 'value': 2448000.123456789, 'unit': 'detections/s', 'n_gpus': 8, 'steps': 20, 'warmup': 5,
        'ms_per_step': 26.77123456789, 'higher_is_better': True, 'scaling': 'weak', 'vs_baseline': None, 'dtype': 'int32',
        'data': 'synthetic (seeded Rayleigh draws on the device)', 'config': bench.config(args),
        'e2e': {'value': 2434000.987654321, 'unit': 'detections/s', 'h2d_bytes_per_step': 1090519040,
                'd2h_bytes_per_step': 8650752, 'ms_per_step': 26.912345678, 'steps': 20, 'path': 'p' * 300},
        'stages_ms': {'map': 2.9123456789, 'anneal': 22.812345678, 'readout': 1.012345678},
        'roofline': {'bound': 'int_issue', 'achieved': 23456.789012345, 'peak': 34567.890123456, 'unit': 'Gop/s',
                     'frac': 0.678901234567, 'traffic': 1234567890.123, 'kernel': 'k_anneal_grp<8, 8, 2, first accept>',
                     'ops_model': 'm' * 200, 'peak_source': 's' * 200},
        'roofline_issue': {'frac': 0.8123}, 'latency': {'p50_us': 64.123, 'p99_us': 71.456}, 'ber': big,
        'mdi_x16': {'value': 251234.5}, 'extra': {'chord_x32': {'value': 865444.77, 'more': big}},
        'warm_vs_plain': {k: {'plain': big, 'warm': {'speedup_vs_plain': 1.3456}} for k in ('x32', 'x64')},
        'serving': {'rates': {'1e+05 frames/s': {'per_class': {k: {'p99_us': 700.0 + i} for i, k in enumerate(big)}}}},
        'mixed': {'value': 1760000.0, 'more': big}, 'gpu_launches': 60,
        'clocks': {'sm_mhz': 1965.0, 'sm_max_mhz': 1965.0, 'reasons': [], 'samples': 166},
        'cpu_baseline': {'value': 1199.7795659102437, 'unit': 'detections/s', 'cores': 192, 'kind': 'port',
                         'sample': '14399 channel uses of the same workload (' + 'd' * 200}}


@pytest.mark.parametrize('blocks', [True, False])
def test_line_fits(blocks):
    import bench
    args = type('A', (), dict(batch=65536, anneals=32, world=8))()
    line = full_line(bench, args)
    if not blocks:
        for k in ('roofline_issue', 'cpu_baseline', 'mdi_x16', 'extra', 'warm_vs_plain', 'serving', 'mixed'):
            line[k] = None
        del line['cpu_baseline']
    text = json.dumps(bench.short(line))
    assert '\n' not in text and len(text) < 2500, len(text)
    out = json.loads(text)
    for k in ('metric', 'value', 'unit', 'n_gpus', 'steps', 'warmup', 'ms_per_step', 'higher_is_better', 'scaling',
              'vs_baseline', 'dtype', 'data', 'config', 'gpu_launches', 'clocks'):
        assert out[k] == line[k], k
    for k in ('value', 'unit', 'h2d_bytes_per_step', 'd2h_bytes_per_step'):
        assert out['e2e'][k] == line['e2e'][k], k
    assert out['summary']['serving_1e5_p99_ms'] == (739.0 / 1e3 if blocks else None)
