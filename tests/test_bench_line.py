"""bench.py's line of results."""
import json

import bench


def test_the_line_leaves_the_jobs_records_out(capsys):
    jobs = [{"name": "lif100x100", "served_latency_s": 1.25, "plain_setup_s": 0.1}] * 64
    line = {"metric": "m", "value": 1.0, "served": {"jobs": 64, "per_job": jobs}, "clocks": {"sm_mhz": 1}}
    bench.print_line(line)
    out, err = capsys.readouterr()
    assert json.loads(out) == {"metric": "m", "value": 1.0, "served": {"jobs": 64}, "clocks": {"sm_mhz": 1}}
    assert json.loads(err) == {"served": {"per_job": jobs}}
    assert line["served"]["per_job"] is jobs
