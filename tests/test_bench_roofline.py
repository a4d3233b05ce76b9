"""bench.py's FP32 roofline (CPU): a filtered CRS search does not evaluate the candidates that
the algorithm's count holds, so no count of its own operations stands beside it."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_filtered_search_has_no_count_of_its_own_operations():
    if ROOT not in sys.path:
        sys.path.insert(0, ROOT)
    import bench
    import semb
    st = dict(window=3, ncdps=10, ns=100, ncand=1000)
    direct = bench.fp32_roofline(semb.CRS, st, 5000, 1.0, 77.8)
    filtered = bench.fp32_roofline(semb.CRS, st, 5000, 1.0, 77.8, filtered=True)
    assert direct["filtered"] is False and 0 < direct["frac_own_ops"] < direct["frac"]
    assert filtered["filtered"] is True and filtered["frac"] == direct["frac"]
    assert filtered["frac_own_ops"] is None and filtered["achieved_own_ops"] is None
