"""The launch configuration of the batched march that nobody set: it can be
read, written back and restored by the autotuner without becoming a set one."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_the_unset_configuration_survives_a_round_trip():
    from lunarscout_b200.autotune import tune_batch
    from lunarscout_b200.cuda_backend import BatchConfig, CudaSession

    session = CudaSession(0)
    try:
        unset = session.batch_config()
        assert unset.lanes_per_azimuth == 0  # each traversal's own
        session.set_batch_config(unset)
        assert session.batch_config() == unset
        tune_batch(session, [object()], device_out=0, apply=False, run=lambda s, t: 1.0)
        assert session.batch_config() == unset
        session.set_batch_config(BatchConfig(16, 6))
        assert session.batch_config() == BatchConfig(16, 6)
        session.set_batch_config(unset)
        assert session.batch_config() == unset
        for lanes in (-1, 3, 64):
            with pytest.raises(ValueError):
                session.set_batch_config(BatchConfig(lanes, 8))
        assert session.batch_config() == unset
    finally:
        session.close()
