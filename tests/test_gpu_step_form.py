"""The engine's tests again with one launch per cycle: networks of their sizes run many cycles per
launch by default, so this is where the step kernel's push, pull and tiled delivery, its graphs and
its hand-overs are held against the oracle (the launch shape is fixed to what the engine would take;
every run is checked to take that form)."""
import pytest

import bsim_b200 as B
from test_drive_neurons import (test_mixed_network_exact_vs_oracle, test_mixed_network_ordered_vs_reference_order,  # noqa: F401
                                test_mixed_networks_batched_equal_alone)
from test_fp64_rates import test_engine_rates_vs_double_reference  # noqa: F401
from test_gpu_edges import (test_bounded_wait_times_out_with_a_device_error, test_every_neuron_fires_every_cycle,  # noqa: F401
                            test_no_synapses, test_ragged_sizes, test_raster_into_caller_buffer,
                            test_silent_sources_and_unreached_targets,
                            test_tiled_segment_lengths_around_the_bank_ordering_limit)
from test_gpu_parity import (c0, test_auto_delivery_vs_oracle_switching_modes, test_batched_equals_alone,  # noqa: F401
                             test_c0_exact_push_vs_oracle, test_c0_ordered_pull_bit_exact_vs_reference_order,
                             test_device_builder_matches_host_builder, test_push_pull_graph_identical,
                             test_scaled_replicas_vs_oracle, test_square_wave_drive_vs_oracle,
                             test_tiled_batched_long_delays_equal_alone, test_tiled_delivery_identical_to_push,
                             test_tiled_delivery_rates_over_a_full_second,
                             test_tiled_delivery_vs_oracle_at_bench_shapes, test_unit_nets_exact_bit_exact,
                             test_unit_nets_ordered_bit_exact)
from test_predictor import (test_auto_without_tiled_copy_pushes_every_cycle, test_autotune_keeps_dynamics,  # noqa: F401
                            test_autotune_of_a_tiled_engine_keeps_dynamics,
                            test_exact_schedule_switches_modes_and_keeps_dynamics,
                            test_population_degrees_from_every_synapse_copy,
                            test_predictor_scheduling_keeps_rasters_identical, trained)
from test_trace import test_trace_equals_per_cycle_state, test_trace_restart_and_partial_read  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def one_launch_per_cycle(monkeypatch):
    default, run = B.options, B.Engine.run

    def options(**kw):
        return default(**{"block_threads": 512, **kw})

    def checked_run(self, steps):
        run(self, steps)
        i = self.info()
        assert i.many_cycles == 0
        if i.delivery == B.DELIVERY_TILE:
            self._tiled = getattr(self, "_tiled", 0) + steps
            assert i.tile_cycles >= self._tiled

    monkeypatch.setattr(B, "options", options)
    monkeypatch.setattr(B.Engine, "run", checked_run)


@pytest.mark.parametrize("delivery,form", [(B.DELIVERY_PUSH, 1), (B.DELIVERY_TILE, 1), (B.DELIVERY_AUTO, 1),
                                           (B.DELIVERY_PULL, 2)])
def test_the_reported_form_follows_the_engine(delivery, form):
    """A network of this size runs many cycles per launch unless the launch shape or the graph length
    asks for one launch per cycle; the cycles delivered tiled are counted."""
    from bsim_b200 import workloads as W
    sp = W.cuba(4, 200, 500, 6, seed=2)
    for kw, want in ((dict(block_threads=0), form), (dict(), 0), (dict(block_threads=0, grid_blocks=64), 0),
                     (dict(block_threads=0, graph_steps=0), 0)):
        eng = B.Engine.generated(sp, 1e-4, opts=B.options(delivery=delivery, **kw))
        B._check(B.lib().bsim_run(eng._h, 70))
        i = eng.info()
        assert i.many_cycles == want
        assert i.tile_cycles == (70 if want == 0 and delivery == B.DELIVERY_TILE else 0)
        eng.close()
