"""Options given by position keep their meaning."""
import jaxtrace_gb300 as jt


def test_options_by_position():
    names = ["cuda_graph", "stage_fields", "stage_chunk", "stage_overlap", "row_sink", "record_path_length"]
    fields = list(jt.TrackerOptions.__dataclass_fields__)
    at = fields.index(names[0])
    assert fields[at:at + len(names)] == names
    before = [getattr(jt.TrackerOptions(), f) for f in fields[:at]]
    o = jt.TrackerOptions(*before, True, False, 16, False, None, True)
    assert [getattr(o, n) for n in names] == [True, False, 16, False, None, True]
