"""Layers whose layout a test of the planners states and whose values a test on the GPU checks.  Math modes by name."""

# N, C, K, spatial, filter, padding; A slots of a converter group of the sweep kernel per mode (TF32 and bf16
# alike; 0: another kernel's).  Filters 3 wide with one to four channels have converters of their own.
SWEEP = [
    ((1, 1, 16, (6, 9, 132), (3, 3, 3), (1, 1, 1)), {"fp32": 2, "bf16": 2}),
    ((2, 2, 5, (5, 7, 140), (3, 3, 3), (1, 1, 1)), {"fp32": 2, "bf16": 2}),
    ((1, 2, 16, (6, 9, 132), (3, 3, 3), (0, 0, 0)), {"fp32": 2, "bf16": 2}),
    ((2, 3, 9, (8, 10, 132), (2, 2, 3), (0, 1, 1)), {"fp32": 2, "bf16": 2}),
    ((1, 3, 12, (6, 9, 200), (3, 3, 3), (1, 1, 1)), {"fp32": 2, "bf16": 2}),
    ((1, 4, 16, (7, 9, 140), (3, 3, 3), (1, 1, 1)), {"fp32": 2, "bf16": 2}),
    ((1, 4, 16, (148, 16, 132), (3, 3, 3), (1, 1, 1)), {"fp32": 1, "bf16": 2}),
    # the general converter: more channels, filters 2, 4 and 5 wide
    ((1, 5, 16, (6, 9, 132), (3, 3, 3), (1, 1, 1)), {"fp32": 2, "bf16": 2}),
    ((1, 12, 16, (5, 6, 132), (3, 3, 3), (1, 1, 1)), {"fp32": 0, "bf16": 2}),
    ((1, 16, 13, (6, 9, 132), (3, 3, 3), (1, 1, 1)), {"fp32": 0, "bf16": 1}),
    ((1, 2, 16, (9, 11, 132), (3, 3, 2), (1, 1, 0)), {"fp32": 2, "bf16": 2}),
    ((1, 3, 16, (6, 9, 128), (3, 3, 4), (1, 1, 2)), {"fp32": 2, "bf16": 2}),
    ((1, 3, 16, (6, 9, 132), (3, 3, 5), (1, 1, 2)), {"fp32": 2, "bf16": 2}),
    ((1, 4, 12, (7, 9, 136), (4, 3, 3), (1, 1, 1)), {"fp32": 0, "bf16": 2}),
]

# N, C, K, spatial, filter, stride: rows that the shift kernel lays side by side in parts, last parts short
STRIDED_ROWS_IN_PARTS = [(1, 8, 24, (40, 60, 132), (3, 3, 3), 2), (1, 16, 8, (40, 60, 131), (3, 3, 3), 2)]
# ... with the passes that do so per mode (some layers are next to such ones)
ROWS_IN_PARTS = [
    ((1, 32, 24, (9, 33, 64), (3, 3, 3), 1), {"fp32": ("fwd", "bwd_data"), "bf16": ("fwd",)}),
    ((2, 24, 28, (7, 20, 132), (3, 3, 3), 1), {"fp32": ("fwd", "bwd_data"), "bf16": ("fwd", "bwd_data")}),
    ((1, 12, 20, (9, 31, 177), (3, 3, 3), 1), {"fp32": ("fwd", "bwd_data"), "bf16": ("fwd", "bwd_data")}),
    ((1, 8, 8, (12, 40, 66), (3, 3, 3), 1), {"fp32": ("fwd", "bwd_data"), "bf16": ("fwd", "bwd_data")}),
    ((2, 32, 16, (75, 65), (3, 3), 1), {"fp32": ("bwd_data",), "bf16": ()}),
    ((1, 16, 24, (11, 23, 160), (3, 3, 3), 2), {"fp32": (), "bf16": ()}),
    (STRIDED_ROWS_IN_PARTS[0], {"fp32": ("fwd", "bwd_data"), "bf16": ("fwd", "bwd_data")}),
    (STRIDED_ROWS_IN_PARTS[1], {"fp32": ("fwd", "bwd_data"), "bf16": ("bwd_data",)}),
]

# N, C, K, spatial, filter, stride: forward by whole rows and bulk stores
STATISTICS_BY_BULK_STORES = (1, 24, 16, (64, 64, 64), (3, 3, 3), 1)
