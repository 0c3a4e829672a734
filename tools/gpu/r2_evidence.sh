#!/bin/bash
# Traffic of one training step, one GPU. No counter sets on full-size workloads: each capture below is one pass per launch, and runs
# only after the same command has ended well without ncu.
#   1. ncu launch list of one bench step (shares per kernel)                 -> <tag>_launches.csv
#   2. per-launch DRAM bytes + duration of every GEMM of the bench's shapes  -> <tag>_gemm_dram.csv + <tag>_gemm_shapes.json
# usage: bash tools/gpu/r2_evidence.sh <tag>
mkdir -p gpurun_out
TAG=${1:-r2f}
B="python bench.py --steps 1 --warmup 1 --no-cpu-baseline --no-torch-baseline --no-extras"
$B > gpurun_out/${TAG}_plain_bench.log 2>&1 &&
ncu --metrics gpu__time_duration.sum --clock-control none -c 12000 --csv --log-file gpurun_out/${TAG}_launches.csv \
  $B > gpurun_out/${TAG}_ncu_bench.log 2>&1
rc=$?
echo "launch list: $(grep -c gpu__time_duration gpurun_out/${TAG}_launches.csv) rows"
[ $rc -eq 0 ] || exit $rc
T="python tools/gemm_shape_trace.py --out gpurun_out/${TAG}_gemm_shapes.json"
$T > gpurun_out/${TAG}_plain_trace.log 2>&1 &&
ncu --metrics dram__bytes_read.sum,dram__bytes_write.sum,gpu__time_duration.sum --clock-control none \
  -k regex:gemm --csv --log-file gpurun_out/${TAG}_gemm_dram.csv $T > gpurun_out/${TAG}_gemm_trace.log 2>&1
rc=$?
tail -1 gpurun_out/${TAG}_gemm_trace.log
exit $rc
