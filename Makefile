# Build the llark_b200 C-ABI library (sm_100a only).
NVCC ?= /usr/local/cuda/bin/nvcc
ARCH := -gencode arch=compute_100a,code=sm_100a
NVFLAGS := $(ARCH) -std=c++17 -O3 -lineinfo -Xcompiler -fPIC -Xptxas -v
SRC := $(wildcard llark_b200/csrc/*.cu)
OBJ := $(patsubst llark_b200/csrc/%.cu,build/%.o,$(SRC))
LIB := llark_b200/libllark_b200.so

# the subset a native checkpoint of a layer-list decoder needs: GEMM core, decode linears, generation-path ops
SERVE_OBJ := build/gemm_tcgen05.o build/gemv.o build/skinny.o build/attn_step.o build/seq_ops.o build/seq_mixers.o build/seq_swa_mma.o \
             build/seq_swa_tc.o build/seq_delta.o build/seq_latent.o build/seq_moe.o build/seq_decay.o build/seq_chunk.o
LIB_SERVE := llark_b200/libllark_serve.so

# a shared link accepts what it cannot resolve, and the library then fails to load: make that an error of the build
LDFLAGS := -shared -Xlinker --no-undefined

# the entry points as Python functions, for the interpreter PYTHON and under its name for extension modules, so that no other one takes them
# (without Python's headers the package calls the library through ctypes)
PYTHON ?= python3
PY := $(shell $(PYTHON) -c "import sysconfig as s; print(s.get_paths()['include'], s.get_config_var('EXT_SUFFIX'))" 2>/dev/null)
CALLS := $(if $(wildcard $(firstword $(PY))/Python.h),llark_b200/_calls$(lastword $(PY)))

all: $(LIB) $(CALLS)
serve: $(LIB_SERVE) $(CALLS)

ifneq ($(CALLS),)
$(CALLS): llark_b200/csrc/calls.cpp include/llark_b200.h
	@rm -f llark_b200/_calls.so
	g++ -std=c++17 -O2 -shared -fPIC -I$(firstword $(PY)) -I$(dir $(shell command -v $(NVCC)))../include -o $@ $< -ldl
endif

# all headers are behind all objects: a list for each was found short of one
build/%.o: llark_b200/csrc/%.cu $(wildcard llark_b200/csrc/*.cuh) include/llark_b200.h
	@mkdir -p build
	$(NVCC) $(NVFLAGS) -c $< -o $@ 2> build/$*.ptxas.log || (cat build/$*.ptxas.log; exit 1)

# the ALiBi instantiation #includes the attention source: rebuild it when that changes
build/attention_tc_alibi.o: llark_b200/csrc/attention_tc.cu

$(LIB): $(OBJ)
	$(NVCC) $(ARCH) $(LDFLAGS) -o $@ $(OBJ) -lnccl

$(LIB_SERVE): $(SERVE_OBJ)
	$(NVCC) $(ARCH) $(LDFLAGS) -o $@ $(SERVE_OBJ)

clean:
	rm -rf build $(LIB) $(LIB_SERVE) $(wildcard llark_b200/_calls*.so)
.PHONY: all serve clean
